"""CPU checks of the engine's host code against a CUDA runtime that delays queued
work as long as it may (tests/engine_host.cpp): what a call leaves queued, and in
which order tables reach device memory."""
import ctypes as C
import re
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "nqpu_b200" / "csrc"
SO = ROOT / "tests" / "_build" / "libenginehost.so"


@pytest.fixture(scope="module")
def eng():
    SO.parent.mkdir(exist_ok=True)
    srcs = [ROOT / "tests" / "engine_host.cpp", *(CSRC / f for f in ("engine.cpp", "planner.cpp", "tileprog.cpp"))]
    deps = srcs + list(CSRC.glob("*.h"))
    if not SO.exists() or SO.stat().st_mtime < max(d.stat().st_mtime for d in deps):
        subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-Wl,-z,defs,-Bsymbolic", "-I",
                        "/usr/local/cuda/include", "-I", str(CSRC), *map(str, srcs), "-o", str(SO)], check=True)
    return C.CDLL(str(SO))


@pytest.mark.parametrize("size", [0, 1, 16, 100000])
def test_table_has_landed_when_its_upload_returns(eng, size):
    assert eng.check_upload(size) == 0


def test_no_copy_on_the_default_stream():
    # states, batches and request lanes run on non-blocking streams, which do not
    # wait for what a plain cudaMemcpy of pageable memory leaves in flight
    plain = re.compile(r"\bcudaMemcpy\s*\(")
    found = [f"{p.name}:{i}" for p in sorted(CSRC.iterdir()) if p.suffix in (".cu", ".cpp", ".h", ".cuh")
             for i, line in enumerate(p.read_text().splitlines(), 1) if plain.search(line.split("//")[0])]
    assert not found, found


@pytest.mark.parametrize("what", [0, 1, 2])
def test_no_measurement_outlives_an_error(eng, what):
    assert eng.check_measure_error(what) == 0


@pytest.mark.parametrize("n", [12, 17, 22])
def test_auto_plans_a_tiled_circuit_once(eng, n):
    assert eng.check_auto_plans_once(n) == 0


def test_auto_chooses_again_for_another_tile_size(eng):
    assert eng.check_auto_follows_tiles() == 0


def test_a_pass_is_launched_where_its_tiles_fit(eng):
    assert eng.check_launch_config() == 0


def test_sweeps_alternate_where_the_l2_does_not_hold_the_state(eng):
    assert eng.check_sweeps() == 0
