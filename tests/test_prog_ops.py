"""CPU check of lowered ops beyond what the interface's gates lower to, through the
stage program compiler (tests/prog_ops.cpp)."""
import ctypes as C
import itertools
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
SO = ROOT / "tests" / "_build" / "libprogops.so"
CSRC = ROOT / "nqpu_b200" / "csrc"


@pytest.fixture(scope="module")
def ops():
    SO.parent.mkdir(exist_ok=True)
    srcs = [ROOT / "tests" / "prog_ops.cpp", CSRC / "planner.cpp", CSRC / "tileprog.cpp"]
    deps = srcs + [ROOT / "tests" / "prog_emulator.cpp"] + [CSRC / h for h in ("sv_types.h", "planner.h", "tileprog.h")]
    if not SO.exists() or SO.stat().st_mtime < max(d.stat().st_mtime for d in deps):
        subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", str(CSRC), *map(str, srcs), "-o",
                        str(SO)], check=True)
    lib = C.CDLL(str(SO))
    lib.controlled_2x2.restype = C.c_double
    return lib


@pytest.mark.parametrize("c64", [0, 1])
def test_controlled_2x2(ops, c64):
    n = 5 if c64 else 4
    for t in range(n):
        others = [q for q in range(n) if q != t]
        for k in range(4):
            for cs in itertools.combinations(others, k):
                mask = sum(1 << q for q in cs)
                # 11 gates: operands rounded to 2^-24 (complex64), FP64 otherwise
                assert 0 <= ops.controlled_2x2(c64, t, mask) <= (11 * 2.0 ** -24 if c64 else 1e-14)
                assert ops.controlled_records(c64, t, mask) == (1 if k else 0)
