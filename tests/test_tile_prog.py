"""CPU check of the stage programs the tile kernels run: tests/prog_emulator.cpp
interprets the compiled words and the result is compared with the oracle, gate
mix by gate mix (merged phases, real and cross 2x2s, sign flips, records)."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from nqpu_b200 import circuits
from oracle.oracle import OracleState

ROOT = Path(__file__).resolve().parent.parent
SO = ROOT / "tests" / "_build" / "libprogemu.so"
CSRC = ROOT / "nqpu_b200" / "csrc"


@pytest.fixture(scope="module")
def emu():
    SO.parent.mkdir(exist_ok=True)
    srcs = [ROOT / "tests" / "prog_emulator.cpp", CSRC / "planner.cpp", CSRC / "tileprog.cpp"]
    deps = srcs + [CSRC / h for h in ("sv_types.h", "planner.h", "tileprog.h")]
    if not SO.exists() or SO.stat().st_mtime < max(d.stat().st_mtime for d in deps):
        subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", str(CSRC), *map(str, srcs), "-o",
                        str(SO)], check=True)
    lib = C.CDLL(str(SO))
    lib.prog_run.restype = C.c_int
    return lib


def run(lib, n, c64, gates, kmax=None):
    flat = np.ascontiguousarray(circuits.flatten(gates))
    st = np.zeros(2 << n)
    st[0] = 1.0
    stats = (C.c_int64 * 3)()
    ptr = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))  # noqa: E731
    rc = lib.prog_run(n, int(c64), kmax or (12 if c64 else 12), ptr(flat), len(flat), ptr(st), stats)
    assert rc == 0
    return st.view(np.complex128), list(stats)


def random_unitary(rng, d):
    q, r = np.linalg.qr(rng.normal(size=(d, d)) + 1j * rng.normal(size=(d, d)))
    return q * (np.diag(r) / np.abs(np.diag(r)))


MIXES = {
    "any": [k for k in circuits.ARITY if k != "u2lo"],
    "diagonal": ["z", "s", "t", "rz", "p", "cz", "cp", "crz", "rzz", "ccz", "h", "ry", "rx"],
    "one_qubit": ["h", "x", "y", "sx", "rx", "ry", "rz", "u3", "custom1", "t", "z", "cx"],
    "controlled": ["cx", "ccx", "cswap", "crx", "cry", "crz", "cu", "cz", "ccz", "swap", "iswap", "ry", "p"],
}


def mixed(rng, n, count, names):
    names = [k for k in names if circuits.ARITY[k] <= n]
    gates = [("u3", (q,), tuple(rng.uniform(0, 6, 3))) for q in range(n)]
    for _ in range(count):
        name = names[int(rng.integers(len(names)))]
        qs = tuple(int(x) for x in rng.choice(n, size=circuits.ARITY[name], replace=False))
        m = {"custom1": 2, "custom2": 4}.get(name)
        gates.append((name, qs, (), random_unitary(rng, m)) if m else (name, qs, tuple(rng.uniform(-6, 6, 4))))
    return gates


def check(got, gates, n, c64):
    o = OracleState(n)
    o.apply(gates)
    # complex64 operands are rounded to 2^-24 (angles to 2^-33 turns): at most one
    # such error per gate, in all under 2^-24 x gates
    tol = len(gates) * 2.0 ** -24 if c64 else 1e-12
    assert np.abs(got - o.amplitudes()).max() <= tol


@pytest.mark.parametrize("c64", [False, True])
@pytest.mark.parametrize("mix", sorted(MIXES))
@pytest.mark.parametrize("n,kmax", [(5, 12), (7, 12), (10, 7), (13, 12)])
def test_mixes(emu, mix, n, kmax, c64):
    for seed in range(4):
        rng = np.random.default_rng(1000 * n + seed)
        gates = mixed(rng, n, 14 * n, MIXES[mix])
        got, _ = run(emu, n, c64, gates, kmax)
        check(got, gates, n, c64)


@pytest.mark.parametrize("c64", [False, True])
@pytest.mark.parametrize("n", [8, 13])
def test_workloads(emu, n, c64):
    for gates in (circuits.qft(n), circuits.tfim_trotter(n, 4, 2)[0], circuits.hea(n, 4, np.random.default_rng(3)),
                  circuits.brickwork(n, 6, 5)):
        prep = [("u3", (q,), (0.3 + q, 0.2 * q, 1.0)) for q in range(n)]
        got, _ = run(emu, n, c64, prep + gates)
        check(got, prep + gates, n, c64)


@pytest.mark.parametrize("n,dtype", [(5, "c64"), (4, "c128")])
def test_compile_time_is_linear_in_the_gates(n, dtype):
    # a circuit on as many qubits as a stage has register bits is one stage: 8 times the gates may take 8 times as
    # long (64 times if every round walked all of them); a factor of 3 for noise
    import time

    from nqpu_b200.state import Circuit

    def best(steps):
        c = Circuit(n, circuits.tfim_trotter(n, steps, 1)[0])
        times = []
        for _ in range(3):
            t = time.perf_counter()
            c.plan_stats(n, dtype, "tiled")
            times.append(time.perf_counter() - t)
        return min(times)

    assert best(2000) <= 24 * best(250)


def test_compile_time_against_lowering():
    # a circuit that runs once pays for its programs: planning and compiling a
    # 17-qubit brickwork takes 9 times as long as lowering its gates (15 times with
    # an angle per phase table entry and the matrices tested at every look)
    import time

    from nqpu_b200.state import Circuit

    c = Circuit(17, circuits.brickwork(17, 15, 1))

    def best(mode):
        times = []
        for _ in range(100):
            t = time.perf_counter()
            c.plan_stats(17, "c64", mode)
            times.append(time.perf_counter() - t)
        return min(times)

    assert best("tiled") <= 12 * best("pergate")
