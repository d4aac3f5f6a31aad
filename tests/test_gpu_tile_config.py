"""Every configuration of the tiled pass kernel against the oracle, and the library's
own choice where it takes complex64 tiles of 13 qubits.  Tolerances are the
engine's: complex128 1e-12 per amplitude (under 10 roundings of 2^-53 per gate, 1000
gates), complex64 1 - fidelity <= 1e-5.
"""
import numpy as np
import pytest

from nqpu_b200 import _lib, circuits
from nqpu_b200.state import Circuit, StateVector
from oracle import oracle as O

pytestmark = pytest.mark.gpu
C128, C64 = 0, 1
EVERY = [k for k in circuits.ARITY if k != "u2lo"]


def unitary(rng, d):
    q, r = np.linalg.qr(rng.normal(size=(d, d)) + 1j * rng.normal(size=(d, d)))
    return q * (np.diag(r) / np.abs(np.diag(r)))


def mixed(rng, n, count):
    gates = [("u3", (q,), tuple(rng.uniform(0, 6, 3))) for q in range(n)]
    for _ in range(count):
        name = EVERY[int(rng.integers(len(EVERY)))]
        qs = tuple(int(x) for x in rng.choice(n, size=circuits.ARITY[name], replace=False))
        d = {"custom1": 2, "custom2": 4}.get(name)
        gates.append((name, qs, (), unitary(rng, d)) if d else (name, qs, tuple(rng.uniform(-6, 6, 4))))
    return gates


@pytest.fixture
def tile_config():
    lib = _lib.load()
    saved = [lib.nqpu_tile_config_get(d) for d in (C128, C64)]
    yield lambda dtype, cfg: _lib.check(lib.nqpu_tile_config_set(C64 if dtype == "c64" else C128, cfg))
    for d in (C128, C64):
        lib.nqpu_tile_config_set(d, saved[d])


def check(n, dtype, circuit, gates):
    with StateVector(n, dtype) as sv:
        circuit.execute(sv, "tiled")
        got = sv.amplitudes()
    o = O.OracleState(n)
    o.apply(gates)
    ref = o.amplitudes()
    if dtype == "c128":
        assert np.abs(got - ref).max() <= 1e-12
    assert 1 - abs(np.vdot(got, ref)) ** 2 / (np.vdot(got, got).real * np.vdot(ref, ref).real) <= 1e-5


# the smallest state, one partly filled tile, one whole tile, two, several per SM
@pytest.mark.parametrize("n", [5, 8, 12, 13, 14, 18, 21])
@pytest.mark.parametrize("cfg", [1, 2, 4])
@pytest.mark.parametrize("dtype", ["c64", "c128"])
def test_configurations(tile_config, dtype, cfg, n):
    gates = mixed(np.random.default_rng(100 * n + cfg), n, 150 if n < 20 else 80)
    tile_config(dtype, cfg)
    check(n, dtype, Circuit(n, gates), gates)


def test_one_circuit_under_every_configuration(tile_config):
    n = 16
    gates = mixed(np.random.default_rng(3), n, 120)
    c = Circuit(n, gates)
    for cfg in (0, 4, 1, 2, 4, 0):
        tile_config("c64", cfg)
        check(n, "c64", c, gates)


def test_library_takes_13_bit_tiles(tile_config):
    n = 23
    gates = [("ry", (q,), (0.3 + 0.1 * q,)) for q in range(0, 5)] + circuits.qft(n)
    c = Circuit(n, gates)
    passes = {}
    for cfg in (2, 4, 0):
        tile_config("c64", cfg)
        passes[cfg] = c.plan_stats(n, "c64", "tiled")["passes"]
    assert passes[0] == passes[2] < passes[4]
    check(n, "c64", c, gates)


# per-gate launches in both directions: 128 MB of state, every kind of gate
@pytest.mark.parametrize("n,dtype", [(24, "c64"), (23, "c128")])
def test_pergate_both_directions(n, dtype):
    rng = np.random.default_rng(n)
    gates = [("u3", (q,), tuple(rng.uniform(0, 6, 3))) for q in range(0, n, 3)]
    for name in EVERY + ["x", "x", "rz", "rz", "swap", "cx"]:
        qs = tuple(int(x) for x in rng.choice(n, size=circuits.ARITY[name], replace=False))
        d = {"custom1": 2, "custom2": 4}.get(name)
        gates.append((name, qs, (), unitary(rng, d)) if d else (name, qs, tuple(rng.uniform(-6, 6, 4))))
    gates += [("x", (0,), ()), ("rz", (0,), (0.3,)), ("h", (0,), ()), ("cz", (0, n - 1), ()), ("cp", (1, 0), (0.4,))]
    with StateVector(n, dtype) as sv:
        Circuit(n, gates).execute(sv, "pergate")
        got = sv.amplitudes()
    o = O.OracleState(n)
    o.apply(gates)
    ref = o.amplitudes()
    if dtype == "c128":
        assert np.abs(got - ref).max() <= 1e-12
    assert 1 - abs(np.vdot(got, ref)) ** 2 / (np.vdot(got, got).real * np.vdot(ref, ref).real) <= 1e-5
