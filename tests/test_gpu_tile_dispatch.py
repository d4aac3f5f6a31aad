"""The tiled, per-gate and measurement paths at the sizes where their dispatch
changes, against the oracle.  Tolerances are the engine's: complex128 1e-12 per
amplitude (under 10 roundings of 2^-53 per gate, 1000 gates), complex64
1 - fidelity <= 1e-5.
"""
import numpy as np
import pytest

from nqpu_b200 import _lib, circuits
from nqpu_b200.state import Circuit, StateVector
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def unitary(rng, d):
    q, r = np.linalg.qr(rng.normal(size=(d, d)) + 1j * rng.normal(size=(d, d)))
    return q * (np.diag(r) / np.abs(np.diag(r)))


def mixed(rng, n, count, names, qubits=None):
    gates = [("u3", (q,), tuple(rng.uniform(0, 6, 3))) for q in range(n)]
    for _ in range(count):
        name = names[int(rng.integers(len(names)))]
        qs = tuple(int(x) for x in rng.choice(qubits or n, size=circuits.ARITY[name], replace=False))
        d = {"custom1": 2, "custom2": 4}.get(name)
        gates.append((name, qs, (), unitary(rng, d)) if d else (name, qs, tuple(rng.uniform(-6, 6, 4))))
    return gates


EVERY = [k for k in circuits.ARITY if k != "u2lo"]


def check(n, dtype, gates, mode):
    with StateVector(n, dtype) as sv:
        Circuit(n, gates).execute(sv, mode)
        got = sv.amplitudes()
    o = O.OracleState(n)
    o.apply(gates)
    ref = o.amplitudes()
    if dtype == "c128":
        assert np.abs(got - ref).max() <= 1e-12
    assert 1 - abs(np.vdot(got, ref)) ** 2 / (np.vdot(got, got).real * np.vdot(ref, ref).real) <= 1e-5


# one CTA with most of the SM's shared memory; programs beyond it (1500 4x4s of 144
# bytes, 800 of 272); one tile per SM and, from 20 qubits on, several; complex64
# on 13-bit tiles from 22 qubits
@pytest.mark.parametrize("n,dtype,count,names,qubits", [
    (8, "c64", 200, EVERY, None), (8, "c128", 200, EVERY, None),
    (8, "c64", 1500, ["custom2"], 4), (8, "c128", 800, ["custom2"], 4),
    (18, "c64", 100, ["cu", "crx", "cry", "h"], None), (18, "c128", 100, ["cu", "crx", "cry", "h"], None),
    (19, "c128", 150, EVERY, None), (20, "c128", 150, EVERY, None), (21, "c64", 150, EVERY, None)])
def test_tiled(n, dtype, count, names, qubits):
    check(n, dtype, mixed(np.random.default_rng(n), n, count, names, qubits), "tiled")


@pytest.mark.parametrize("n", [21, 22])
def test_wide_tiles(n):
    prep = [("u3", (q,), (0.3 + q, 0.2 * q, 1.0)) for q in range(n)]
    check(n, "c64", prep + circuits.qft(n), "tiled")


@pytest.mark.parametrize("dtype", ["c64", "c128"])
def test_pergate_sweeps(dtype):
    check(21, dtype, mixed(np.random.default_rng(5), 21, 15, EVERY), "pergate")


# more outcomes than one queue holds; complex64 pairs share a vector at qubit 0
@pytest.mark.parametrize("dtype", ["c64", "c128"])
def test_many_outcomes(dtype):
    gates = []
    for i in range(1100):
        gates += [("ry", (i % 3,), (0.7 + 0.001 * i,)), ("cx", (i % 3, (i + 1) % 3), ()),
                  ("reset" if i % 4 == 3 else "measure", ((i + i // 5) % 3,), ())]
    with StateVector(3, dtype) as sv:
        _lib.load().nqpu_set_seed(77)
        got = Circuit(3, gates).execute_measured(sv, "tiled")
        amps = sv.amplitudes()
    o = O.OracleState(3)
    O.set_seed(77)
    o.apply(gates)
    np.testing.assert_array_equal(got, o.take_outcomes())
    assert np.abs(amps - o.amplitudes()).max() <= (1e-5 if dtype == "c64" else 1e-12)


# shots beyond what the pinned buffer holds
@pytest.mark.parametrize("shots", [2016, 2017, 5000])
def test_many_shots(shots):
    rng = np.random.default_rng(shots)
    a = rng.normal(size=4096) + 1j * rng.normal(size=4096)
    a /= np.linalg.norm(a)
    p = np.abs(a) ** 2
    pick = rng.integers(4096, size=shots)
    u = np.cumsum(p)[pick] - 0.5 * p[pick]
    pick, u = pick[p[pick] > 1e-9], u[p[pick] > 1e-9]
    with StateVector(12, "c128") as sv:
        sv.set_amplitudes(a)
        np.testing.assert_array_equal(sv.sample_with_uniforms(u), pick.astype(np.uint64))


# A gate without a diagonal moves amplitudes and turns their phases: a small one keeps
# its digits beside a large one.  Per amplitude: 2^-22 (complex64: entries, a phase and
# the state's own rounding, 2^-24 each) and 2^-50 of its own size.
@pytest.mark.parametrize("n", [5, 9, 14])
@pytest.mark.parametrize("dtype,gate", [
    ("c64", ("y", ())), ("c64", ("rx", (np.pi,))), ("c64", ("ry", (np.pi,))), ("c64", ("u3", (np.pi, 0.4, 0.9))),
    ("c128", ("y", ())), ("c128", ("custom1", ()))])
def test_exchanged_amplitudes_keep_their_digits(n, dtype, gate):
    name, params = gate
    rng = np.random.default_rng(n)
    a = np.exp(2j * np.pi * rng.random(1 << n)) * 10.0 ** -rng.integers(0, 9, 1 << n)
    a = a.astype(np.complex64 if dtype == "c64" else np.complex128).astype(np.complex128)
    m = {"y": [[0, -1j], [1j, 0]], "rx": [[0, -1j], [-1j, 0]], "ry": [[0, -1], [1, 0]],
         "u3": [[0, -np.exp(0.9j)], [np.exp(0.4j), 0]], "custom1": [[0, np.exp(0.3j)], [np.exp(-1.1j), 0]]}[name]
    for q in {0, 2, n - 1}:
        g = (name, (q,), params) if name != "custom1" else (name, (q,), (), np.array(m))
        with StateVector(n, dtype) as sv:
            sv.set_amplitudes(a)
            Circuit(n, [g]).execute(sv, "tiled")
            got = sv.amplitudes()
        v = a.reshape(-1, 2, 1 << q)
        want = np.stack([m[0][1] * v[:, 1], m[1][0] * v[:, 0]], axis=1).reshape(-1)
        assert (np.abs(got - want) <= (2.0 ** -20 if dtype == "c64" else 2.0 ** -49) * np.abs(want)).all()
