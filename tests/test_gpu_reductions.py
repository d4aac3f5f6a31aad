"""Reductions at the edges of their launch shapes, against plain numpy in FP64.

All sums run in FP64 over at most 2^23 values in trees and compensated
accumulators; numpy's pairwise sum of the same values is good to a few 2^-53 of
the sum of magnitudes, and 1e-13 of it leaves two orders of room for either.
"""
import numpy as np
import pytest

from nqpu_b200.state import StateVector

pytestmark = pytest.mark.gpu


def random_state(n, dtype, seed):
    rng = np.random.default_rng(seed)
    a = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    a *= rng.random(1 << n) < 0.7  # some zero amplitudes
    a[0] = 1.0
    a /= np.linalg.norm(a)
    a = a.astype(np.complex64 if dtype == "c64" else np.complex128).astype(np.complex128)
    sv = StateVector(n, dtype)
    sv.set_amplitudes(a)
    return a, sv


# one chunk and less, one block, the step to several blocks, the full grid
@pytest.mark.parametrize("dtype", ["c64", "c128"])
@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 10, 13, 14, 15, 16, 20, 22])
def test_z_and_fidelity(n, dtype):
    a, sv = random_state(n, dtype, n)
    p = np.abs(a) ** 2
    idx = np.arange(1 << n)
    want = [p[(idx >> q) & 1 == 0].sum() - p[(idx >> q) & 1 == 1].sum() for q in range(n)]
    np.testing.assert_allclose(sv.expectation_z_all(), want, rtol=0, atol=1e-13)
    for other in ("c64", "c128"):
        b, sb = random_state(n, other, n + 100)
        assert abs(sv.fidelity(sb) - abs(np.vdot(a, b)) ** 2) <= 1e-13
        sb.close()
    sv.close()


# less than a segment, one segment, several, more than one tile of the scan
@pytest.mark.parametrize("dtype", ["c64", "c128"])
@pytest.mark.parametrize("n", [1, 2, 8, 9, 11, 12, 13, 18])
def test_sample_picks_the_bin(n, dtype):
    a, sv = random_state(n, dtype, n)
    p = np.abs(a) ** 2
    cum = np.cumsum(p)
    rng = np.random.default_rng(n)
    pick = np.concatenate([[0], rng.choice(np.nonzero(p)[0], size=500)])
    u = cum[pick] - 0.5 * p[pick]  # the middle of the bin: 1e-9 from its edges at least
    pick, u = pick[p[pick] > 1e-9], u[p[pick] > 1e-9]
    np.testing.assert_array_equal(sv.sample_with_uniforms(u), pick.astype(np.uint64))
    np.testing.assert_array_equal(sv.sample_with_uniforms([1.0 - 1e-17, 2.0]), [(1 << n) - 1] * 2)
    sv.close()


def pauli_value(a, s):
    n = len(s)
    idx = np.arange(1 << n)
    x = sum(1 << q for q in range(n) if s[q] in "XY")
    z = sum(1 << q for q in range(n) if s[q] in "ZY")
    par = idx & z
    for sh in (16, 8, 4, 2, 1):
        par = par ^ (par >> sh)
    v = np.conj(a) * (1 - 2 * (par & 1)) * a[idx ^ x]
    return float((1j ** s.count("Y") * v.sum()).real)


def random_strings(rng, n, count):
    out = []
    for i in range(count):
        w = int(rng.integers(0, min(n, 7) + 1))
        s = ["I"] * n
        for q in rng.choice(n, size=w, replace=False):
            s[q] = "XYZ"[int(rng.integers(3))]
        out.append("".join(s))
    return out


# fewer qubits than a register set, less than a unit of work, several chunks;
# 900 strings need more table than the small buffers hold
@pytest.mark.parametrize("dtype", ["c64", "c128"])
@pytest.mark.parametrize("n,count", [(1, 8), (3, 20), (4, 60), (5, 60), (8, 900), (11, 60), (12, 60), (13, 60), (23, 12)])
def test_pauli_sum(n, count, dtype):
    a, sv = random_state(n, dtype, n)
    rng = np.random.default_rng(n)
    strings = random_strings(rng, n, count) + ["I" * n, "Z" * n, "Y" + "Z" * (n - 1), "I" * (n - 1) + "X"]
    c = rng.normal(size=len(strings))
    want = np.array([pauli_value(a, s) for s in strings])
    scale = np.abs(c).sum()
    assert abs(sv.expectation_pauli_sum(list(zip(c, strings))) - c @ want) <= 1e-13 * scale
    for s, w in list(zip(strings, want))[-6:]:
        assert abs(sv.expectation_pauli_string(s) - w) <= 1e-13
    assert abs(sv.expectation_x(n - 1) - want[-1]) <= 1e-13
    sv.close()


# finite coefficients whose double or sum is not, and ones whose share of an
# amplitude would be subnormal; the sum is scaled exactly, so the bound is that of
# coefficients near 1
@pytest.mark.parametrize("dtype", ["c64", "c128"])
@pytest.mark.parametrize("n", [2, 5, 13])
@pytest.mark.parametrize("size", [1.7e308, 1e305, 1e-303])
def test_pauli_sum_of_extreme_coefficients(size, n, dtype):
    a, sv = random_state(n, dtype, n)
    strings = ["X" + "I" * (n - 1), "Z" * n, "Y" + "Z" * (n - 1), "I" * (n - 1) + "Z", "ZZ" + "I" * (n - 2)]
    unit = np.array([1.0, 0.9, -0.8, 0.7, 0.6])
    want = unit @ np.array([pauli_value(a, s) for s in strings])
    assert abs(want) < 1.05  # and 1.05 * 1.7e308 is finite
    got = sv.expectation_pauli_sum(list(zip(unit * size, strings)))
    assert abs(got / size - want) <= 1e-13 * unit.size
    sv.close()


# many shots: one row and less, each number of rows of a single step, several steps,
# several segments.  The middle of a bin of at least 1e-9 is far from any rounding.
@pytest.mark.parametrize("dtype", ["c64", "c128"])
@pytest.mark.parametrize("n", [1, 2, 5, 6, 7, 8, 9, 10, 12, 13, 18])
def test_many_shots_pick_the_bin(n, dtype):
    a, sv = random_state(n, dtype, n)
    p = np.abs(a) ** 2
    cum = np.cumsum(p)
    pick = np.random.default_rng(n).choice(np.nonzero(p > 1e-9)[0], size=4000)
    u = cum[pick] - 0.5 * p[pick]
    np.testing.assert_array_equal(sv.sample_with_uniforms(u), pick.astype(np.uint64))
    beyond = np.full(2017, 2.0)
    np.testing.assert_array_equal(sv.sample_with_uniforms(beyond), [(1 << n) - 1] * 2017)
    sv.close()


def test_many_shots_read_whole_lines():
    # both types read a segment's vectors alike: complex128, twice the bytes, takes
    # little longer (1.7 times as long with eight consecutive vectors per lane)
    import time

    best = {}
    u = np.random.default_rng(0).random(100000)
    for dtype in ("c64", "c128"):
        _, sv = random_state(13, dtype, 13)
        times = []
        for _ in range(10):
            t = time.perf_counter()
            sv.sample_with_uniforms(u)
            times.append(time.perf_counter() - t)
        best[dtype] = min(times)
        sv.close()
    assert best["c128"] <= 1.3 * best["c64"]


# strings on the lowest qubits of a large complex128 state, alone, two in one set, and
# among others; every value against numpy
def test_pauli_strings_on_the_lowest_qubits():
    n = 23
    a, sv = random_state(n, "c128", n)

    def on(**q):
        return "".join(q.get(f"q{i}", "I") for i in range(n))

    strings = [on(q0="X", q1="X", q2="X"), on(q0="X", q1="Y", q2="Y", q9="Z"), on(q0="Y", q1="X", q2="X", q20="X"),
               on(q5="X", q6="Y"), on(q0="Z", q22="Z"), on(q0="X", q1="X", q2="Y", q3="Z")]
    want = np.array([pauli_value(a, s) for s in strings])
    for s, w in zip(strings, want):
        assert abs(sv.expectation_pauli_string(s) - w) <= 1e-13
    c = np.array([0.3, -1.2, 0.8, 0.5, -0.9, 1.1])
    for k in range(2, 7):
        assert abs(sv.expectation_pauli_sum(list(zip(c[:k], strings[:k]))) - c[:k] @ want[:k]) <= 1e-13 * np.abs(c).sum()
    sv.close()


def test_a_string_on_the_lowest_qubits_takes_no_longer():
    import time

    n = 25
    best = []
    with StateVector(n, "c128") as sv:
        for s in ("XXX" + "I" * (n - 3), "IIIXXX" + "I" * (n - 6)):
            times = []
            for _ in range(20):
                t = time.perf_counter()
                sv.expectation_pauli_string(s)
                times.append(time.perf_counter() - t)
            best.append(min(times))
    assert best[0] <= 1.25 * best[1]  # 1.5 times as long from a register set
