"""Timed cases of the engine: what its users run, through the public entry points.

Every case is a dict of plain values; its "kind" names what a program does:

  evolve   reset a state, execute a circuit on it, read all <Z_i> (and shots, or
           the whole statevector of a small register)
  energy   <H> of an Ising Hamiltonian as a Pauli sum, on a state in hand
  readout  all <Z_i>, the fidelity with a second state, and shots
  measured a circuit with mid-circuit measurements and resets
  gates    a circuit applied gate by gate (one call per gate)
  batch    many ansatz circuits of mixed sizes in one launch, <H> of each

Angles, fields and amplitudes come from the seed; sizes, gate sequences and
options from the case.  What is read from a complex64 state after it has been
evolved is kept in single precision, as the state is; what is reduced from
amplitudes in hand is FP64 throughout.
"""
import ctypes
import math

import numpy as np
import torch

import nqpu_b200
from nqpu_b200 import circuits
from nqpu_b200.batch import Batch, ising_terms
from nqpu_b200.state import Circuit, StateVector

DEV = "cuda" if torch.cuda.is_available() else "cpu"


def listed():
    return [
        # a small register, read out whole: a notebook or the inner loop of a
        # variational search, where launches and latency are all there is
        {"name": "small_hea10_c128", "kind": "evolve", "circuit": "hea", "n": 10, "layers": 4, "dtype": "c128",
         "mode": "tiled", "shots": 0, "whole": True},
        # a mid-size register of odd size in the engine's own mode choice (the
        # middle of the serving mix: 8-28 qubits, depth 10-50)
        {"name": "mid_brick17_c64", "kind": "evolve", "circuit": "brickwork", "n": 17, "layers": 15, "dtype": "c64",
         "mode": "auto", "shots": 0, "whole": False},
        # the 20-qubit complex128 brickwork, 20 layers, all <Z_i> and 1000 shots
        {"name": "brick20_c128_shots", "kind": "evolve", "circuit": "brickwork", "n": 20, "layers": 20, "dtype": "c128",
         "mode": "tiled", "shots": 1000, "whole": False},
        # an ansatz on a larger register in the default type
        {"name": "hea25_c128", "kind": "evolve", "circuit": "hea", "n": 25, "layers": 6, "dtype": "c128",
         "mode": "tiled", "shots": 0, "whole": False},
        # random circuit on a register well beyond the L2
        {"name": "brick26_c64", "kind": "evolve", "circuit": "brickwork", "n": 26, "layers": 12, "dtype": "c64",
         "mode": "auto", "shots": 0, "whole": False},
        # phase estimation: a phase state through the Fourier transform
        {"name": "qpe27_c64", "kind": "evolve", "circuit": "qpe", "n": 27, "layers": 1, "dtype": "c64",
         "mode": "auto", "shots": 0, "whole": False},
        # Trotterised transverse-field Ising evolution between two recordings
        # (every 10 steps) on a large register
        {"name": "tfim30_c64", "kind": "evolve", "circuit": "tfim", "n": 30, "layers": 10, "dtype": "c64",
         "mode": "auto", "shots": 0, "whole": False},
        # the energy of a variational state, 2n - 1 Pauli terms
        {"name": "energy24_c64", "kind": "energy", "n": 24, "dtype": "c64"},
        # what a finished run is read for, states in hand
        {"name": "readout25_c64", "kind": "readout", "n": 25, "dtype": "c64", "shots": 1024},
        # syndrome-like measurements and resets between layers
        {"name": "measured21_c128", "kind": "measured", "n": 21, "layers": 4, "mids": 6, "dtype": "c128",
         "mode": "tiled"},
        # the per-gate interface, one launch over the state per gate
        {"name": "gates24_c64", "kind": "gates", "n": 24, "layers": 1, "dtype": "c64"},
        # ansatz batch with the Hamiltonians of its circuits (10-20 qubits, 2-12 layers)
        {"name": "batch256", "kind": "batch", "count": 256, "nmin": 10, "nmax": 20},
    ]


def draw(rng):
    kind = rng.choice(["evolve"] * 6 + ["energy", "energy", "readout", "readout", "measured", "gates", "batch"])
    dtype = rng.choice(["c64", "c128"])
    if kind == "evolve":
        circuit = rng.choice(["hea", "brickwork", "qpe", "tfim"])
        n = rng.randint(6, 29 if dtype == "c64" else 26)
        layers = rng.randint(2, 12) if n > 22 else rng.randint(2, 24)
        if circuit == "tfim":
            layers = min(layers, 10)
        mode = "tiled" if dtype == "c128" else rng.choice(["auto", "auto", "tiled"])
        whole = n <= 12 and dtype == "c128" and rng.random() < 0.5
        shots = 0
        if dtype == "c128" and not whole and rng.random() < 0.5:
            shots = int(round(2 ** rng.uniform(6, 13)))
        return {"kind": kind, "circuit": circuit, "n": n, "layers": 1 if circuit == "qpe" else layers,
                "dtype": dtype, "mode": mode, "shots": shots, "whole": whole}
    if kind == "energy":
        return {"kind": kind, "n": rng.randint(8, 25 if dtype == "c64" else 24), "dtype": dtype}
    if kind == "readout":
        return {"kind": kind, "n": rng.randint(8, 25 if dtype == "c64" else 24), "dtype": dtype,
                "shots": int(round(2 ** rng.uniform(4, 17)))}
    if kind == "measured":
        return {"kind": kind, "n": rng.randint(6, 24), "layers": rng.randint(2, 6), "mids": rng.randint(1, 8),
                "dtype": dtype, "mode": "tiled" if dtype == "c128" else "auto"}
    if kind == "gates":
        return {"kind": kind, "n": rng.randint(4, 26), "layers": rng.randint(1, 4), "dtype": dtype}
    nmin = rng.randint(6, 14)
    return {"kind": kind, "count": int(round(2 ** rng.uniform(4, 9))), "nmin": nmin, "nmax": rng.randint(nmin, 20)}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------

def gate_list(case, seed):
    """The circuit of an evolve or gates case."""
    n, layers = case["n"], case["layers"]
    kind = case.get("circuit", "brickwork")
    if kind == "brickwork":
        return circuits.brickwork(n, layers, seed)
    if kind == "hea":
        return circuits.hea(n, layers, np.random.default_rng(seed))
    if kind == "tfim":
        return circuits.tfim_trotter(n, layers, seed)[0]
    # phase estimation: the register holds sum_k exp(-2 pi i phi k) |k>, which the
    # Fourier transform turns into a peak at phi 2^n
    phi = float(np.random.default_rng(seed).random())
    gates = []
    for q in range(n):
        gates.append(("h", (q,), ()))
        gates.append(("p", (q,), (-2.0 * math.pi * math.fmod(phi * 2.0 ** q, 1.0),)))
    return gates + circuits.qft(n)


def measured_list(case, seed):
    """Layers of a brickwork with measurements and resets after each; none last."""
    n, layers, mids = case["n"], case["layers"], case["mids"]
    rng = np.random.default_rng([seed, 1])
    body = circuits.brickwork(n, layers, seed)
    per = len(body) // layers
    gates = []
    for i in range(layers):
        gates += body[i * per:(i + 1) * per if i + 1 < layers else len(body)]
        if i + 1 < layers:
            for j in range(mids // (layers - 1) + (i < mids % (layers - 1))):
                gates.append(("reset" if j % 3 == 2 else "measure", (int(rng.integers(n)),), ()))
    return gates


def start_index(case):
    return circuits.neel_index(case["n"]) if case.get("circuit") == "tfim" else 0


def amplitudes(n, seed, dtype):
    """A correlated state with expectation values of order one: a product state
    with random angles, every amplitude turned by a random phase."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    rng = np.random.default_rng([seed, 2])
    psi = torch.ones(1, dtype=torch.complex128, device=DEV)
    for q in range(n):
        th, ph = math.pi * rng.random(), 2.0 * math.pi * rng.random()
        one = torch.tensor([math.cos(th / 2), math.sin(th / 2) * complex(math.cos(ph), math.sin(ph))],
                           dtype=torch.complex128, device=DEV)
        psi = torch.kron(one, psi)
    psi *= torch.exp(0.5j * torch.randn(psi.numel(), generator=g, device=DEV, dtype=torch.float64))
    return psi.to(torch.complex64 if dtype == "c64" else torch.complex128)


def state_of(n, seed, dtype):
    sv = StateVector(n, dtype)
    sv.set_amplitudes(amplitudes(n, seed, dtype).cpu().numpy())
    return sv


def hamiltonian(n, seed):
    return circuits.ising_hamiltonian(n, np.random.default_rng([seed, 3]))


def batch_items(case, seed):
    return circuits.hea_batch(case["count"], seed, nmin=case["nmin"], nmax=case["nmax"], arrays=True)


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "evolve":
        s["state"] = StateVector(case["n"], case["dtype"])
        s["circuit"] = Circuit(case["n"], gate_list(case, seed))
        s["uniforms"] = np.random.default_rng([seed, 4]).random(case["shots"])
    elif kind == "energy":
        s["state"] = state_of(case["n"], seed, case["dtype"])
        s["terms"] = ising_terms(case["n"], *hamiltonian(case["n"], seed))
    elif kind == "readout":
        s["state"] = state_of(case["n"], seed, case["dtype"])
        other = amplitudes(case["n"], seed, case["dtype"])
        other[1::3] *= 0.9j
        s["other"] = StateVector(case["n"], case["dtype"])
        s["other"].set_amplitudes(other.cpu().numpy())
        s["uniforms"] = np.random.default_rng([seed, 4]).random(case["shots"])
    elif kind == "measured":
        s["state"] = StateVector(case["n"], case["dtype"])
        s["circuit"] = Circuit(case["n"], measured_list(case, seed))
        s["seed"] = seed + 1
    elif kind == "gates":
        s["state"] = StateVector(case["n"], case["dtype"])
        s["gates"] = gate_list(case, seed)
    else:
        s["batch"] = Batch()
        s["batch"].add_ising_arrays(batch_items(case, seed))
        s["batch"].prepare()
    return s


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------

def z_values(state, case):
    z = state.expectation_z_all()
    return z.astype(np.float32) if case["dtype"] == "c64" else z


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "evolve":
        state = s["state"]
        state.set_basis(start_index(case))
        s["circuit"].execute(state, case["mode"])
        out = {"z": z_values(state, case)}
        if case["whole"]:
            out["amplitudes"] = state.amplitudes()
        if case["shots"]:
            out["shots"] = state.sample_with_uniforms(s["uniforms"])
        return out
    if kind == "energy":
        return {"energy": s["state"].expectation_pauli_sum(s["terms"])}
    if kind == "readout":
        state = s["state"]
        return {"z": state.expectation_z_all(), "fidelity": state.fidelity(s["other"]),
                "shots": state.sample_with_uniforms(s["uniforms"])}
    if kind == "measured":
        state = s["state"]
        state.reset()
        nqpu_b200.load().nqpu_set_seed(ctypes.c_uint64(s["seed"]))
        outcomes = s["circuit"].execute_measured(state, case["mode"])
        return {"outcomes": outcomes, "z": z_values(state, case)}
    if kind == "gates":
        state = s["state"]
        state.reset()
        state.apply_gates(s["gates"])
        return {"z": z_values(state, case)}
    # the batch's states are complex64
    return {"energies": s["batch"].run().astype(np.float32)}


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------

def work(case):
    kind = case["kind"]
    if kind == "batch":
        states = flops = 0
        for n, (codes, _, _), _, _ in batch_items(case, 0):
            names = {v: k for k, v in circuits.GATE_CODES.items()}
            flops += circuits.algorithmic_flops([(names[int(c)],) for c in codes], n)
            states += 8 << n
        return {"bytes": states, "flops": flops}
    size = (8 if case["dtype"] == "c64" else 16) << case["n"]
    if kind == "energy":  # the state read once; n - 1 bonds from |a|^2 and n overlaps of a pair
        return {"bytes": size, "flops": (4 + 4 * case["n"]) << case["n"]}
    if kind == "readout":  # both states read once
        return {"bytes": 2 * size, "flops": 12 << case["n"]}
    # the state written once; the circuit's gates
    gates = measured_list(case, 0) if kind == "measured" else gate_list(case, 0)
    return {"bytes": size, "flops": circuits.algorithmic_flops([g for g in gates if g[0] not in circuits.MID_GATES],
                                                               case["n"])}


# ---------------------------------------------------------------------------
# The same results in 64 bits, in plain torch
# ---------------------------------------------------------------------------

def matrix_of(name, p):
    if name == "u3":
        c, s = math.cos(p[0] / 2), math.sin(p[0] / 2)
        return [[c, -s * complex(math.cos(p[2]), math.sin(p[2]))],
                [s * complex(math.cos(p[1]), math.sin(p[1])), c * complex(math.cos(p[1] + p[2]), math.sin(p[1] + p[2]))]]
    if name == "h":
        return [[math.sqrt(0.5), math.sqrt(0.5)], [math.sqrt(0.5), -math.sqrt(0.5)]]
    c, s = math.cos(p[0] / 2), math.sin(p[0] / 2)
    if name == "rx":
        return [[c, -1j * s], [-1j * s, c]]
    return [[c, -s], [s, c]]  # ry


def apply_gate(psi, n, g):
    name, qs, p = g[0], g[1], g[2]
    if len(qs) == 1:
        v = psi.view(-1, 2, 1 << qs[0])
        a, b = v[:, 0], v[:, 1]
        if name == "rz":
            a *= complex(math.cos(p[0] / 2), -math.sin(p[0] / 2))
            b *= complex(math.cos(p[0] / 2), math.sin(p[0] / 2))
        elif name == "p":
            b *= complex(math.cos(p[0]), math.sin(p[0]))
        else:
            m = matrix_of(name, p)
            new = m[0][0] * a
            new += m[0][1] * b
            b *= m[1][1]
            b += m[1][0] * a
            a.copy_(new)
        return
    lo, hi = min(qs), max(qs)
    v = psi.view(-1, 2, 1 << (hi - lo - 1), 2, 1 << lo)

    def part(bits):  # bits of (qs[0], qs[1])
        b = dict(zip(qs, bits))
        return v[:, b[hi], :, b[lo]]

    if name == "cz":
        part((1, 1)).neg_()
    elif name == "cp":
        part((1, 1)).mul_(complex(math.cos(p[0]), math.sin(p[0])))
    elif name == "rzz":
        e = complex(math.cos(p[0] / 2), math.sin(p[0] / 2))
        for bits in ((0, 0), (0, 1), (1, 0), (1, 1)):
            part(bits).mul_(e if bits[0] != bits[1] else e.conjugate())
    else:  # cx, swap
        x, y = (part((1, 0)), part((1, 1))) if name == "cx" else (part((0, 1)), part((1, 0)))
        t = x.clone()
        x.copy_(y)
        y.copy_(t)


def probabilities(psi):
    p = torch.view_as_real(psi).square_()  # in place: the amplitudes are not needed again
    return p[..., 0].add_(p[..., 1])


def z_of(prob, n):
    """All <Z_i>; folds the register qubit by qubit from the top."""
    out = []
    p = prob
    for _ in range(n):
        h = p.numel() // 2
        out.append((p[:h].sum() - p[h:].sum()))
        p = p[:h] + p[h:]
    return torch.stack(out[::-1]).cpu().numpy()


def basis(n, index):
    psi = torch.zeros(1 << n, dtype=torch.complex128, device=DEV)
    psi[index] = 1
    return psi


def exact_measured(case, seed):
    n = case["n"]
    rng = seed + 1  # the thread-local xorshift64* of nqpu_set_seed
    psi = basis(n, 0)
    outcomes = []
    for g in measured_list(case, seed):
        if g[0] not in circuits.MID_GATES:
            apply_gate(psi, n, g)
            continue
        rng ^= rng >> 12
        rng ^= (rng << 25) & (2 ** 64 - 1)
        rng ^= rng >> 27
        r = ((rng * 0x2545F4914F6CDD1D) % 2 ** 64 >> 11) / 2.0 ** 53
        v = psi.view(-1, 2, 1 << g[1][0])
        p0 = float(torch.view_as_real(v[:, 0]).square().sum())
        k = 0 if r < p0 else 1
        v[:, 1 - k] = 0
        v[:, k] *= 1.0 / math.sqrt(p0 if k == 0 else 1.0 - p0)
        if g[0] == "measure":
            outcomes.append(k)
        elif k == 1:
            v[:, 0] = v[:, 1]
            v[:, 1] = 0
    return {"outcomes": np.array(outcomes, dtype=np.uint32), "z": z_of(probabilities(psi), n)}


def exact_energy(psi, n, J, h):
    """sum_i J_i <Z_i Z_{i+1}> + sum_i h_i <X_i>"""
    e = 0.0
    for q in range(n):
        v = psi.view(-1, 2, 1 << q)
        a, b = v[:, 0].reshape(-1), v[:, 1].reshape(-1)
        e += 2.0 * float(h[q]) * float(torch.vdot(a, b).real)
    p = probabilities(psi)
    for q in range(n - 1):
        v = p.view(-1, 2, 2, 1 << q)
        e += float(J[q]) * float((v[:, 0, 0] + v[:, 1, 1] - v[:, 0, 1] - v[:, 1, 0]).sum())
    return e


def exact_batch(case, seed):
    names = {v: k for k, v in circuits.GATE_CODES.items()}
    signs = {}
    out = []
    for n, (codes, qs, ps), J, h in batch_items(case, seed):
        if n not in signs:  # the CZ ladder as one diagonal
            i = torch.arange(1 << n, device=DEV)
            m = i & (i >> 1)
            odd = torch.zeros_like(m)
            for q in range(n):
                odd ^= (m >> q) & 1
            signs[n] = (1 - 2 * odd).to(torch.float64)
        psi = basis(n, 0)
        per = 3 * n - 1
        for k in range(len(codes) // per):
            for j in range(k * per, k * per + 2 * n, 2):
                th, ph = float(ps[j, 0]), float(ps[j + 1, 0])
                assert names[int(codes[j])] == "ry" and names[int(codes[j + 1])] == "rz"
                m = torch.tensor(matrix_of("ry", (th,)), dtype=torch.complex128)
                m *= torch.tensor([[complex(math.cos(ph / 2), -math.sin(ph / 2))],
                                   [complex(math.cos(ph / 2), math.sin(ph / 2))]])
                v = psi.view(-1, 2, 1 << int(qs[j, 0]))
                psi = torch.matmul(m.to(DEV), v).reshape(-1)
            psi = psi * signs[n]
        out.append(exact_energy(psi, n, J, h))
    return {"energies": np.array(out)}


def exact(case, seed):
    kind, n = case["kind"], case.get("n", 0)
    if kind == "batch":
        return exact_batch(case, seed)
    if kind == "measured":
        return exact_measured(case, seed)
    if kind == "energy":
        psi = amplitudes(n, seed, case["dtype"]).to(torch.complex128)
        return {"energy": exact_energy(psi, n, *hamiltonian(n, seed))}
    if kind == "readout":
        psi = amplitudes(n, seed, case["dtype"])
        other = psi.clone()
        other[1::3] *= 0.9j
        psi, other = psi.to(torch.complex128), other.to(torch.complex128)
        f = float(torch.vdot(psi, other).abs().square())
        return {"z": z_of(probabilities(psi), n), "fidelity": f, "shots": None}
    psi = basis(n, start_index(case))
    for g in gate_list(case, seed):
        apply_gate(psi, n, g)
    out = {}
    if case.get("whole"):
        out["amplitudes"] = psi.cpu().numpy().copy()
    if case.get("shots"):
        out["shots"] = None
    out["z"] = z_of(probabilities(psi), n)
    return out
