"""The work that users of this framework have it do, as measurable cases.

Each case goes through a public entry point (the `quantum_sim_v3` module, `llgpu.State`,
`llgpu.Adjoint`, `llgpu.Traj`, `llgpu.Batch`, `llgpu.DensityMatrix`) and returns everything that
call gives back: whole states, energies with their gradients, every trajectory's result.  Sizes
are those of the benchmark's five configurations and of the tests, with smaller and ragged ones
between them.

`listed()` has the named cases, `draw(rng)` more of the same ranges, `prepare` / `run` a user's
program, `work` the bytes and operations that one pass cannot do without, and `exact` the results
in 64 bits from plain torch and numpy.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lightning-lite-quantum-simulator_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

TWO_PI = 2.0 * math.pi


# ---------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------
def listed():
    return [
        # one energy of a small variational circuit, as an optimiser asks for it thousands of times:
        # all latency (launches, planning, the readback of one number)
        {"name": "energy_hea_8q", "kind": "energy", "ansatz": "hea", "n": 8, "layers": 3, "precision": "complex128"},
        # an energy of a QAOA circuit on a register that fills the GPU, the state stays on the device
        {"name": "energy_qaoa_23q", "kind": "energy", "ansatz": "qaoa", "n": 23, "layers": 2, "precision": "complex128"},
        # the published Lightning-Lite workload: 12 qubits, 1000 H / CNOT gates, amplitudes read back
        {"name": "h_cnot_12q", "kind": "circuit", "circuit": "h_cnot", "n": 12, "layers": 1000, "precision": "complex128"},
        # layered rotations with a CNOT brickwork (the headline circuit) on an odd, small register
        {"name": "layered_17q", "kind": "circuit", "circuit": "layered", "n": 17, "layers": 20, "precision": "complex128"},
        # the same on an ordinary register
        {"name": "layered_22q", "kind": "circuit", "circuit": "layered", "n": 22, "layers": 20, "precision": "complex128"},
        # the same at its largest here: 2 GiB of amplitudes, all twenty layers
        {"name": "layered_27q", "kind": "circuit", "circuit": "layered", "n": 27, "layers": 20, "precision": "complex128"},
        # the opt-in formats on large registers: pairs of floats, and complex64
        {"name": "layered_24q_df64", "kind": "circuit", "circuit": "layered", "n": 24, "layers": 20, "precision": "df64"},
        {"name": "layered_25q_c64", "kind": "circuit", "circuit": "layered", "n": 25, "layers": 12, "precision": "complex64"},
        # training a variational circuit: energies and all gradients of a batch of parameter sets
        {"name": "adjoint_hea_20q", "kind": "adjoint", "n": 20, "layers": 10, "batch": 8, "precision": "complex128"},
        # a noisy-circuit ensemble: amplitude and phase damping after every gate
        {"name": "traj_14q", "kind": "traj", "n": 14, "layers": 8, "ntraj": 512, "precision": "complex128"},
        # many circuits of uneven sizes in one launch, all their states read back
        {"name": "mixed_batch_10_18q", "kind": "batch", "lo": 10, "hi": 18, "count": 36, "depth": 200, "precision": "complex128"},
        # a density matrix through a noisy circuit: gates, damping on every qubit, two-qubit
        # depolarizing, the whole matrix read back
        {"name": "density_11q", "kind": "density", "n": 11, "layers": 2, "precision": "complex128"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    precision = rng.choice(["complex128"] * 5 + ["df64", "complex64"])
    kind = rng.choice(["energy", "energy", "circuit", "circuit", "circuit", "circuit", "adjoint", "traj", "batch", "density"])
    if kind == "energy":
        n = rng.randint(4, 25)
        return {"kind": kind, "ansatz": rng.choice(["hea", "qaoa"]), "n": n, "layers": rng.randint(1, 4 if n > 20 else 8),
                "precision": precision}
    if kind == "circuit":
        if rng.random() < 0.3:
            return {"kind": kind, "circuit": "h_cnot", "n": rng.randint(5, 24), "layers": _log_int(rng, 20, 1000),
                    "precision": precision}
        n = rng.randint(6, 27)
        return {"kind": kind, "circuit": "layered", "n": n, "layers": _log_int(rng, 1, 20), "precision": precision}
    if kind == "adjoint":
        n = rng.randint(6, 20)
        return {"kind": kind, "n": n, "layers": rng.randint(1, 10), "batch": rng.randint(1, 8), "precision": precision}
    if kind == "traj":
        return {"kind": kind, "n": rng.randint(6, 14), "layers": rng.randint(1, 8), "ntraj": _log_int(rng, 40, 600),
                "precision": precision}
    if kind == "batch":
        lo = rng.randint(6, 12)
        return {"kind": kind, "lo": lo, "hi": lo + rng.randint(2, 7), "count": rng.randint(5, 48),
                "depth": _log_int(rng, 40, 300), "precision": precision}
    return {"kind": kind, "n": rng.randint(4, 12), "layers": rng.randint(1, 3), "precision": precision}


# ---------------------------------------------------------------------------------------------
# the circuits: lists of (gate, q0, q1, angle, parameter)
# ---------------------------------------------------------------------------------------------
def _layered(n, layers, rng):
    g = []
    for layer in range(layers):
        for q in range(n):
            for name in ("rx", "ry", "rz"):
                g.append((name, q, 0, rng.uniform(0.0, TWO_PI), -1))
        for i in range(layer % 2, n - 1, 2):
            g.append(("cnot", i, i + 1, 0.0, -1))
    return g


def _h_cnot(n, count, rng):
    g = []
    for _ in range(count):
        if rng.random() < 0.5:
            g.append(("h", int(rng.integers(n)), 0, 0.0, -1))
        else:
            c, t = rng.choice(n, size=2, replace=False)
            g.append(("cnot", int(c), int(t), 0.0, -1))
    return g


def _hea(n, layers, params=None):
    g, k = [], 0
    for _ in range(layers):
        for name in ("ry", "rz"):
            for q in range(n):
                g.append((name, q, 0, 0.0 if params is None else float(params[k]), k))
                k += 1
        for q in range(n):
            g.append(("cz", q, (q + 1) % n, 0.0, -1))
    return g


def _qaoa(n, layers, rng):
    g = [("h", q, 0, 0.0, -1) for q in range(n)]
    for _ in range(layers):
        gamma, beta = rng.uniform(0.2, 1.2), rng.uniform(0.2, 1.2)
        for a, b in _qaoa_edges(n):
            g += [("cnot", a, b, 0.0, -1), ("rz", b, 0, gamma, -1), ("cnot", a, b, 0.0, -1)]
        for q in range(n):
            g.append(("rx", q, 0, 2.0 * beta, -1))
    return g


def _qaoa_edges(n):
    """A ring with chords: about 1.5 edges a vertex."""
    e = [(q, (q + 1) % n) for q in range(n)]
    return e + [(q, (q + n // 2) % n) for q in range(0, n // 2, 1) if q % 2 == 0 and n > 4]


def _noisy(n, layers, rng):
    g = []
    for _ in range(layers):
        for q in range(n):
            g.append(("rx", q, 0, rng.uniform(0.0, TWO_PI), -1))
            g.append(("ry", q, 0, rng.uniform(0.0, TWO_PI), -1))
        for i in range(n - 1):
            g.append(("cnot", i, i + 1, 0.0, -1))
    return g


def _random_circuit(n, depth, rng):
    g = []
    for _ in range(depth):
        name = ("h", "rx", "ry", "rz", "cnot", "cz")[int(rng.integers(6))]
        if name in ("cnot", "cz"):
            a, b = rng.choice(n, size=2, replace=False)
            g.append((name, int(a), int(b), 0.0, -1))
        else:
            g.append((name, int(rng.integers(n)), 0, 0.0 if name == "h" else rng.uniform(0.0, TWO_PI), -1))
    return g


GAMMA, LAMBDA, DEPOL = 0.002, 0.003, 0.01


def _inputs(case, seed):
    """(gate list(s), everything else drawn from the seed) of a case."""
    rng = np.random.default_rng(seed)
    k, n = case["kind"], case.get("n", 0)
    if k == "energy":
        if case["ansatz"] == "qaoa":
            return _qaoa(n, case["layers"], rng)
        return _hea(n, case["layers"], rng.uniform(0.0, TWO_PI, 2 * n * case["layers"]))
    if k == "circuit":
        return (_h_cnot if case["circuit"] == "h_cnot" else _layered)(n, case["layers"], rng)
    if k == "adjoint":
        return _hea(n, case["layers"]), rng.uniform(0.0, TWO_PI, (case["batch"], 2 * n * case["layers"]))
    if k == "traj":
        return _noisy(n, case["layers"], rng), int(rng.integers(1, 1 << 30))
    if k == "batch":
        sizes = _batch_sizes(case)
        return sizes, [_random_circuit(m, case["depth"], rng) for m in sizes]
    return _layered(n, case["layers"], rng)  # density


def _batch_sizes(case):
    lo, hi = case["lo"], case["hi"]
    return [lo + (7 * i) % (hi - lo + 1) for i in range(case["count"])]


def _records(gates):
    import llgpu

    kinds = {"h": llgpu.OP_H, "rx": llgpu.OP_RX, "ry": llgpu.OP_RY, "rz": llgpu.OP_RZ, "cnot": llgpu.OP_CNOT, "cz": llgpu.OP_CZ}
    ops = np.zeros(len(gates), dtype=llgpu.OP_DTYPE)
    ops["kind"] = [kinds[g[0]] for g in gates]
    ops["q0"] = [g[1] for g in gates]
    ops["q1"] = [g[2] for g in gates]
    ops["theta"] = [g[3] for g in gates]
    ops["param"] = [g[4] for g in gates]
    return ops


# ---------------------------------------------------------------------------------------------
# a user's program
# ---------------------------------------------------------------------------------------------
def prepare(case, seed):
    import llgpu

    k, n, precision = case["kind"], case.get("n", 0), case["precision"]
    made = _inputs(case, seed)
    if k == "energy":
        pairs = _qaoa_edges(n) if case["ansatz"] == "qaoa" else [(q, (q + 1) % n) for q in range(n)]
        terms = [p[0] for p in pairs], [p[1] for p in pairs], [1.0] * len(pairs)
        return {"case": case, "ops": _records(made), "state": llgpu.State(n, precision), "terms": terms}
    if k == "circuit":
        import quantum_sim_v3

        sv = quantum_sim_v3.StateVector(n, precision)
        sv.get_numpy_view()  # the object's host view, which it keeps
        return {"case": case, "ops": _records(made), "sv": sv}
    if k == "adjoint":
        gates, params = made
        ring = list(range(n)), [(q + 1) % n for q in range(n)], [1.0] * n
        handle = llgpu.Adjoint(n, _records(gates), params.shape[1], ring, case["batch"], precision)
        return {"case": case, "handle": handle, "params": params}
    if k == "traj":
        gates, s = made
        return {"case": case, "handle": llgpu.Traj(n, _records(gates), GAMMA, LAMBDA, case["ntraj"], precision), "seed": s}
    if k == "batch":
        sizes, circuits = made
        ops = np.concatenate([_records(c) for c in circuits])
        offsets = np.arange(len(sizes) + 1, dtype=np.int64) * case["depth"]
        return {"case": case, "batch": llgpu.Batch(sizes, ops, offsets, precision), "count": len(sizes)}
    host = torch.empty(2 << (2 * n), dtype=torch.float64, pin_memory=True)
    return {"case": case, "ops": _records(made), "dm": llgpu.DensityMatrix(n, precision), "host": host,
            "view": host.numpy().view(np.complex128), "ad": llgpu.amplitude_damping(0.05), "dep": llgpu.depolarizing(DEPOL, 2)}


def run(state):
    case = state["case"]
    k = case["kind"]
    if k == "energy":
        st = state["state"]
        st.reset(case["n"])
        st.apply_ops(state["ops"])
        return st.expect_zz(*state["terms"])
    if k == "circuit":
        sv = state["sv"]
        sv.reset(case["n"])
        sv.apply_ops(state["ops"])
        return sv.get_numpy_view()
    if k == "adjoint":
        energies, grads = state["handle"].run(state["params"])
        return {"energies": energies, "grads": grads}
    if k == "traj":
        z0, jumps, _ = state["handle"].launch(state["seed"], case["ntraj"])
        return {"z0": z0, "jumps": jumps}
    if k == "batch":
        state["batch"].run()
        return [state["batch"].state(i) for i in range(state["count"])]
    dm, n = state["dm"], case["n"]
    dm.state.reset(2 * n)
    per = len(state["ops"]) // case["layers"]
    for layer in range(case["layers"]):
        dm.apply_ops(state["ops"][layer * per:(layer + 1) * per])
        for q in range(n):
            dm.kraus(state["ad"], [q])
        for q in range(0, n - 1, 2):
            dm.kraus(state["dep"], [q, q + 1])
    return dm.state.state(state["view"])


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------
def _matvecs(gates, n):
    """One-qubit matrices left when neighbours on a qubit are merged (two-qubit gates only move
    amplitudes or change signs)."""
    open_, count = [False] * n, 0
    for name, a, b, _, _ in gates:
        if name in ("cnot", "cz"):
            open_[a] = open_[b] = False
        elif not open_[a]:
            open_[a] = True
            count += 1
    return count


def work(case):
    k, n, amp = case["kind"], case.get("n", 0), 8 if case["precision"] == "complex64" else 16
    flops_gate = 14.0  # of a complex 2x2 product, per amplitude
    if k == "energy":
        return {"bytes": float(amp << n), "flops": (flops_gate * _matvecs(_inputs(case, 1), n) + 4.0) * 2.0 ** n}
    if k == "circuit":
        return {"bytes": float(16 << n), "flops": flops_gate * _matvecs(_inputs(case, 1), n) * 2.0 ** n}
    if k == "adjoint":
        gates, params = _inputs(case, 1)
        # forward, and back: the state, the adjoint state and one inner product a rotation
        per = 3 * flops_gate * _matvecs(gates, n) + 4.0 * params.shape[1]
        return {"bytes": 3.0 * case["batch"] * (amp << n), "flops": per * case["batch"] * 2.0 ** n}
    if k == "traj":
        gates, _ = _inputs(case, 1)
        sites = sum(2 if g[0] == "cnot" else 1 for g in gates)
        per = flops_gate * _matvecs(gates, n) + 5.0 * sites  # a site: P(1) and the no-jump factors
        return {"bytes": 12.0 * case["ntraj"], "flops": per * case["ntraj"] * 2.0 ** n}
    if k == "batch":
        sizes, circuits = _inputs(case, 1)
        amps = float(sum(1 << m for m in sizes))
        return {"bytes": 16.0 * amps, "flops": sum(flops_gate * _matvecs(c, m) * 2.0 ** m for m, c in zip(sizes, circuits))}
    gates = _inputs(case, 1)
    per = 2 * flops_gate * _matvecs(gates, n) + case["layers"] * (5.0 * n + 12.0 * (n // 2))
    return {"bytes": float(16 << (2 * n)), "flops": per * 4.0 ** n}


# ---------------------------------------------------------------------------------------------
# the results in 64 bits, from plain torch
# ---------------------------------------------------------------------------------------------
def _matrix(name, theta):
    c, s = math.cos(0.5 * theta), math.sin(0.5 * theta)
    if name == "h":
        r = math.sqrt(0.5)
        return [[r, r], [r, -r]]
    if name == "rx":
        return [[c, -1j * s], [-1j * s, c]]
    if name == "ry":
        return [[c, -s], [s, c]]
    return [[c - 1j * s, 0], [0, c + 1j * s]]


def _apply(psi, n, name, a, b, theta, conj=False):
    """A gate on the last axis (2^n long) of `psi`, in place."""
    if name in ("cnot", "cz"):
        hi, lo = max(a, b), min(a, b)
        v = psi.view(-1, 1 << (n - 1 - hi), 2, 1 << (hi - lo - 1), 2, 1 << lo)
        if name == "cz":
            v[:, :, 1, :, 1] *= -1
        elif a == hi:  # the control is the higher qubit
            v[:, :, 1] = v[:, :, 1].flip(3)
        else:
            v[:, :, :, :, 1] = v[:, :, :, :, 1].flip(2)
        return
    m = _matrix(name, theta)
    if conj:
        m = [[complex(x).conjugate() for x in row] for row in m]
    v = psi.view(-1, 2, 1 << a)
    if name == "rz":
        v[:, 0] *= m[0][0]
        v[:, 1] *= m[1][1]
        return
    x, y = v[:, 0].clone(), v[:, 1].clone()
    v[:, 0] = m[0][0] * x + m[0][1] * y
    v[:, 1] = m[1][0] * x + m[1][1] * y


def _zero_state(n, batch=1):
    psi = torch.zeros(batch, 1 << n, dtype=torch.complex128, device="cuda")
    psi[:, 0] = 1.0
    return psi


def _diagonal(n, pairs):
    i = torch.arange(1 << n, device="cuda")
    d = torch.zeros(1 << n, dtype=torch.float64, device="cuda")
    for a, b in pairs:
        d += 1.0 - 2.0 * (((i >> a) ^ (i >> b)) & 1).double()
    return d


def _run_gates(n, gates):
    psi = _zero_state(n)
    for name, a, b, theta, _ in gates:
        _apply(psi, n, name, a, b, theta)
    return psi[0]


def _exact_adjoint(case, gates, params):
    n, batch = case["n"], case["batch"]
    diag = _diagonal(n, [(q, (q + 1) % n) for q in range(n)])
    energies, grads = np.zeros(batch), np.zeros(params.shape)
    for j in range(batch):
        psi = _run_gates(n, [(g[0], g[1], g[2], params[j, g[4]] if g[4] >= 0 else 0.0, -1) for g in gates])
        lam = psi * diag
        energies[j] = float(torch.sum(psi.abs().square() * diag))
        got = []
        for name, a, b, _, p in reversed(gates):
            if p < 0:
                _apply(psi, n, name, a, b, 0.0)
                _apply(lam, n, name, a, b, 0.0)
                continue
            u, v = lam.view(-1, 2, 1 << a), psi.view(-1, 2, 1 << a)
            # dE/dtheta = Im <lam| P |psi> with P = Y or Z, both vectors after the gate
            if name == "rz":
                d = (u[:, 0].conj() * v[:, 0]).sum() - (u[:, 1].conj() * v[:, 1]).sum()
            else:
                d = -1j * (u[:, 0].conj() * v[:, 1]).sum() + 1j * (u[:, 1].conj() * v[:, 0]).sum()
            got.append((p, d.imag))
            _apply(psi, n, name, a, b, -params[j, p])
            _apply(lam, n, name, a, b, -params[j, p])
        for p, d in got:
            grads[j, p] += float(d)
    return {"energies": energies, "grads": grads}


def _philox_uniform(seed, traj, site):
    """The first 53-bit uniform of Philox4x32-10 (Salmon, Moraes, Dror and Shaw, SC'11) with key
    `seed` and counter (site, trajectory), for arrays of trajectories and sites."""
    u64, low = np.uint64, np.uint64(0xFFFFFFFF)
    site, traj = np.broadcast_arrays(np.asarray(site, u64), np.asarray(traj, u64))
    c = [site & low, site >> u64(32), traj & low, traj >> u64(32)]
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    for _ in range(10):
        p0, p1 = u64(0xD2511F53) * c[0], u64(0xCD9E8D57) * c[2]
        c = [(p1 >> u64(32)) ^ c[1] ^ u64(k0), p1 & low, (p0 >> u64(32)) ^ c[3] ^ u64(k1), p0 & low]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return (((c[1] << u64(32)) | c[0]) >> u64(11)).astype(np.float64) * 2.0 ** -53


def _exact_traj(case, gates, seed):
    n, count = case["n"], case["ntraj"]
    psi = _zero_state(n, count)
    jumps = torch.zeros(count, dtype=torch.int64, device="cuda")
    sites = 2 * sum(2 if g[0] == "cnot" else 1 for g in gates)
    uniforms = torch.from_numpy(_philox_uniform(seed, np.arange(count)[None, :], np.arange(sites)[:, None])).cuda()
    site = 0
    for name, a, b, theta, _ in gates:
        _apply(psi, n, name, a, b, theta)
        for q in ((a, b) if name == "cnot" else (a,)):
            v = psi.view(count, -1, 2, 1 << q)
            p1 = torch.view_as_real(v[:, :, 1]).square().sum(dim=(1, 2, 3))
            # amplitude damping, then phase damping: the factors of both act together below
            survive = 1.0 - GAMMA * p1
            ad = (uniforms[site] >= survive) & (GAMMA * p1 > 0)
            s0, s1 = survive.rsqrt(), math.sqrt(1.0 - GAMMA) * survive.rsqrt()
            down = torch.where(ad, p1.rsqrt(), torch.zeros_like(p1))  # |1> moves to |0>
            s0, s1 = torch.where(ad, torch.zeros_like(s0), s0), torch.where(ad, torch.zeros_like(s1), s1)
            q1 = torch.where(ad, torch.zeros_like(p1), (1.0 - GAMMA) * p1 / survive)
            survive = 1.0 - LAMBDA * q1
            pd = (uniforms[site + 1] >= survive) & (LAMBDA * q1 > 0)
            f0 = torch.where(pd, torch.zeros_like(q1), survive.rsqrt())
            f1 = torch.where(pd, q1.clamp_min(1e-300).rsqrt(), math.sqrt(1.0 - LAMBDA) * survive.rsqrt())
            one = v[:, :, 1].clone()
            v[:, :, 0] *= (s0 * f0)[:, None, None]
            if bool(ad.any()):
                v[:, :, 0] += (down * f0)[:, None, None] * one
            v[:, :, 1] *= (s1 * f1)[:, None, None]
            jumps += ad.long() + pd.long()
            site += 2
    p = torch.view_as_real(psi).square().sum(dim=2).view(count, -1, 2).sum(dim=1)
    return {"z0": (p[:, 0] - p[:, 1]).cpu().numpy(), "jumps": None}


def _exact_density(case, gates):
    n, size = case["n"], 1 << case["n"]
    # rows in the low bits: element (row, col) at row + col * 2^n, as the framework stores it
    rho = _zero_state(2 * n)
    per = len(gates) // case["layers"]

    def channel(ops, qs):
        total = torch.zeros_like(rho)
        for weight, letters in ops:
            t = rho.clone()
            for q, letter in zip(qs, letters):
                for shift in (0, n):
                    v = t.view(-1, 2, 1 << (q + shift))
                    if letter == "x" or letter == "y":
                        v.copy_(v.flip(1))
                    if letter == "z" or letter == "y":
                        v[:, 1] *= -1  # y = z x up to a phase that cancels between row and column
            total += weight * t
        rho.copy_(total)

    for layer in range(case["layers"]):
        for name, a, b, theta, _ in gates[layer * per:(layer + 1) * per]:
            _apply(rho, 2 * n, name, a, b, theta)
            _apply(rho, 2 * n, name, a + n, b + n, theta, conj=True)
        for q in range(n):
            v = rho.view(1 << (n - 1 - q), 2, 1 << (n - 1), 2, 1 << q)
            v[:, 0, :, 0] += 0.05 * v[:, 1, :, 1]
            v[:, 1, :, 1] *= 0.95
            v[:, 0, :, 1] *= math.sqrt(0.95)
            v[:, 1, :, 0] *= math.sqrt(0.95)
        for q in range(0, n - 1, 2):
            paulis = [(DEPOL / 15.0, i + j) for i in "ixyz" for j in "ixyz" if i + j != "ii"]
            channel([(1.0 - DEPOL, "ii")] + paulis, (q, q + 1))
    return rho[0, :size * size].cpu().numpy()


def exact(case, seed):
    k, n = case["kind"], case.get("n", 0)
    made = _inputs(case, seed)
    if k == "energy":
        pairs = _qaoa_edges(n) if case["ansatz"] == "qaoa" else [(q, (q + 1) % n) for q in range(n)]
        return float(torch.sum(_run_gates(n, made).abs().square() * _diagonal(n, pairs)))
    if k == "circuit":
        return _run_gates(n, made).cpu().numpy()
    if k == "adjoint":
        return _exact_adjoint(case, *made)
    if k == "traj":
        return _exact_traj(case, *made)
    if k == "batch":
        return [_run_gates(m, c).cpu().numpy() for m, c in zip(*made)]
    return _exact_density(case, made)
