"""2x2 gates that are not unitary beside gates that mix: scaled rotations, Kraus operators, projectors, singular
matrices.  Blocks hold their products against 1, so such lists have to keep the result's own relative accuracy some other
way.  Flushes, batches and adjoint sweeps, against the oracle and relative to the result's norm."""
from __future__ import annotations

import numpy as np
import pytest

import llgpu
import oracle
from llgpu import OP_CNOT, OP_RY, OP_RZ, OP_U2, make_ops

pytestmark = pytest.mark.gpu

# of the result's norm: some hundred FP64 roundings of 2^-53; double-float holds 2^-47 of an amplitude
TOL = {"complex128": 1e-13, "df64": 1e-11}


@pytest.fixture(scope="module", autouse=True)
def _built(built):
    assert llgpu.device_count() > 0


def ry(t):
    c, s = np.cos(t / 2), np.sin(t / 2)
    return np.array([[c, -s], [s, c]])


GATES = {
    "half": lambda rng: 0.5 * ry(rng.uniform(0, 6)),
    "0.1": lambda rng: 0.1 * ry(rng.uniform(0, 6)),
    "1e-3": lambda rng: 1e-3 * ry(rng.uniform(0, 6)),
    "1e-4": lambda rng: 1e-4 * ry(rng.uniform(0, 6)),
    "1e-9 of the identity": lambda rng: 1e-9 * np.eye(2),
    "kraus": lambda rng: np.diag([1.0, np.sqrt(1 - 0.999999)]),
    "jump": lambda rng: np.array([[0.0, 1e-5], [0.0, 0.0]]),
    "projector": lambda rng: np.outer(*[ry(rng.uniform(0, 6))[:, 0]] * 2),
}


def circuit(n, layers, gate, rng):
    recs = []
    for layer in range(layers):
        for q in range(n):
            recs.append((OP_RY, q, 0, rng.uniform(0.3, 2.8)))
            recs.append((OP_RZ, q, 0, rng.uniform(0, 6)))
            if layer == 1:
                recs.append((OP_U2, q, 0, 0.0, None, GATES[gate](rng)))
        for q in range(layer % 2, n - 1, 2):
            recs.append((OP_CNOT, q, q + 1))
    return make_ops(recs)


def close(got, want, tol):
    norm = np.linalg.norm(want)
    assert norm > 0.0 and np.linalg.norm(got - want) <= tol * norm


@pytest.mark.parametrize("precision", ["complex128", "df64"])
@pytest.mark.parametrize("gate", list(GATES))
@pytest.mark.parametrize("n", [9, 12, 14])
def test_flush(n, gate, precision):
    ops = circuit(n, 6, gate, np.random.default_rng(n))
    want = oracle.run_ops(n, ops)
    if precision == "df64" and np.linalg.norm(want) < 2.0 ** -66:
        pytest.skip("amplitudes of 2^-7 of the norm would have low parts, 2^-53 below them, under the floats' 2^-126")
    st = llgpu.State(n, precision)
    st.apply_ops(ops)
    close(st.state(), want, TOL[precision])
    st.renormalize()
    close(st.state(), want / np.linalg.norm(want), TOL[precision])
    st.close()


@pytest.mark.parametrize("gate", list(GATES))
def test_batch(gate):
    rng = np.random.default_rng(5)
    sizes = [12, 13, 12, 14, 11]
    circuits = [circuit(n, 8, gate, rng) for n in sizes]
    off = np.concatenate([[0], np.cumsum([len(c) for c in circuits])])
    b = llgpu.Batch(np.array(sizes), np.concatenate(circuits), off, "complex128")
    b.run()
    for i, n in enumerate(sizes):
        close(b.state(i), oracle.run_ops(n, circuits[i]), TOL["complex128"])
    b.close()


@pytest.mark.parametrize("gate", ["half", "1e-3", "1e-4"])
def test_adjoint_energies(gate):
    n, layers = 14, 10
    ops = circuit(n, layers, gate, np.random.default_rng(3))
    first = int(np.flatnonzero(ops["kind"] == OP_RY)[0])
    ops["param"][first] = 0
    theta = float(ops["theta"][first])
    a, b, c = llgpu.ring_zz_terms(n)
    h = llgpu.Adjoint(n, ops, 1, (a, b, c), 1)
    e, _ = h.run(np.array([[theta]]), grads=False)
    h.close()
    ops["param"][first] = -1
    psi = oracle.run_ops(n, ops)
    i = np.arange(1 << n)
    p = np.abs(psi) ** 2
    want = sum(w * np.sum(p * (1 - 2 * (((i >> x) ^ (i >> y)) & 1))) for x, y, w in zip(a, b, c))
    assert np.sum(p) > 0 and abs(e[0] - want) <= 1e-11 * np.sum(p)
