"""Amplitudes far below their neighbours, each against itself: rotations by small angles, whose products a block would
hold in units of its largest, and gates that only move amplitudes or turn their phases."""
from __future__ import annotations

import numpy as np
import pytest

import llgpu
from llgpu import OP_CNOT, OP_CZ, OP_RX, OP_RY, OP_RZ, OP_X, make_ops

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built(built):
    assert llgpu.device_count() > 0


def product(n, angle, layers):
    """RY(angle) `layers` times on every qubit with RZs between (at the end of no effect on the sizes)."""
    recs = []
    for _ in range(layers):
        recs += [(OP_RY, q, 0, angle) for q in range(n)]
    recs += [(OP_RZ, q, 0, 0.3 + q) for q in range(n)]
    c, s = np.cos(layers * angle / 2), np.sin(layers * angle / 2)
    ones = np.array([bin(i).count("1") for i in range(1 << n)])
    return make_ops(recs), c ** (n - ones) * s ** ones


@pytest.mark.parametrize("angle", [2e-5, 2e-4])
@pytest.mark.parametrize("n", [9, 12, 14])
def test_small_rotations(n, angle):
    # one merged gate a qubit: some ten roundings of 2^-53 for each factor
    ops, want = product(n, angle, 20)
    st = llgpu.State(n, "complex128")
    st.apply_ops(ops)
    assert np.max(np.abs(np.abs(st.state()) / want - 1.0)) <= 1e-12
    st.close()


def test_small_rotations_in_a_batch():
    sizes = [12, 13, 12, 14]
    made = [product(n, 2e-5, 20) for n in sizes]
    off = np.concatenate([[0], np.cumsum([len(m[0]) for m in made])])
    b = llgpu.Batch(np.array(sizes), np.concatenate([m[0] for m in made]), off, "complex128")
    b.run()
    for i, (_, want) in enumerate(made):
        assert np.max(np.abs(np.abs(b.state(i)) / want - 1.0)) <= 1e-12
    b.close()


@pytest.mark.parametrize("precision,tol", [("complex128", 1e-13), ("df64", 1e-12)])
@pytest.mark.parametrize("n", [9, 12, 15, 20])
def test_moves_and_phases_keep_every_amplitude(n, precision, tol):
    rng = np.random.default_rng(n)
    size = 10.0 ** rng.uniform(-20, 0, 1 << n)
    psi = size * np.exp(1j * rng.uniform(0, 6.28, 1 << n))
    idx = np.arange(1 << n)
    recs = []
    want = psi.copy()
    for _ in range(300):
        k = int(rng.choice([OP_CNOT, OP_CZ, OP_X, OP_RZ]))
        a, b = (int(x) for x in rng.choice(n, size=2, replace=False))
        if k == OP_RZ:
            recs.append((k, a, 0, 0.1 * b + 0.3))
            continue
        recs.append((k, a, b) if k != OP_X else (k, a))
        if k == OP_X:
            want = want[idx ^ (1 << a)]
        elif k == OP_CNOT:
            want = want[np.where(idx >> a & 1, idx ^ (1 << b), idx)]
    st = llgpu.State(precision=precision, amps=psi)
    start = np.abs(st.state())
    st.apply_ops(make_ops(recs))
    got = np.abs(st.state())
    ref = np.abs(want) * 1.0
    assert np.max(np.abs(got / ref - 1.0)) <= tol + np.max(np.abs(start / np.abs(psi) - 1.0))
    st.close()
