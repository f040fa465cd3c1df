"""Gate blocks on registers of 6 to 11 qubits, which fill a part of the kernel's one tile: deep circuits, from the
zero state and from the host, read back through the state and through a pinned view, against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import llgpu
import oracle
import workloads
from llgpu import OP_CNOT, OP_CZ, OP_H, OP_MCZ, OP_RX, OP_RZ, make_ops

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built(built):
    assert llgpu.device_count() > 0


@pytest.mark.parametrize("precision,tol", [("complex128", 1e-13), ("df64", 1e-12)])
@pytest.mark.parametrize("n", [6, 7, 8, 9, 10, 11])
def test_deep_circuits(n, precision, tol):
    ops = workloads.layered_rotations(n, 20)
    want = oracle.run_ops(n, ops)
    st = llgpu.State(n, precision)
    st.apply_ops(ops)
    assert np.max(np.abs(st.state() - want)) <= tol
    tiles = llgpu.State(n, precision)
    tiles.set_fusion("tile", 12)
    tiles.apply_ops(ops)
    assert np.max(np.abs(tiles.state() - want)) <= tol
    # from the host, in two flushes, with gates on every pair and a sign flip on six qubits
    rng = np.random.default_rng(n)
    psi = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    psi /= np.linalg.norm(psi)
    recs = [(OP_H, q) for q in range(n)]
    for a in range(n):
        for b in range(n):
            if a != b:
                recs += [(OP_CNOT if (a + b) % 2 else OP_CZ, a, b), (OP_RX, a, 0, 0.1 * a + 0.3), (OP_RX, b, 0, 0.7),
                         (OP_RZ, b, 0, 0.2 * b)]
    recs.append((OP_MCZ, 0, 0, 0.0, 0b111111))
    more = make_ops(recs + recs[:40])
    st = llgpu.State(precision=precision, amps=psi)
    st.apply_ops(more)
    st.flush()
    st.apply_ops(ops)
    both = np.concatenate([more, ops])
    assert np.max(np.abs(st.state() - oracle.run_ops(n, both, psi))) <= tol


def test_infinite_amplitudes_stay_off_the_blocks():
    n = 9
    psi = np.zeros(1 << n, dtype=np.complex128)
    psi[3] = np.inf
    ops = workloads.layered_rotations(n, 20)
    st, tiles = llgpu.State(amps=psi), llgpu.State(amps=psi)
    tiles.set_fusion("tile", 12)
    for s in (st, tiles):
        s.apply_ops(ops)
    assert np.array_equal(st.state(), tiles.state(), equal_nan=True)
