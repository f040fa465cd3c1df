"""Flushes that begin as gate blocks and end as tile passes: every gate runs once and in an order that the list allows, with
sign flips on many qubits, channels and the state written to a pinned mirror by the last pass."""
from __future__ import annotations

import numpy as np
import pytest

import llgpu
import oracle
from llgpu import OP_CNOT, OP_CZ, OP_H, OP_MCZ, OP_RX, OP_RY, OP_RZ, OP_U2, OP_X, make_ops
from test_engine_host_cpu import changing

pytestmark = pytest.mark.gpu

TOL = {"complex128": 1e-12, "df64": 1e-11}


@pytest.fixture(scope="module", autouse=True)
def _built(built):
    assert llgpu.device_count() > 0


def passes(st, f):
    """(gate blocks, all fused passes) of f()."""
    st.profile(True)
    st.profile_read()
    before = llgpu.gate_block_launches()
    f()
    blocks = llgpu.gate_block_launches() - before
    return blocks, st.profile_read()["tile"][1]


def tail(n, rng, count):
    recs = []
    for _ in range(count):
        a, b = (int(x) for x in rng.choice(n, size=2, replace=False))
        recs.append((OP_CNOT, a, b))
        if rng.random() < 0.05:
            recs.append((int(rng.choice([OP_CZ, OP_CNOT])), b, a))
            recs.append((OP_MCZ, 0, 0, 0.0, sum(1 << int(q) for q in rng.choice(n, size=int(rng.integers(1, n)), replace=False))))
            u = np.linalg.qr(rng.normal(size=(2, 2)) + 1j * rng.normal(size=(2, 2)))[0]
            recs += [(OP_X, a), (OP_H, b), (OP_RZ, a, 0, 0.7), (OP_U2, b, 0, 0.0, None, u), (OP_RX, a, 0, 0.2), (OP_RY, a, 0, 0.9)]
    return make_ops(recs)


@pytest.mark.parametrize("n,precision", [(8, "complex128"), (10, "complex128"), (11, "complex128"), (12, "df64"), (14, "df64")])
@pytest.mark.parametrize("pinned", [False, True])
def test_against_oracle(n, precision, pinned):
    ops = np.concatenate([changing(n, 120, 40), tail(n, np.random.default_rng(n), 500)])
    want = oracle.run_ops(n, ops)
    if pinned:
        torch = pytest.importorskip("torch")
        out = torch.empty(2 << n, dtype=torch.float64, pin_memory=True).numpy().view(np.complex128)
    else:
        out = np.empty(1 << n, dtype=np.complex128)
    st = llgpu.State(n, precision)
    st.apply_ops(ops)
    blocks, fused = passes(st, lambda: st.state(out))
    assert 0 < blocks < fused
    assert np.max(np.abs(out - want)) <= TOL[precision]
    st.close()


def test_with_channels():
    n = 6
    rng = np.random.default_rng(4)
    dm = llgpu.DensityMatrix(n, "df64")
    want = oracle.dm_zero(n)
    first, second = changing(n, 100, 0), changing(n, 0, 3000)
    for ops in (first, second):
        dm.apply_ops(ops)
        want = oracle.dm_apply_ops(want, n, ops)
        for q in (0, 3, 5):
            dm.kraus(llgpu.amplitude_damping(0.1), [q])
            want = oracle.kraus_apply(want, n, llgpu.amplitude_damping(0.1), [q])
    blocks, fused = passes(dm.state, dm.state.sync)
    assert 0 < blocks < fused
    assert np.max(np.abs(dm.rho() - want)) <= TOL["df64"]
    dm.close()
