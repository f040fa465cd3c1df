"""Gate blocks on registers of 6 to 9 qubits, where some lanes of a warp hold no group: the same bits every time, and
every amplitude right, with targets that leave the lanes of a group next to each other and far apart."""
from __future__ import annotations

import numpy as np
import pytest

import llgpu
import oracle
import workloads

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built(built):
    assert llgpu.device_count() > 0


# 20 layers of rotations: a few hundred products of unitary matrices, each rounded once
@pytest.mark.parametrize("precision,tol", [("complex128", 1e-13), ("df64", 1e-12)])
@pytest.mark.parametrize("n", [6, 7, 8, 9])
def test_lanes_without_a_group(n, precision, tol):
    ops = workloads.layered_rotations(n, 20)
    want = oracle.run_ops(n, ops)
    st = llgpu.State(n, precision)
    first = None
    for _ in range(20):
        st.reset(n)
        st.apply_ops(ops)
        got = st.state()
        first = got if first is None else first
        assert np.array_equal(got, first)
    assert np.max(np.abs(first - want)) <= tol
    st.close()
