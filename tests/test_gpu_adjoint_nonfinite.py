"""Angles that are not finite, in one parameter set of several: that set's energy and gradients are NaN, as in the tile
passes, and the other sets keep theirs."""
from __future__ import annotations

import numpy as np
import pytest

import llgpu
import workloads

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built(built):
    assert llgpu.device_count() > 0


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("n,layers", [(12, 8), (14, 6)])
@pytest.mark.parametrize("where", ["first", "last", "unused"])
def test_one_set_of_several(n, layers, where, value):
    ops = workloads.hea_ansatz(n, layers)
    params = workloads.hea_params(n, layers, 4)
    used = params.shape[1]
    params = np.concatenate([params, np.full((4, 1), 0.5)], axis=1)  # a parameter that no gate has
    params[2, {"first": 0, "last": used - 1, "unused": used}[where]] = value
    h = llgpu.Adjoint(n, ops, used + 1, llgpu.ring_zz_terms(n), 4)
    before = llgpu.gate_block_launches()
    e, g = h.run(params)
    only, _ = h.run(params, grads=False)
    assert llgpu.gate_block_launches() > before
    h.set_threads(128)
    et, gt = h.run(params)
    h.close()
    assert np.array_equal(np.isnan(e), np.isnan(et)) and np.array_equal(np.isnan(g), np.isnan(gt))
    assert np.array_equal(e, only, equal_nan=True)
    assert np.isnan(et[2]) == (where != "unused")
    ok = ~np.isnan(et)
    assert np.max(np.abs(e[ok] - et[ok])) <= 1e-12 and np.max(np.abs(g[ok] - gt[ok])) <= 1e-12
