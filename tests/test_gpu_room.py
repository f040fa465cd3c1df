"""Device memory that the block forms take beside the states: a part of what is free, so that the caller's next allocation has
room, and tile passes where that part is too small."""
from __future__ import annotations

import numpy as np
import pytest

import llgpu
import oracle
import workloads
from test_gpu_batch_blocks import batch

pytestmark = pytest.mark.gpu
MB = 1 << 20


@pytest.fixture(scope="module", autouse=True)
def _built(built):
    assert llgpu.device_count() > 0


@pytest.fixture
def nearly_full():
    """All but some 400 MB of the device taken by the test."""
    torch = pytest.importorskip("torch")
    torch.cuda.init()
    torch.cuda.synchronize()
    free, _ = torch.cuda.mem_get_info()
    try:
        hold = torch.empty(free - 400 * MB, dtype=torch.uint8, device="cuda")
    except torch.cuda.OutOfMemoryError:
        pytest.skip("the device's memory cannot be taken in one piece")
    yield lambda: torch.cuda.mem_get_info()[0]
    del hold
    torch.cuda.empty_cache()


def test_batch(nearly_full):
    sizes = [12, 13, 14] * 12
    circuits = batch(sizes, [1500] * len(sizes), 5)
    off = np.concatenate([[0], np.cumsum([len(c) for c in circuits])])
    before = nearly_full()
    tiles = llgpu.Batch(np.array(sizes), np.concatenate(circuits), off, "complex128", 12)
    form = before - nearly_full()  # the states and all that tile passes need
    tiles.close()
    before = nearly_full()
    b = llgpu.Batch(np.array(sizes), np.concatenate(circuits), off, "complex128")
    taken = before - nearly_full()
    b.run()
    for i in (0, 19, 35):
        assert np.max(np.abs(b.state(i) - oracle.run_ops(sizes[i], circuits[i]))) <= 1e-12
    b.close()
    assert taken <= form + (before - sum(16 << n for n in sizes)) // 4 + 8 * MB


def test_adjoint(nearly_full):
    n, layers, sets = 14, 12, 96
    ops = workloads.hea_ansatz(n, layers)
    params = workloads.hea_params(n, layers, sets)
    h = llgpu.Adjoint(n, ops, params.shape[1], llgpu.ring_zz_terms(n), sets)
    before = nearly_full()
    blocks = llgpu.gate_block_launches()
    e, g = h.run(params)
    taken = before - nearly_full()
    assert llgpu.gate_block_launches() > blocks
    h.set_threads(128)
    et, gt = h.run(params)
    h.close()
    assert np.max(np.abs(e - et)) <= 1e-12 and np.max(np.abs(g - gt)) <= 1e-12
    assert taken <= before // 4 + 32 * MB
