"""Complex128 batches whose larger circuits run as gate blocks: against the oracle, with circuits that keep
tile passes beside them, uneven block counts, one-tile and many-tile states, and graph replays."""
from __future__ import annotations

import numpy as np
import pytest

import llgpu
import oracle
from llgpu import OP_CNOT, OP_CZ, OP_H, OP_MCZ, OP_RX, OP_RZ, OP_U2, make_ops

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built(built):
    assert llgpu.device_count() > 0


def batch(sizes, depths, seed, wide=()):
    """One random circuit per size; those whose index is in `wide` hold a sign flip on 6 qubits (no block plan)."""
    rng = np.random.default_rng(seed)
    circuits = []
    for i, (n, depth) in enumerate(zip(sizes, depths)):
        recs = []
        for _ in range(depth):
            k, q = int(rng.integers(6)), int(rng.integers(n))
            if k == 0:
                recs.append((OP_H, q))
            elif k < 3:
                recs.append(((OP_RX, OP_RZ)[k - 1], q, 0, float(rng.uniform(0, 6.28))))
            elif k == 3:
                u, _ = np.linalg.qr(rng.normal(size=(2, 2)) + 1j * rng.normal(size=(2, 2)))
                recs.append((OP_U2, q, 0, 0.0, None, u.reshape(4)))
            else:
                a, b = (int(x) for x in rng.choice(n, 2, replace=False))
                recs.append(((OP_CNOT, OP_CZ)[k - 4], a, b))
        if i in wide:
            recs.insert(depth // 2, (OP_MCZ, 0, 0, 0.0, 0b101111 << (n - 6)))
        circuits.append(make_ops(recs))
    return circuits


@pytest.mark.parametrize("sizes,wide", [
    ([12], ()),
    ([10, 11, 12, 11, 10, 13], ()),
    ([12, 13, 12, 14, 16, 12], ()),
    ([3, 17, 12, 2, 15, 13, 8, 10, 14, 12], (4,)),
    ([12] * 90 + [13] * 80 + [5] * 20, ()),
])
def test_blocks_match_oracle(sizes, wide):
    rng = np.random.default_rng(len(sizes))
    depths = [int(rng.integers(60, 260)) for _ in sizes]
    circuits = batch(sizes, depths, 7, wide)
    off = np.concatenate([[0], np.cumsum([len(c) for c in circuits])])
    b = llgpu.Batch(np.array(sizes), np.concatenate(circuits), off, "complex128")
    tiles = llgpu.Batch(np.array(sizes), np.concatenate(circuits), off, "complex128", 12)
    tiles.run()
    for _ in range(2):
        b.run()
    check = range(len(sizes)) if len(sizes) < 20 else range(0, len(sizes), 13)
    for i in check:
        want = oracle.run_ops(sizes[i], circuits[i])
        assert np.max(np.abs(b.state(i) - want)) <= 1e-13, i
        assert np.max(np.abs(tiles.state(i) - want)) <= 1e-13, i
    b.close()
    tiles.close()


def test_autotune_keeps_the_fastest():
    llgpu.tune_cache_clear()
    sizes = [12, 14, 16, 16, 9]
    circuits = batch(sizes, [150] * 5, 3)
    off = np.concatenate([[0], np.cumsum([len(c) for c in circuits])])
    b = llgpu.Batch(np.array(sizes), np.concatenate(circuits), off, "complex128", llgpu.TUNE_AUTO)
    b.run()
    for i, n in enumerate(sizes):
        assert np.max(np.abs(b.state(i) - oracle.run_ops(n, circuits[i]))) <= 1e-13, i
    b.close()
