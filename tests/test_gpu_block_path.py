"""That the circuits of the gate-block tests run as gate blocks: the choice rests on fitted costs, on the gates' norms and
on free memory, and where it fell to tile passes those tests would compare tile passes with themselves."""
from __future__ import annotations

import numpy as np
import pytest

import llgpu
import test_gpu_adjblock
import test_gpu_batch_blocks
import test_gpu_gateblock
import workloads

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built(built):
    assert llgpu.device_count() > 0


def launches(f):
    before = llgpu.gate_block_launches()
    f()
    return llgpu.gate_block_launches() - before


def flush_launches(st, ops):
    st.apply_ops(ops)
    return launches(st.sync)


@pytest.mark.parametrize("precision", ["complex128", "df64"])
@pytest.mark.parametrize("n,depth", [(12, 12), (13, 8), (17, 6), (20, 4)])
def test_fused_circuits(precision, n, depth):
    ops = test_gpu_gateblock._circuit(n, depth, n)
    st = llgpu.State(n, precision)
    steps, _ = llgpu.block_plan_export(n, ops)
    assert flush_launches(st, ops) == int(steps["is_block"].sum())
    st.set_fusion("tile", 11)
    assert flush_launches(st, ops) == 0
    st.close()


@pytest.mark.parametrize("precision", ["complex128", "df64"])
@pytest.mark.parametrize("n", [6, 7, 8, 9, 10, 11])
def test_small_registers(n, precision):
    st = llgpu.State(n, precision)
    assert flush_launches(st, workloads.layered_rotations(n, 20)) > 0
    st.close()


def test_more_blocks_than_slots():
    st = llgpu.State(12, "complex128")
    assert flush_launches(st, np.concatenate([test_gpu_gateblock._circuit(12, 40, 5)] * 2)) > 128
    st.close()


def test_channels():
    dm = llgpu.DensityMatrix(6)
    ops = test_gpu_gateblock._circuit(8, 1, 0)
    dm.apply_ops(ops[(ops["q0"] < 6) & (ops["q1"] < 6) & (ops["kind"] != llgpu.OP_MCZ)])
    for q in range(6):
        dm.kraus(llgpu.amplitude_damping(0.1), [q])
    assert launches(dm.state.sync) > 0
    dm.close()


def test_batches():
    sizes = [12, 13, 12, 14, 16, 12]
    circuits = test_gpu_batch_blocks.batch(sizes, [100] * 6, 7)
    off = np.concatenate([[0], np.cumsum([len(c) for c in circuits])])
    b = llgpu.Batch(np.array(sizes), np.concatenate(circuits), off, "complex128")
    assert launches(b.run) > 0
    tiles = llgpu.Batch(np.array(sizes), np.concatenate(circuits), off, "complex128", 12)
    assert launches(tiles.run) == 0
    b.close()
    tiles.close()


# (five sets of 12 qubits and three layers are left to tile passes, which are no slower there)
@pytest.mark.parametrize("n,depth,batch", [(12, 4, 1), (12, 8, 5), (13, 4, 3), (17, 4, 2)])
def test_adjoint(n, depth, batch):
    nparams = 9
    ops = test_gpu_adjblock._circuit(n, depth, nparams, 10 * n + batch)
    h = llgpu.Adjoint(n, ops, nparams, llgpu.ring_zz_terms(n), batch)
    params = np.random.default_rng(n).uniform(0, 6, (batch, nparams))
    got = {}
    assert launches(lambda: got.update(blocks=h.run(params))) > 0
    h.set_threads(128)
    assert launches(lambda: got.update(tiles=h.run(params))) == 0
    h.close()
    for x, y in zip(got["blocks"], got["tiles"]):
        assert np.max(np.abs(x - y)) <= 1e-12
