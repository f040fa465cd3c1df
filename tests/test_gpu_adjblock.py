"""Adjoint gradients by 5-qubit blocks (csrc/llg_adjblock.cu) against the CPU oracle's parameter shift and
the tile passes: every gate kind, shared parameters, states that sit in few amplitudes, observables of
very different size, one tile and several CTAs a state, more sets than CTAs."""
from __future__ import annotations

import numpy as np
import pytest

import llgpu
import oracle
import workloads
from llgpu import OP_CNOT, OP_CZ, OP_H, OP_MCZ, OP_RX, OP_RY, OP_RZ, OP_U2, OP_X, make_ops

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built(built):
    assert llgpu.device_count() > 0


def _circuit(n, depth, nparams, seed, mix=True):
    rng = np.random.default_rng(seed)
    recs = []
    for d in range(depth):
        for q in range(n):
            k = int(rng.integers(6))
            if k < 3:
                recs.append(((OP_RX, OP_RY, OP_RZ)[k], q, 0, 0.0, None, None, int(rng.integers(nparams))))
            elif k == 3:
                u = np.linalg.qr(rng.normal(size=(2, 2)) + 1j * rng.normal(size=(2, 2)))[0]
                recs.append((OP_U2, q, 0, 0.0, None, u) if mix else (OP_RZ, q, 0, 0.4))
            elif k == 4:
                recs.append((OP_H, q) if mix else (OP_X, q))
        for _ in range(n // 2):
            a, b = (int(x) for x in rng.choice(n, size=2, replace=False))
            recs.append(((OP_CNOT, OP_CZ)[int(rng.integers(2))], a, b))
        qs = rng.choice(n, size=int(rng.integers(1, 6)), replace=False)
        recs.append((OP_MCZ, int(qs[0]), 0, 0.0, sum(1 << int(q) for q in qs)))
    return make_ops(recs)


def _both(n, ops, nparams, obs, params):
    """(energies, gradients) by blocks and by tile passes (a set CTA size asks for those)."""
    h = llgpu.Adjoint(n, ops, nparams, obs, params.shape[0])
    blocks = h.run(params)
    only_e, none = h.run(params, grads=False)
    assert none is None and np.array_equal(only_e, blocks[0])
    h.set_threads(128)
    tiles = h.run(params)
    h.close()
    return blocks, tiles


@pytest.mark.parametrize("n,depth,batch", [(12, 4, 1), (12, 3, 5), (13, 4, 3), (17, 4, 2)])
def test_every_gate_kind(n, depth, batch):
    nparams = 9
    ops = _circuit(n, depth, nparams, 10 * n + batch)
    rng = np.random.default_rng(n)
    params = rng.uniform(0, 2 * np.pi, (batch, nparams))
    a, b, c = llgpu.ring_zz_terms(n)
    (e, g), (et, gt) = _both(n, ops, nparams, (a + [0], b + [-1], c + [0.37]), params)
    # FP64 sums of norm |O| ~ n: a few hundred units of 2^-53
    assert np.max(np.abs(e - et)) <= 1e-12 and np.max(np.abs(g - gt)) <= 1e-12


def test_against_oracle_parameter_shift():
    n, layers = 12, 2
    ops = workloads.hea_ansatz(n, layers)
    params = workloads.hea_params(n, layers, 1)
    a, b, c = llgpu.ring_zz_terms(n)
    h = llgpu.Adjoint(n, ops, params.shape[1], (a, b, c), 1)
    e, g = h.run(params)
    ew, gw = oracle.param_shift(n, ops, params[0], np.array(a), np.array(b), np.array(c))
    assert abs(e[0] - ew) <= 1e-10 and np.max(np.abs(g[0] - gw)) <= 1e-10
    h.close()


@pytest.mark.parametrize("scale", [1e-30, 1.0, 1e25])
def test_concentrated_states_and_scaled_observables(scale):
    # angles near 0: nearly all weight in one amplitude, gradients far below the largest products
    n, nparams = 13, 6
    ops = _circuit(n, 3, nparams, 4, mix=False)
    params = np.array([[1e-3, 2e-4, 5e-2, 1e-6, 3e-3, 0.0], [0.0] * nparams])
    obs = ([0, 3, 12], [1, -1, 7], [scale, -0.5 * scale, 2.0 * scale])
    (e, g), (et, gt) = _both(n, ops, nparams, obs, params)
    assert np.max(np.abs(e - et)) <= 1e-13 * scale and np.max(np.abs(g - gt)) <= 1e-13 * scale


def test_more_sets_than_ctas():
    n, layers, batch = 12, 1, 200
    ops = workloads.hea_ansatz(n, layers)
    params = workloads.hea_params(n, layers, batch)
    (e, g), (et, gt) = _both(n, ops, params.shape[1], llgpu.ring_zz_terms(n), params)
    assert np.max(np.abs(e - et)) <= 1e-12 and np.max(np.abs(g - gt)) <= 1e-12
