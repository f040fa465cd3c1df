"""Complex128 trajectories under weak noise, whose gates take one pass each with the Kraus factors carried:
jump logs bit for bit against the oracle's, <Z_0> and margins to the bounds of the general kernel.  The
cases meet every kind of pass, a cluster's exchanges of its top qubit, gates that keep the general code,
jumps (the seeds' runs have some), factors far from one, several trajectories per CTA and uniforms drawn
in more than one chunk."""
from __future__ import annotations

import numpy as np
import pytest

import llgpu
import oracle
from llgpu import OP_CNOT, OP_CZ, OP_H, OP_MCZ, OP_RX, OP_RY, OP_RZ, OP_X, make_ops

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built(built):
    assert llgpu.device_count() > 0


def circuit(n, gates, seed, general=0):
    rng = np.random.default_rng(seed)
    recs = []
    for i in range(gates):
        kind = int(rng.integers(7))
        q = int(rng.integers(n))
        if general and i % general == 0:
            if rng.integers(2):
                recs.append((OP_X, q))
            else:
                qs = rng.choice(n, 3, replace=False)
                recs.append((OP_MCZ, 0, 0, 0.0, int(sum(1 << int(x) for x in qs))))
        elif kind < 3:
            recs.append(((OP_RX, OP_RY, OP_RZ)[kind], q, 0, float(rng.uniform(0, 6.28))))
        elif kind == 3:
            recs.append((OP_H, q))
        else:
            a, b = (int(x) for x in rng.choice(n, 2, replace=False))
            recs.append((OP_CZ if kind == 4 else OP_CNOT, a, b))
    return make_ops(recs)


def check(n, ops, gamma, lam, seed, count):
    sites = llgpu.noise_sites(ops)
    z, j, log, margin = llgpu.traj_run(n, ops, gamma, lam, seed, count, 0, "fp64", log=True)
    zo, jo, logo, margin_o = oracle.traj_run(n, ops, gamma, lam, seed, 0, count, log_sites=sites)
    assert margin_o > 1e-12, "a near-tie decision: choose another seed"
    assert np.array_equal(log, logo)
    assert np.array_equal(j, jo)
    assert np.max(np.abs(z - zo)) <= 1e-10
    assert abs(margin - margin_o) <= 1e-9
    return j


@pytest.mark.parametrize("n", [3, 4, 5, 6, 7, 9, 12, 13, 14])
@pytest.mark.parametrize("general", [0, 6])
def test_weak_noise_jumps_bit_exact(n, general):
    j = check(n, circuit(n, 150, seed=10 * n + general, general=general), 0.03, 0.02, seed=5 + n, count=24)
    assert j.sum() > 0


@pytest.mark.parametrize("n,cluster,threads", [(4, 2, 32), (8, 2, 64), (11, 2, 512), (13, 2, 96 * 4), (10, 1, 96), (13, 1, 1024)])
def test_shapes_agree(n, cluster, threads):
    ops = circuit(n, 120, seed=n, general=9)
    z, j, _ = llgpu.Traj(n, ops, 0.02, 0.03, 40, "fp64").launch(6, 40)
    z2, j2, _ = llgpu.Traj(n, ops, 0.02, 0.03, 40, "fp64", cluster, threads).launch(6, 40)
    assert np.array_equal(j, j2) and np.max(np.abs(z - z2)) <= 1e-10


@pytest.mark.parametrize("n,threads", [(13, 32), (13, 64), (12, 32), (9, 256)])
def test_factors_of_looped_qubits_are_applied(n, threads):
    # all qubits first, then runs of gates on the lowest ones: the others' factors go before each run
    rng = np.random.default_rng(n)
    recs = []
    for _ in range(3):
        for q in range(n):
            recs += [(OP_RX, q, 0, float(rng.uniform(0, 6.28))), (OP_CNOT, q, (q + 1) % n)]
        for _ in range(12):
            recs += [(OP_RY, int(rng.integers(3)), 0, float(rng.uniform(0, 6.28))), (OP_CNOT, 0, 2)]
    ops = make_ops(recs)
    z, j, _ = llgpu.Traj(n, ops, 0.03, 0.02, 24, "fp64", 1, threads).launch(6, 24)
    zo, jo, _, margin_o = oracle.traj_run(n, ops, 0.03, 0.02, 6, 0, 24, log_sites=llgpu.noise_sites(ops))
    assert margin_o > 1e-12 and np.array_equal(j, jo) and np.max(np.abs(z - zo)) <= 1e-10


def test_many_gates_on_few_qubits():
    # the factors of two qubits grow for 700 gates, past the spread that the planner allows
    n = 6
    rng = np.random.default_rng(3)
    recs = []
    for _ in range(350):
        recs += [(OP_RZ, int(rng.integers(2)), 0, 0.4), (OP_RX, int(rng.integers(2)), 0, 0.01)]
    check(n, make_ops(recs), 0.1, 0.02, seed=4, count=8)


def test_without_noise_and_without_gates():
    check(9, circuit(9, 60, seed=1), 0.0, 0.0, seed=2, count=4)
    z, j, _, margin = llgpu.traj_run(9, make_ops([]), 0.01, 0.01, 1, 3, 0, "fp64", log=True)
    assert np.array_equal(z, np.ones(3)) and j.sum() == 0 and margin == 1.0


def test_several_trajectories_per_cta():
    ops = circuit(14, 30, seed=8)
    z, j, _, _ = llgpu.traj_run(14, ops, 0.05, 0.05, 3, 400, 0, "fp64", log=True)
    z2, j2, _, _ = llgpu.traj_run(14, ops, 0.05, 0.05, 3, 40, 360, "fp64", log=True)
    assert np.array_equal(z[360:], z2) and np.array_equal(j[360:], j2)
