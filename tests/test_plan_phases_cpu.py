"""Carried phases under long runs of CNOTs: the tile plan pushes them through the CNOTs, which multiplies the roundings of
their moduli; run by numpy against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import llgpu
import oracle
from llgpu import OP_CNOT, OP_RZ, OP_RY, OP_RX, make_ops
from planexec import execute

pytestmark = pytest.mark.usefixtures("built")


def circuit(n, cnots, seed):
    rng = np.random.default_rng(seed)
    recs = [(k, q, 0, float(rng.uniform(0.2, 3))) for q in range(n) for k in (OP_RY, OP_RZ)]
    for i in range(cnots):
        recs.append((OP_CNOT, *(int(x) for x in rng.choice(n, size=2, replace=False))))
        if i % 200 == 100:
            recs.append((OP_RX, int(rng.integers(n)), 0, 0.7))
    return make_ops(recs)


@pytest.mark.parametrize("tables", [False, True])
@pytest.mark.parametrize("n,tile,cnots", [(2, 2, 400), (5, 5, 600), (8, 8, 1500), (9, 7, 1000)])
def test_many_cnots(n, tile, cnots, tables):
    ops = circuit(n, cnots, n)
    psi = np.zeros(1 << n, dtype=complex)
    psi[0] = 1.0
    plan = llgpu.plan_export(n, ops, tile, zyz=True, tables=tables)
    c = plan[1]["c"]
    assert np.all(np.isfinite(c)) and np.max(np.abs(c)) < 16.0
    got = execute(psi, n, *plan)
    # a rounding of a phase and of an amplitude a CNOT
    assert np.max(np.abs(got - oracle.run_ops(n, ops))) <= 2.0 ** -53 * 4 * cnots
