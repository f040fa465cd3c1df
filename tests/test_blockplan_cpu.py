"""The plan of dense 5-qubit blocks (csrc/llg_blockplan.cpp), run by numpy, against the oracle: every
gate kind, targets and controls in both orders, wide sign flips, diagonal gates that change places,
the lists that have no block plan."""
from __future__ import annotations

import numpy as np
import pytest

import llgpu
import oracle
import workloads
from llgpu import OP_CNOT, OP_CZ, OP_H, OP_MCZ, OP_RX, OP_RY, OP_RZ, OP_U2, OP_X

pytestmark = pytest.mark.usefixtures("built")


def _apply(psi, n, g, qubits):
    """One gate of a step; `qubits` maps the gate's bits to global qubits."""
    idx = np.arange(1 << n)
    if g["kind"] == 0:
        q = qubits[g["q0"]]
        m = (g["m"][0::2] + 1j * g["m"][1::2]).reshape(2, 2)
        v = psi.reshape(-1, 2, 1 << q)
        return np.einsum("ab,xby->xay", m, v).reshape(-1)
    if g["kind"] == 1:
        c, t = qubits[g["q0"]], qubits[g["q1"]]
        return psi[np.where(idx >> c & 1, idx ^ (1 << t), idx)]
    mask = sum(1 << qubits[b] for b in range(len(qubits)) if int(g["mask"]) >> b & 1)
    return np.where(idx & mask == mask, -psi, psi)


def run_plan(n, ops):
    steps, gates = llgpu.block_plan_export(n, ops)
    psi = np.zeros(1 << n, dtype=complex)
    psi[0] = 1.0
    for s in steps:
        qubits = list(s["q"]) if s["is_block"] else list(range(n))
        if s["is_block"]:
            assert sorted(set(qubits)) == qubits and 0 <= qubits[0] and qubits[-1] < n
        for g in gates[s["gate_begin"]:s["gate_begin"] + s["ngates"]]:
            psi = _apply(psi, n, g, qubits)
    return psi, steps, gates


def _random_ops(n, count, seed):
    rng = np.random.default_rng(seed)
    recs = []
    for _ in range(count):
        k = int(rng.choice([OP_H, OP_X, OP_RX, OP_RY, OP_RZ, OP_CNOT, OP_CZ, OP_MCZ, OP_U2]))
        a, b = (int(x) for x in rng.choice(n, size=2, replace=False))
        if k in (OP_CNOT, OP_CZ):
            recs.append((k, a, b))
        elif k == OP_MCZ:
            qs = rng.choice(n, size=int(rng.integers(1, 9)), replace=False)
            recs.append((k, int(qs[0]), 0, 0.0, sum(1 << int(q) for q in qs)))
        elif k == OP_U2:
            u = np.linalg.qr(rng.normal(size=(2, 2)) + 1j * rng.normal(size=(2, 2)))[0]
            recs.append((k, a, 0, 0.0, None, u * (0.5 if rng.random() < 0.2 else 1.0)))
        else:
            recs.append((k, a, 0, float(rng.uniform(0, 7))))
    return llgpu.make_ops(recs)


@pytest.mark.parametrize("n,ops", [(12, workloads.layered_rotations(12, 5)), (13, workloads.hea_ansatz(13, 4)),
                                   (12, workloads.mixed_h_cnot(12, 300)), (14, workloads.mixed_batch(1, 14, 14, 200)[1]),
                                   (12, llgpu.make_ops([(OP_H, 3)])), (12, llgpu.make_ops([(OP_CNOT, 11, 0)]))],
                         ids=["layered", "hea", "h_cnot", "mixed", "one_gate", "one_cnot"])
def test_block_plan_matches_oracle(n, ops):
    if (ops["param"] >= 0).any():
        ops = workloads.bind_params(ops, workloads.hea_params(13, 4, 1)[0])
    got, _, _ = run_plan(n, ops)
    assert np.max(np.abs(got - oracle.run_ops(n, ops))) <= 1e-12


@pytest.mark.parametrize("seed", range(8))
def test_block_plan_of_random_gates(seed):
    n = 12 + seed % 2
    ops = _random_ops(n, 120, seed)
    got, _, _ = run_plan(n, ops)
    assert np.max(np.abs(got - oracle.run_ops(n, ops))) <= 1e-12


def test_block_plan_holds_every_gate_once():
    n = 12
    ops = _random_ops(n, 200, 99)
    _, steps, gates = run_plan(n, ops)
    assert steps["ngates"].sum() == len(gates)
    assert np.isin(ops["kind"], [OP_CNOT]).sum() == (gates["kind"] == 1).sum()
    assert np.isin(ops["kind"], [OP_CZ, OP_MCZ]).sum() == (gates["kind"] == 2).sum()


def test_lists_without_a_block_plan():
    with pytest.raises(ValueError):
        llgpu.block_plan_export(11, llgpu.make_ops([(OP_H, 0)]))
    with pytest.raises(ValueError):  # a norm above 1 would outgrow the weights' range
        llgpu.block_plan_export(12, llgpu.make_ops([(OP_U2, 0, 0, 0.0, None, [[2, 0], [0, 1]])]))
    with pytest.raises(ValueError):
        llgpu.block_plan_export(12, llgpu.make_ops([(OP_H, 12)]))
    steps, gates = llgpu.block_plan_export(12, llgpu.make_ops([]))
    assert len(steps) == 0 and len(gates) == 0
