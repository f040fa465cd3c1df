"""The pipelined 5-qubit tensor-core blocks (csrc/llg_gateblock.cu) against the oracle: one tile, a
partly filled last wave, every kind of target set, groups of zeros, of subnormals and with an
infinity."""
from __future__ import annotations

import numpy as np
import pytest

import llgpu
import oracle

pytestmark = pytest.mark.gpu

# the result's largest error over its largest amplitude: an FP64 product of 64 terms rounds to a few
# 2^-53; a double-float state holds 2^-47 of each amplitude, and its 7 digits drop 2^-50 of the group
TOL = {"complex128": 2e-15, "df64": 5e-14}


@pytest.fixture(scope="module", autouse=True)
def _built(built):
    assert llgpu.device_count() > 0


def _unitary(rng):
    return np.linalg.qr(rng.normal(size=(32, 32)) + 1j * rng.normal(size=(32, 32)))[0]


@pytest.mark.parametrize("precision", ["complex128", "df64"])
@pytest.mark.parametrize("n,targets", [(12, [0, 1, 2, 3, 4]), (12, [11, 3, 7, 0, 9]), (13, [12, 11, 10, 9, 8]),
                                       (17, [0, 7, 8, 9, 16]), (20, [6, 2, 19, 13, 1]), (20, [19, 18, 17, 16, 15])])
def test_five_qubit_block(precision, n, targets):
    rng = np.random.default_rng(n + sum(targets))
    psi = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    psi[: 1 << (n - 2)] = 0.0  # whole groups of zeros
    psi /= np.linalg.norm(psi)
    st = llgpu.State(precision=precision, amps=psi)
    want = st.state()
    for _ in range(2):  # the second block reads what the first one wrote
        m = _unitary(rng)
        st.apply_matrix(targets, m)
        oracle.apply_matrix(want, n, targets, m)
    assert np.max(np.abs(st.state() - want)) <= TOL[precision] * np.max(np.abs(want))
    st.close()


def test_small_and_special_groups():
    n, targets = 12, [0, 1, 2, 3, 4]  # group g holds amplitudes 32 g .. 32 g + 31
    rng = np.random.default_rng(7)
    psi = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    scales = {1: 2.0 ** -1021, 2: 2.0 ** -1040, 3: 0.0, 4: 2.0 ** -960, 5: 2.0 ** 900}
    for g, s in scales.items():
        psi[32 * g:32 * (g + 1)] *= s
    psi[32 * 6 + 5] = np.inf
    st = llgpu.State(precision="complex128", amps=psi)
    m = _unitary(rng)
    st.apply_matrix(targets, m)
    got = st.state()
    ok = np.arange(1 << n) // 32 != 6
    clean = psi.copy()
    clean[~ok] = 0.0
    # the small groups are multiplied 2^60 up, where numpy's own products are not subnormal
    up = np.where(np.max(np.abs(clean.reshape(-1, 32)), axis=1) < 2.0 ** -900, 2.0 ** 60, 1.0)[:, None]
    want = (((m @ (clean.reshape(-1, 32) * up).T).T) / up).reshape(-1)
    assert not np.any(np.isfinite(got[~ok].real))  # an infinity times a dense row
    for g in list(scales) + [0, 7, 127]:
        sl = slice(32 * g, 32 * (g + 1))
        # relative to the group's largest amplitude, or one unit of the smallest subnormal
        bound = max(TOL["complex128"] * np.max(np.abs(want[sl])), 2.0 ** -1073)
        assert np.max(np.abs(got[sl] - want[sl])) <= bound, g
    st.close()


def _circuit(n, depth, seed):
    """Every gate kind, with sign flips on more than five qubits and lone CNOTs between layers."""
    rng = np.random.default_rng(seed)
    recs = []
    for d in range(depth):
        for q in range(n):
            u = np.linalg.qr(rng.normal(size=(2, 2)) + 1j * rng.normal(size=(2, 2)))[0]
            recs.append((llgpu.OP_U2, q, 0, 0.0, None, u) if d % 2 else (llgpu.OP_RY, q, 0, rng.uniform(0, 6)))
            recs.append((llgpu.OP_RZ, q, 0, rng.uniform(0, 6)))
        for _ in range(n // 2):
            a, b = (int(x) for x in rng.choice(n, size=2, replace=False))
            recs.append((int(rng.choice([llgpu.OP_CNOT, llgpu.OP_CZ])), a, b))
        recs.append((llgpu.OP_MCZ, 0, 0, 0.0, (1 << 7) - 1))
    return llgpu.make_ops(recs)


@pytest.mark.parametrize("precision", ["complex128", "df64"])
@pytest.mark.parametrize("n,depth", [(12, 12), (13, 8), (17, 6), (20, 4)])
def test_fused_blocks_match_oracle(precision, n, depth):
    ops = _circuit(n, depth, n)
    want = oracle.run_ops(n, ops)
    st = llgpu.State(n, precision)
    st.profile(True)
    st.apply_ops(ops)
    assert np.max(np.abs(st.state() - want)) <= 1e-12
    # the same gates as tile passes
    st.set_fusion("tile", 11)
    st.reset(n)
    st.apply_ops(ops)
    assert np.max(np.abs(st.state() - want)) <= 1e-12
    st.close()


def test_block_plans_over_many_weights():
    # more blocks than weights are held at once, in one flush
    n = 12
    ops = np.concatenate([_circuit(n, 40, 5)] * 2)
    st = llgpu.State(n, "complex128")
    st.apply_ops(ops)
    assert np.max(np.abs(st.state() - oracle.run_ops(n, ops))) <= 1e-12
    st.close()


def test_states_that_are_not_finite_keep_to_the_tile_passes():
    # a block would spread an infinity over its 32 amplitudes; the gates alone reach half of the pairs
    n = 12
    psi = np.zeros(1 << n, dtype=complex)
    psi[0], psi[5] = 1.0, np.inf
    ops = llgpu.make_ops([(llgpu.OP_RY, 3, 0, 0.7), (llgpu.OP_CNOT, 3, 4)] * 30)
    st = llgpu.State(precision="complex128", amps=psi)
    st.apply_ops(ops)
    got = st.state()
    ref = llgpu.State(precision="complex128", amps=psi)
    ref.set_fusion("tile", 12)
    ref.apply_ops(ops)
    want = ref.state()
    assert np.array_equal(np.isfinite(got), np.isfinite(want)) and np.isfinite(got).sum() > (1 << n) - 32
    st.close()
    ref.close()


def test_gates_of_norm_above_one_grow_the_state():
    # 2x2s that double the norm, far past what integers against a group's largest could hold
    n = 12
    grow = llgpu.make_ops([(llgpu.OP_U2, q % n, 0, 0.0, None, [[4.0, 0], [0, 4.0]]) for q in range(300)])
    mix = _circuit(n, 6, 3)
    st = llgpu.State(n, "complex128")
    st.apply_ops(mix)
    st.apply_ops(grow)
    st.flush()
    st.apply_ops(mix)
    got = np.ldexp(st.state().view(np.float64), -600).view(np.complex128)
    want = oracle.run_ops(n, np.concatenate([mix, mix]))
    assert np.max(np.abs(got - want)) <= 1e-12
    st.close()


def test_channels_join_blocks():
    # a density matrix of 2^12 elements: dense, diagonal and complex channels between gates, one and two targets
    # in both orders, read in the middle; the same with one pass a channel
    n = 6
    rng = np.random.default_rng(2)
    k1 = np.linalg.qr(rng.normal(size=(6, 2)) + 1j * rng.normal(size=(6, 2)))[0].reshape(3, 2, 2)
    k2 = np.linalg.qr(rng.normal(size=(12, 4)) + 1j * rng.normal(size=(12, 4)))[0].reshape(3, 4, 4)
    want = oracle.dm_zero(n)
    fused, plain = llgpu.DensityMatrix(n), llgpu.DensityMatrix(n)
    plain.state.set_fusion("tile", 12)
    for step in range(4):
        ops = _circuit(n + 2, 1, step)  # gates of every kind on the qubits that exist
        ops = ops[(ops["q0"] < n) & (ops["q1"] < n) & (ops["kind"] != llgpu.OP_MCZ)]
        want = oracle.dm_apply_ops(want, n, ops)
        channels = [(llgpu.amplitude_damping(0.1), [q]) for q in range(n)] + [(llgpu.phase_damping(0.2), [step])]
        channels += [(k1, [5 - step]), (k2, [step, 5]), (k2, [4, 0]), (llgpu.depolarizing(0.05, 2), [3, 1])]
        for dm in (fused, plain):
            dm.apply_ops(ops)
        for ks, targets in channels:
            for dm in (fused, plain):
                dm.kraus(ks, targets)
            want = oracle.kraus_apply(want, n, ks, targets)
        if step == 1:
            assert np.max(np.abs(fused.rho() - want)) <= 1e-12
    assert np.max(np.abs(fused.rho() - want)) <= 1e-12
    assert np.max(np.abs(plain.rho() - want)) <= 1e-12
    fused.close()
    plain.close()
