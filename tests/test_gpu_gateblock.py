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
