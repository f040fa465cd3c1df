"""Expectations of complex128 states with an infinite amplitude, or one whose square is: terms that are even there leave it
out.  (The compensated sums of the other formats turn an infinity into NaN.)"""
from __future__ import annotations

import numpy as np
import pytest

import llgpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built(built):
    assert llgpu.device_count() > 0


@pytest.mark.parametrize("value", [np.inf, 1e200])
@pytest.mark.parametrize("n", [3, 9, 14])
def test_even_terms_leave_it_out(n, value):
    psi = np.full(1 << n, 2.0 ** (-n / 2), dtype=complex)
    psi[0] = value  # every parity is even at 0
    st = llgpu.State(precision="complex128", amps=psi)
    a, b, c = list(range(n)), [-1] * (n - 1) + [0], [1.0] * n
    assert st.expect_zz(a, b, c) == np.inf
    assert st.expect_zz(a, b, [1.0] + [0.5] * (n - 1)) == np.inf  # two classes
    st.close()
