"""Expectations of Z and ZZ sums, whose kernel counts odd parities by rows of 256 amplitudes: terms inside a row,
across it and above it, one to four coefficient classes, states smaller than a row and of several rows a block."""
from __future__ import annotations

import numpy as np
import pytest

import llgpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built(built):
    assert llgpu.device_count() > 0


@pytest.mark.parametrize("precision,tol", [("complex128", 1e-13), ("df64", 1e-12), ("complex64", 1e-5)])
@pytest.mark.parametrize("n", [1, 4, 8, 9, 13, 21])
@pytest.mark.parametrize("classes", [1, 4])
def test_against_the_state(n, classes, precision, tol):
    rng = np.random.default_rng(100 * n + classes)
    psi = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    psi /= np.linalg.norm(psi)
    terms = [(q, -1) for q in range(n)] + [(a, b) for a in range(n) for b in range(n) if a != b]
    rng.shuffle(terms)
    terms = terms[:40]
    coef = [float(rng.integers(classes)) - 1.5 for _ in terms]
    st = llgpu.State(precision=precision, amps=psi)
    p = np.abs(psi) ** 2
    i = np.arange(1 << n)
    want = 0.0
    for (a, b), c in zip(terms, coef):
        odd = (i >> a) & 1 if b < 0 else ((i >> a) ^ (i >> b)) & 1
        want += c * float(np.sum(p * (1 - 2 * odd)))
    got = st.expect_zz([t[0] for t in terms], [t[1] for t in terms], coef)
    # the terms' sum of sizes bounds the value; an amplitude's weight is a whole number of at most 40
    assert abs(got - want) <= tol * sum(abs(c) for c in coef)
    assert abs(st.expect_zz([t[0] for t in terms], [t[1] for t in terms], coef) - got) == 0.0  # the same sums again
