"""Backward error of the chained solves at the bounds that their theory gives, column by column:
max|B - Z x| / (||Z||_inf max|x|)

* refined form: the stopping rule's eps sqrt(n) in the |re| + |im| norm, a factor of two at most in
  the modulus, plus the four eps that this test's own residual may be off by;
* FP64 form: n eps, the a-priori bound of a well-pivoted factorisation without growth.

Orders at the edges of the 64-row blocks, right-hand sides at those of chains and launches."""
import numpy as np
import pytest

from pssfss_b200 import engine

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


@pytest.mark.parametrize("precision", ["fp64", "fp32r"])
@pytest.mark.parametrize("n,nrhs", [(63, 3), (64, 4), (65, 5), (128, 9), (193, 64), (200, 65), (1000, 130), (1500, 46)])
def test_backward_error(n, nrhs, precision):
    rng = np.random.default_rng(1000 * n + nrhs)
    Z = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 2 * np.sqrt(n) * np.eye(n)
    B = rng.standard_normal((n, nrhs)) + 1j * rng.standard_normal((n, nrhs))
    X, st = engine.lu_solve(Z, B, precision)
    assert st == 0
    back = np.max(np.abs(B - Z @ X), axis=0) / (np.max(np.sum(np.abs(Z), axis=1)) * np.max(np.abs(X), axis=0))
    assert np.max(back) <= (2 * np.sqrt(n) + 4 if precision == "fp32r" else n) * EPS
