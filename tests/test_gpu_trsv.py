"""Chained triangular solves at the edges of their 64-row blocks and of their groups of right-hand
sides (four to a chain, sixteen chains to a launch), in both precisions.

Backward error of each column, max|B - Z x| / (||Z||_inf max|x|), at most 2 eps sqrt(n) in the
refined form (its stopping rule) and n eps in the FP64 form (the a-priori bound of a
well-pivoted factorisation without growth)."""
import numpy as np
import pytest

from pssfss_b200 import engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32r"])
@pytest.mark.parametrize("n,nrhs", [(1, 1), (63, 3), (64, 4), (65, 5), (128, 9), (193, 64), (200, 65), (1000, 130),
                                    (1500, 46)])
def test_solve_blocks_and_right_hand_sides(n, nrhs, precision):
    rng = np.random.default_rng(1000 * n + nrhs)
    Z = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 2 * np.sqrt(n) * np.eye(n)
    B = rng.standard_normal((n, nrhs)) + 1j * rng.standard_normal((n, nrhs))
    X, st = engine.lu_solve(Z, B, precision)
    assert st == 0
    back = np.max(np.abs(B - Z @ X), axis=0) / (np.max(np.sum(np.abs(Z), axis=1)) * np.max(np.abs(X), axis=0))
    eps = 1.1102230246251565e-16
    assert np.max(back) <= (2 * np.sqrt(n) if precision == "fp32r" else n) * 4 * eps
