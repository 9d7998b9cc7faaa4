"""Distance of the solver's answers from the exact ones: on matrices like a moment matrix (an
oscillating kernel that decays with distance, heavier on the diagonal) the mean relative error of
both precision forms is no larger than LAPACK's own FP64 solve's on the same systems.

The exact solution is LAPACK's, refined with residuals in extended precision (64-bit significand:
two steps leave some 1e-19).  Sums that round twice at the running value's size for each complex
product were a fifth further off than LAPACK at order 300 (FP64) and 1501 (refined)."""
import numpy as np
import pytest
import scipy.linalg as sl

from pssfss_b200 import engine

pytestmark = pytest.mark.gpu


def system(n, nrhs, seed):
    rng = np.random.default_rng(seed)
    r = rng.uniform(0, 1, (n, 2))
    d = np.hypot(r[:, None, 0] - r[None, :, 0], r[:, None, 1] - r[None, :, 1])
    A = np.exp(-3j * d) / (d + 0.03) * (1 + 0.3 * rng.standard_normal((n, n))) / np.sqrt(n)
    A[np.arange(n), np.arange(n)] += 6 + 2j * rng.standard_normal(n)
    return A, rng.standard_normal((n, nrhs)) + 1j * rng.standard_normal((n, nrhs))


@pytest.mark.parametrize("n,nrhs,seeds", [(300, 4, 24), (736, 4, 6), (1501, 5, 3)])
def test_no_further_from_exact_than_lapack(n, nrhs, seeds):
    err = {"lapack": [], "fp64": [], "fp32r": []}
    for seed in range(seeds):
        A, B = system(n, nrhs, seed)
        lu = sl.lu_factor(A)
        X0 = sl.lu_solve(lu, B)
        Al, X = A.astype(np.clongdouble), X0.astype(np.clongdouble)
        for _ in range(2):
            R = B - np.stack([(Al * X[None, :, j]).sum(axis=1) for j in range(nrhs)], axis=1)
            X = X + sl.lu_solve(lu, R.astype(complex))
        norm = np.linalg.norm(X.astype(complex))
        for name, Y in (("lapack", X0), ("fp64", engine.lu_solve(A, B, "fp64")[0]),
                        ("fp32r", engine.lu_solve(A, B, "fp32r")[0])):
            err[name].append(np.linalg.norm((Y - X).astype(complex)) / norm)
    mean = {k: float(np.mean(v)) for k, v in err.items()}
    assert mean["fp64"] <= mean["lapack"] and mean["fp32r"] <= mean["lapack"], mean
