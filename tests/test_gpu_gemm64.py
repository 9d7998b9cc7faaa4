"""The FP64 factorisation's update kernel (``k_gemm64``) at the edges of its 64 x 64 tiles and
8-deep slices, and on a caller's matrix that starts on an 8-byte boundary only.

Backward error ||P A - L U|| / ||A|| against LAPACK's on the same matrix: at most 10 times it
(both are a small multiple of the unit roundoff; the factor covers another summation order)."""
import ctypes

import numpy as np
import pytest
import scipy.linalg as sl
import torch

from pssfss_b200 import engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("n", [17, 63, 64, 65, 80, 129, 200, 513, 1000])
def test_fp64_factor_against_lapack(n, shift):
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    buf = torch.zeros(2 * n * n + 2, dtype=torch.float64, device="cuda")
    a = buf[shift:shift + 2 * n * n]
    a.copy_(torch.from_numpy(np.ascontiguousarray(A).view(np.float64).ravel()))
    ipiv = torch.zeros(n, dtype=torch.int32, device="cuda")
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    p = ctypes.c_void_p
    torch.cuda.synchronize()
    rc = engine.lib().pss_lu_factor_noalloc(n, p(a.data_ptr()), n, p(ipiv.data_ptr()), p(info.data_ptr()),
                                            p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert rc == 0 and int(info) == 0
    LU = a.cpu().numpy().view(np.complex128).reshape(n, n)
    PA = A.copy()
    for k, q in enumerate(ipiv.cpu().numpy()):
        PA[[k, q]] = PA[[q, k]]
    back = np.linalg.norm(PA - (np.tril(LU, -1) + np.eye(n)) @ np.triu(LU)) / np.linalg.norm(A)
    lu, piv = sl.lu_factor(A)
    PL = A.copy()
    for k, q in enumerate(piv):
        PL[[k, q]] = PL[[q, k]]
    back_l = np.linalg.norm(PL - (np.tril(lu, -1) + np.eye(n)) @ np.triu(lu)) / np.linalg.norm(A)
    assert back < 10 * back_l, (back, back_l)
