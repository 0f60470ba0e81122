"""GPU tests of the dense FP64 kernels at the edges of their blocking: the 32-row
halves of a factorisation leaf, and both tile shapes of the GEMM around the size
where the dispatch changes between them.  References and tolerances as in
test_gpu_dense.py.
"""
import numpy as np
import pytest

from gammcor_integrals_b200 import _capi
from test_gpu_dense import _spd, _vp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [31, 32, 33, 96, 97, 129])
def test_cholesky_inverse_leaf_halves(gpu_lib, n):
    import torch
    cond = 1e4
    A = _spd(n, n, cond=cond)
    At = torch.tensor(A.T.copy(), device="cuda")
    Xt = torch.full((n, n), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    _capi.check(gpu_lib.gci_cholesky_inverse(n, _vp(At), n, _vp(Xt)))
    L, X = np.tril(At.T.cpu().numpy()), Xt.T.cpu().numpy()
    Lref = np.linalg.cholesky(A)
    eps = np.finfo(float).eps
    assert np.abs(L - Lref).max() <= 50 * eps * cond * np.abs(Lref).max()
    assert np.all(np.triu(X, 1) == 0.0)
    assert np.abs(X @ L - np.eye(n)).max() <= n * eps * cond


@pytest.mark.parametrize("n,bad", [(20, 7), (64, 40), (200, 3), (200, 170)])
def test_first_nonpositive_pivot_is_reported(gpu_lib, n, bad):
    import torch
    A = _spd(n, 5, cond=10.0)
    A[bad, bad] = -1.0   # leading minor of order bad + 1 is indefinite
    At = torch.tensor(A.T.copy(), device="cuda")
    Xt = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert gpu_lib.gci_cholesky_inverse(n, _vp(At), n, _vp(Xt)) == -5   # GCI_ERR_NOT_SPD
    assert gpu_lib.gci_last_error().decode().endswith(f"info={bad + 1}")


# 128 x 128 tiles from 148 of them on, 64 x 64 below
@pytest.mark.parametrize("m,n,k", [(65, 63, 17), (1500, 1500, 40), (1601, 1537, 40)])
def test_dgemm_tile_shapes(gpu_lib, m, n, k):
    import torch
    g = torch.Generator(device="cuda").manual_seed(m)
    A = torch.randn(k, m, dtype=torch.float64, device="cuda", generator=g)
    B = torch.randn(k, n, dtype=torch.float64, device="cuda", generator=g)
    Cm = torch.randn(n, m, dtype=torch.float64, device="cuda", generator=g)
    ref = Cm - B.T @ A
    torch.cuda.synchronize()
    _capi.check(gpu_lib.gci_dgemm(m, n, k, -1.0, _vp(A), m, _vp(B), n, 1.0, _vp(Cm), m))
    bound = 1e-13 * k * float(A.abs().max()) * float(B.abs().max())
    assert float((Cm - ref).abs().max()) <= bound
