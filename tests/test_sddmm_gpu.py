"""SDDMM and eigenvalue adjoint over the forms their kernel distinguishes: columns per lane and
lanes per row (k odd and even, below, at and above the 16 of one round), coefficients by value
(k <= 256) and from memory, rows of 0 entries to more than a warp sweeps, X aligned to 8 bytes only.

Tolerance: each output sums k products of three factors in 64 bits, in some order: an error of at
most (k + 2) eps times the sum of magnitudes (k - 1 additions, 2 multiplications, and the last
rounding); 2 (k + 2) eps leaves room for the reference's own.
"""
import numpy as np
import pytest
import torch

from trl_b200 import native
from trl_b200 import problems as P

from test_kernels_gpu import _long_row_csr, dev, host

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 8, 9, 16, 17, 18, 33, 256, 300])
@pytest.mark.parametrize("offset", [0, 1, 2])
def test_sddmm_forms(cuda_handle, k, offset):
    rng = np.random.default_rng(k)
    for A in (_long_row_csr(rng, 700), P.laplace2d(9), P.diagonal(3)):
        X = rng.standard_normal((A.n, k))
        w = rng.uniform(0.5, 2.0, k)
        Xd = torch.zeros(A.n * k + offset, dtype=torch.float64, device="cuda")[offset:].view(A.n, k)
        Xd.copy_(torch.from_numpy(X))
        rows = A.row_indices()
        terms = w * X[rows] * X[A.colind]
        bound = 2 * (k + 2) * EPS * np.abs(terms).sum(1)
        Ad = native.DeviceCSRTensors.from_host(A)
        out = torch.full((A.nnz,), float("nan"), dtype=torch.float64, device="cuda")
        cuda_handle.sddmm(Ad, Xd, dev(w), out)
        assert np.all(np.abs(host(out) - terms.sum(1)) <= bound)
        out.fill_(float("nan"))
        cuda_handle.eigen_adjoint(Ad, Xd, np.arange(1.0, k + 1.0), w, out)
        assert np.all(np.abs(host(out) - terms.sum(1)) <= bound)


@pytest.mark.parametrize("k", [1, 16, 256, 300])
def test_adjoint_is_complete_on_return(k):
    """Behind work that keeps the stream busy for milliseconds, the gradient is there for any stream when
    the call returns."""
    A = P.laplace2d(9)
    X = torch.randn((A.n, k), dtype=torch.float64, device="cuda")
    Ad = native.DeviceCSRTensors.from_host(A)
    out = torch.empty(A.nnz, dtype=torch.float64, device="cuda")
    a = torch.randn((4096, 4096), dtype=torch.float32, device="cuda")
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    h = native.Handle(0, stream=s)
    try:
        with torch.cuda.stream(s):
            for _ in range(20):
                a @ a
        h.eigen_adjoint(Ad, X, np.arange(1.0, k + 1.0), np.ones(k), out)
        assert s.query()
    finally:
        torch.cuda.synchronize()
        h.close()


def _band(n, width):
    cols = np.sort((np.arange(n)[:, None] + np.arange(width)) % n, axis=1)
    return P._from_coo(n, np.repeat(np.arange(n), width), cols.ravel(), np.ones(n * width))


@pytest.mark.parametrize("n,width", [(4096, 11), (4097, 11), (4097, 12), (8192, 7), (8193, 7), (8193, 8), (8193, 15), (8193, 16), (9001, 1), (500, 300)])
@pytest.mark.parametrize("k,offset", [(1, 0), (3, 0), (6, 0), (8, 1), (8, 2), (34, 0), (62, 0), (66, 0), (5, 0), (20, 0)])
def test_sddmm_either_side_of_the_choice_of_kernel(cuda_handle, n, width, k, offset):
    rng = np.random.default_rng(n + k)
    A = _band(n, width)
    X = rng.standard_normal((n, k))
    w = rng.uniform(0.5, 2.0, k)
    Xd = torch.zeros(n * k + offset, dtype=torch.float64, device="cuda")[offset:].view(n, k)
    Xd.copy_(torch.from_numpy(X))
    terms = w * X[A.row_indices()] * X[A.colind]
    bound = 2 * (k + 2) * EPS * np.abs(terms).sum(1)
    Ad = native.DeviceCSRTensors.from_host(A)
    out = torch.full((A.nnz,), float("nan"), dtype=torch.float64, device="cuda")
    cuda_handle.sddmm(Ad, Xd, dev(w), out)
    assert np.all(np.abs(host(out) - terms.sum(1)) <= bound)
    out.fill_(float("nan"))
    cuda_handle.eigen_adjoint(Ad, Xd, np.arange(1.0, k + 1.0), w, out)
    assert np.all(np.abs(host(out) - terms.sum(1)) <= bound)
