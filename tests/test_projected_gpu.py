"""The projected eigensolver (trl_cuda_small_eigen_partial) where its kernels change shape.

Tolerances, relative to ||T||_2: every stage is backward stable, with an error of a modest
multiple of eps (2.2e-16) that grows at most like N <= 1024: 1e-12 for eigenvalues, 1e-11 for
residuals and orthogonality, as for the larger matrices of test_kernels_gpu.py.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _check(cuda_handle, D, kvec, bs=1, scale=1.0):
    N = D.shape[0]
    nblk = N // bs
    T = (D * scale).reshape(nblk, bs, nblk, bs).transpose(0, 2, 1, 3).copy()
    beta = torch.eye(bs, dtype=torch.float64, device="cuda") * scale
    _, evecs, ev, _ = cuda_handle.small_eigen_partial(torch.from_numpy(T).cuda(), beta, min(N, 4), 1e-8, kvec)
    w = np.linalg.eigvalsh(D)
    w = w[np.argsort(-np.abs(w), kind="stable")]
    nrm = max(np.abs(w).max(), 1e-300)
    X = evecs.cpu().numpy().transpose(0, 2, 1, 3).reshape(N, N)[:, :kvec]
    ev = ev / scale
    assert np.abs(np.abs(ev) - np.abs(w)).max() <= 1e-12 * nrm
    assert np.abs(np.sort(ev) - np.sort(w)).max() <= 1e-12 * nrm
    if kvec == 0:
        return
    assert np.abs(D @ X - X * ev[:kvec]).max() <= 1e-11 * nrm
    assert np.abs(X.T @ X - np.eye(kvec)).max() <= 1e-11


# edges of the tridiagonalisation: rows of one warp (128 apart), the last size with rows in
# registers (512) and in shared memory (624), rows in global memory beyond
@pytest.mark.parametrize("N", [3, 4, 17, 127, 128, 129, 255, 256, 257, 384, 385, 511, 512, 513, 624, 625])
def test_sizes(cuda_handle, N):
    M = np.random.default_rng(N).standard_normal((N, N))
    _check(cuda_handle, M + M.T, min(N, 24))


def test_columns_that_are_already_reduced(cuda_handle):
    """No reflector anywhere (tridiagonal and diagonal matrices), and for a part of the columns."""
    rng = np.random.default_rng(1)
    N = 200
    D = np.diag(rng.uniform(1.0, 2.0, N)) + np.diag(rng.standard_normal(N - 1), 1)
    D = np.triu(D) + np.triu(D, 1).T
    _check(cuda_handle, D, 20)
    _check(cuda_handle, np.diag(np.arange(1.0, N + 1.0)), 20)
    M = rng.standard_normal((N - 70, N - 70))
    D[70:, 70:] += M + M.T
    D[69, 70] = D[70, 69] = 0.0
    _check(cuda_handle, D, 20)


@pytest.mark.parametrize("scale", [2.0 ** 450, 2.0 ** -450])
def test_extreme_scales(cuda_handle, scale):
    M = np.random.default_rng(2).standard_normal((140, 140))
    _check(cuda_handle, M + M.T, 16, bs=4, scale=scale)


# kept vectors at the edges of the 8-vector tiles and 32-entry strips, and groups of equal
# or nearly equal eigenvalues: none, some, one of 40, all
@pytest.mark.parametrize("N,kvec", [(130, 1), (130, 7), (130, 8), (130, 9), (161, 112), (300, 256)])
def test_kept_vectors(cuda_handle, N, kvec):
    M = np.random.default_rng(kvec).standard_normal((N, N))
    _check(cuda_handle, M + M.T, kvec)


@pytest.mark.parametrize("gap", [0.0, 1e-14, 3e-11, 1e-9, 1e-6])
def test_groups_of_close_eigenvalues(cuda_handle, gap):
    rng = np.random.default_rng(3)
    Q, _ = np.linalg.qr(rng.standard_normal((150, 150)))
    lam = np.concatenate([5.0 + gap * np.arange(40), [4.0, 4.0, 3.0], rng.uniform(-1.0, 1.0, 107)])
    _check(cuda_handle, (Q * lam) @ Q.T, 48)


def test_one_eigenvalue(cuda_handle):
    _check(cuda_handle, 3.0 * np.eye(96), 16)


@pytest.mark.parametrize("N", [3, 4, 5, 6, 7, 8, 9, 10, 11, 64, 201])
def test_counts_at_exact_zeros(cuda_handle, N):
    """Integer and singular tridiagonals: pivots and products that are exactly zero at the
    points the bisection tries, repeated blocks, and entries of very different size."""
    i = np.arange(N)
    for d, e in ((np.zeros(N), np.ones(N - 1)), (2.0 * np.ones(N), -np.ones(N - 1)), (i % 3 - 1.0, (i[:-1] % 2) * 1.0), (1.0 * (i == 0), np.zeros(N - 1)),
                 (10.0 ** -(i % 20), 10.0 ** -(i[:-1] % 17)), (np.zeros(N), 1e-25 * np.ones(N - 1) + (i[:-1] == 0))):
        D = np.diag(d) + np.diag(e, 1) + np.diag(e, -1)
        _check(cuda_handle, D, 0 if N > 100 else 1)


@pytest.mark.parametrize("N", [33, 34, 35, 49, 67, 130])
@pytest.mark.parametrize("coupling", [1e-6, 1e-14, 1e-16, 1e-40])
def test_products_that_shrink_between_looks(cuda_handle, N, coupling):
    """Runs of equal diagonal entries and minute couplings: near them every row shrinks the products;
    each half ends in a different number of rows after the last group of eight."""
    d = np.where(np.arange(N) < N // 3, 1.0, 0.25 * (np.arange(N) % 2))
    D = np.diag(d) + np.diag(np.full(N - 1, coupling), 1) + np.diag(np.full(N - 1, coupling), -1)
    _check(cuda_handle, D, 0)


@pytest.mark.parametrize("N", [8, 140])
@pytest.mark.parametrize("g", [2.0 ** -70, 2.0 ** -85, 2.0 ** -98])
def test_reflectors_of_minute_norm(cuda_handle, N, g):
    """Couplings that multiply up to g^3, down to 3e-89: a column of that norm is reduced by a reflector
    whose scale, squared, is out of range."""
    D = np.diag(np.where(np.arange(N) < 6, 0.0, 0.25 * np.arange(N) / (N - 1)))
    for i, j, v in ((0, 1, 1.0), (0, 2, g), (1, 3, 1.0), (2, 3, g), (2, 4, g), (4, 5, g)):
        D[i, j] = D[j, i] = v
    _check(cuda_handle, D, 4)


@pytest.mark.parametrize("N,kvec", [(8, 8), (9, 9), (140, 139)])
@pytest.mark.parametrize("g", [2.0 ** -40, 2.0 ** -60, 2.0 ** -98])
def test_vectors_of_repeated_eigenvalues_with_minute_couplings(cuda_handle, N, kvec, g):
    """Zero diagonals behind couplings that stand for zero: no pivot of the inverse iteration, whichever
    row it comes from, is below the floor."""
    D = np.diag(np.where(np.arange(N) < 6, 0.0, 0.25 * np.arange(N) / (N - 1)))
    for i, j, v in ((0, 1, 1.0), (0, 2, g), (1, 3, 1.0), (2, 3, g), (2, 4, g), (4, 5, g)):
        D[i, j] = D[j, i] = v
    _check(cuda_handle, D, kvec)


@pytest.mark.parametrize("N", [24, 97])
@pytest.mark.parametrize("g", [1e-18, 1e-22, 1e-29])
def test_vectors_of_chains_with_minute_couplings(cuda_handle, N, g):
    """Tridiagonal already: pairs of rows with a strong coupling, minute ones between the pairs, all eigenvalues
    +1 and -1 but for the odd last row."""
    off = np.where(np.arange(N - 1) % 2 == 0, 1.0, g)
    _check(cuda_handle, np.diag(off, 1) + np.diag(off, -1), N)
