"""The kernels of a Lanczos step that add their partial sums up themselves and keep the block in
registers between the passes of a CholQR: row counts at the edges of their tiles, of a group of CTAs,
and of the switch to a second kernel; repeated calls (the ticket counters start at zero again);
blocks aligned to one element only; breakdowns.

Tolerances: sums of n products in 64 bits in any order, n eps sum|terms| (as in test_kernels_gpu.py,
1e-12 of the magnitude for n <= 300,000); CholQR2 leaves |Q^T Q - I| and |Q R - X| at a modest multiple
of the storage's eps (2.2e-16, 6e-8), held to 1e-13 and 1e-6 of the magnitude.
"""
import numpy as np
import pytest
import torch

from trl_b200 import native

from test_kernels_gpu import BS, DT, as_dt, close, dev, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bs", BS)
@pytest.mark.parametrize("dtype", DT)
@pytest.mark.parametrize("n", [1, 255, 257, 512 * 32, 512 * 32 + 1, 131072, 131073])
def test_single_dot_rows(cuda_handle, bs, dtype, n):
    rng = np.random.default_rng(n + bs)
    X, Y = (as_dt(rng.standard_normal((n, bs)), dtype) for _ in range(2))
    Xd, Yd = dev(X, dtype), dev(Y, dtype)
    ref, scale = X.T @ Y, (np.abs(X).T @ np.abs(Y)).max()
    first = None
    for _ in range(3):
        C = torch.full((1, bs, bs), float("nan"), dtype=torch.float64, device="cuda")
        cuda_handle.block_dot(Xd[None], Yd, C)
        close(host(C)[0], ref, scale)
        first = C if first is None else first
        assert torch.equal(C, first)  # one order of additions, whichever CTA adds


@pytest.mark.parametrize("bs", BS)
@pytest.mark.parametrize("dtype", DT)
@pytest.mark.parametrize("passes", [1, 2, 3, 4])
@pytest.mark.parametrize("n,offset", [(16, 0), (33, 0), (4099, 1), (70001, 0)])
def test_cholqr_passes(cuda_handle, bs, dtype, passes, n, offset):
    rng = np.random.default_rng(n + bs)
    X = as_dt(rng.standard_normal((n, bs)) @ (np.eye(bs) + 0.1 * rng.standard_normal((bs, bs))), dtype)
    Xd = torch.zeros(n * bs + offset, dtype=dtype, device="cuda")[offset:].view(n, bs)
    Xd.copy_(dev(X, dtype))
    G0 = dev(X.T @ X)
    R = torch.full((bs, bs), float("nan"), dtype=torch.float64, device="cuda")
    cuda_handle.cholqr_gram(Xd, passes, R, G0)
    cuda_handle.sync()
    Q, Rh = host(Xd), host(R)
    eps = 1e-13 if dtype == torch.float64 else 1e-6
    assert np.array_equal(np.tril(Rh, -1), np.zeros((bs, bs)))
    assert np.abs(Q.T @ Q - np.eye(bs)).max() < (eps if passes > 1 else 100 * eps)
    assert np.abs(Q @ Rh - X).max() < eps * np.abs(X).max()


@pytest.mark.parametrize("bs", BS)
@pytest.mark.parametrize("dtype", DT)
@pytest.mark.parametrize("passes", [1, 2, 3, 4])
def test_cholqr_factor_in_place_of_its_gram_matrix(cuda_handle, bs, dtype, passes):
    n = 300001  # more CTAs than are resident at once
    X = as_dt(np.random.default_rng(bs).standard_normal((n, bs)), dtype)
    Xd, Yd = dev(X, dtype), dev(X, dtype)
    G0 = torch.empty((1, bs, bs), dtype=torch.float64, device="cuda")
    cuda_handle.block_dot(Xd[None], Xd, G0)
    R = torch.empty_like(G0)
    cuda_handle.cholqr_gram(Xd, passes, R, G0)
    for shift in {0, bs * bs - 1}:  # R over all of G0, and over its last entry alone
        Z = Yd.clone()
        both = torch.zeros(2 * bs * bs, dtype=torch.float64, device="cuda")
        both[: bs * bs] = G0.view(-1)
        cuda_handle.cholqr_gram(Z, passes, both[shift:], both)
        cuda_handle.sync()
        assert torch.equal(Z, Xd)
        assert torch.equal(both[shift : shift + bs * bs].view_as(R), R)


@pytest.mark.parametrize("bs", BS)
@pytest.mark.parametrize("columns", ["all", "first", "last"])
@pytest.mark.parametrize("exponent", [-520, -500, 480])
def test_cholqr_of_columns_at_the_ends_of_the_range(cuda_handle, bs, columns, exponent):
    """2^-520: norms whose squares are subnormal, with 42 bits left of the Gram matrix; the second pass makes up
    for them. Held to 1e-12: eps times the columns' condition (below 10) and the rows' sums."""
    n = 300
    scale = np.ones(bs)
    scale[{"all": slice(None), "first": slice(0, 1), "last": slice(bs - 1, bs)}[columns]] = 2.0 ** exponent
    X = np.random.default_rng(bs).standard_normal((n, bs))
    Xd = dev(X * scale, torch.float64)
    R = torch.full((bs, bs), float("nan"), dtype=torch.float64, device="cuda")
    cuda_handle.cholqr(Xd, 2, R)
    cuda_handle.sync()
    Q, Rh = host(Xd), host(R) / scale  # R of X itself
    assert np.abs(Q.T @ Q - np.eye(bs)).max() < 1e-12
    assert np.abs(Q @ Rh - X).max() < 1e-12 * np.abs(X).max()


@pytest.mark.parametrize("bs", BS)
@pytest.mark.parametrize("passes", [1, 2])
def test_cholqr_breakdown_leaves_block_and_factor(cuda_handle, bs, passes):
    X = torch.randn((1000, bs), dtype=torch.float64, device="cuda")
    R = torch.full((bs, bs), 7.0, dtype=torch.float64, device="cuda")
    G0 = -torch.eye(bs, dtype=torch.float64, device="cuda")
    Y = X.clone()
    cuda_handle.cholqr_gram(Y, 1, R, G0)
    with pytest.raises(native.TrlError) as e:
        cuda_handle.sync()
    assert e.value.status == native.TRL_ECHOLESKY
    assert torch.equal(X, Y) and torch.all(R == 7.0)
    if passes == 2:  # the second pass works from the block itself
        R.copy_(torch.eye(bs))
        cuda_handle.cholqr_gram(Y, 2, R, G0)
        with pytest.raises(native.TrlError):
            cuda_handle.sync()
        close(host(Y).T @ host(Y), np.eye(bs), 1.0, 1e-12)
        close(host(Y) @ host(R), host(X), host(X.abs()).max(), 1e-12)


@pytest.mark.parametrize("bs", BS)
@pytest.mark.parametrize("dtype", DT)
@pytest.mark.parametrize("n,nblk", [(40, 1), (353, 3), (2368, 9), (2369, 5), (8192, 17), (8193, 2), (65536, 2), (65537, 2)])
def test_projections_at_the_edges_of_one_launch(cuda_handle, bs, dtype, n, nblk):
    """Rows at the edges of a CTA's share and of the range of the one-launch projection, blocks at those
    of a warp's: the if-needed projection with one and two passes, and the sketch's with a threshold it
    misses and one it exceeds, against numpy's Gram-Schmidt. n eps sum|terms| <= 1e-12 of the
    magnitude in 64 bits, the storage's rounding (2e-6) in 32."""
    if nblk * bs > n:
        nblk = n // bs
    rng = np.random.default_rng(n + bs)
    Vf = as_dt(np.linalg.qr(rng.standard_normal((n, nblk * bs)))[0], dtype)
    V = np.ascontiguousarray(Vf.reshape(n, nblk, bs).transpose(1, 0, 2))
    eps = 1e-12 if dtype == torch.float64 else 2e-6
    Vd = dev(V, dtype)
    for size in (100.0, 1e-3):  # components along V: two passes, one pass
        w = as_dt(Vf @ rng.standard_normal((nblk * bs, bs)) * size + rng.standard_normal((n, bs)), dtype)
        w1 = w - Vf @ (Vf.T @ w)
        lost = np.any((w1 * w1).sum(0) < 0.5 * (w * w).sum(0))
        ref = w1 - Vf @ (Vf.T @ w1) if lost else w1
        for _ in range(2):
            Wd = dev(w, dtype)
            G = torch.full((bs, bs), float("nan"), dtype=torch.float64, device="cuda")
            cuda_handle.project_out(Vd, Wd, native.TRL_CGS_IFNEEDED, G)
            close(host(Wd), ref, np.abs(w).max(), eps)
            close(host(G), host(Wd).T @ host(Wd), max(np.abs(host(G)).max(), 1e-300), 1e-10)
        S = as_dt(sum(V[j] @ (rng.standard_normal((bs, bs)) / np.sqrt(bs)) for j in range(nblk)), dtype)
        est = np.linalg.norm(S.T @ w) / np.linalg.norm(w)
        for thr, out in ((est * 100, w), (est / 100, ref)):
            Wd = dev(w, dtype)
            G = torch.full((bs, bs), float("nan"), dtype=torch.float64, device="cuda")
            cuda_handle.project_out_sketch(Vd, Wd, dev(S, dtype), thr, G)
            close(host(Wd), out, np.abs(w).max(), eps)
            close(host(G), host(Wd).T @ host(Wd), max(np.abs(host(G)).max(), 1e-300), 1e-10)
    cuda_handle.sync()


@pytest.mark.parametrize("dtype", DT)
@pytest.mark.parametrize("n", [1, 15, 17, 48, 63, 65, 113, 127, 129, 3584, 3585, 3601, 20011])
@pytest.mark.parametrize("nblk", [1, 2, 4, 5, 9])
def test_wide_blocks_at_tile_edges(cuda_handle, dtype, n, nblk):
    # 16 columns: tiles of 64 (FP64) and 128 (FP32) rows in pieces of 16, updates of 8 and 24 rows per warp
    bs = 16
    rng = np.random.default_rng(n + nblk)
    V, W = (as_dt(rng.standard_normal(s) / np.sqrt(n), dtype) for s in ((nblk, n, bs), (n, bs)))
    # n rows of a larger block, NaN behind them
    Vd, Wd = (torch.full((m, bs), float("nan"), dtype=dtype, device="cuda") for m in (nblk * n + 8, n + 8))
    Vd[: nblk * n].copy_(dev(V, dtype).view(-1, bs))
    Wd[:n].copy_(dev(W, dtype))
    Vd, Wd = Vd[: nblk * n].view(nblk, n, bs), Wd[:n]
    C = torch.full((nblk, bs, bs), float("nan"), dtype=torch.float64, device="cuda")
    cuda_handle.block_dot(Vd, Wd, C)
    ref = np.einsum("jnb,nc->jbc", V, W)
    close(host(C), ref, np.einsum("jnb,nc->jbc", np.abs(V), np.abs(W)).max())
    G = torch.full((bs, bs), float("nan"), dtype=torch.float64, device="cuda")
    cuda_handle.project_out(Vd, Wd, native.TRL_CGS_ONE, G)
    out = W - np.einsum("jnb,jbc->nc", V, ref)
    size = np.abs(W).max() + np.einsum("jnb,jbc->nc", np.abs(V), np.abs(ref)).max()
    got = host(Wd)
    assert np.abs(got - out).max() <= (1e-12 if dtype == torch.float64 else 1.2e-7) * size
    close(host(G), got.T @ got, (np.abs(got).T @ np.abs(got)).max())


@pytest.mark.parametrize("dtype", DT)
@pytest.mark.parametrize("n,nblk,bs", [(17500, 20, 4), (17501, 20, 4), (32768, 3, 1), (32769, 3, 1), (32768, 2, 8), (32769, 2, 8),
                                       (4096, 2, 16), (4097, 2, 16), (24576, 3, 16), (24577, 3, 16)])
def test_projections_where_the_launches_split(cuda_handle, dtype, n, nblk, bs):
    test_projections_at_the_edges_of_one_launch(cuda_handle, bs, dtype, n, nblk)
