"""The work that is measured: the kernels and steps of a block Lanczos solve, called as a
program calls them through ``trl_b200.native`` (the bindings of include/trl_cuda.h).

A solve spends its time in these calls: the SpMM of the prepared operator, the three-term
step with its reorthogonalisation and Cholesky-QR, the projected eigenproblem and the
rotation of each restart, the multi-block SpMM of the Chebyshev filter (mixed precision),
and, for a differentiable solve, the adjoint of the eigenvalues. The matrices are those of
trl_b200/problems.py (built here on the GPU from the seed): the 7-point anisotropic stencil,
the 27-point elasticity coupling, the Zipf pattern, the 5-point Laplacian and the 5-point
diffusion operator.
"""
import math

import numpy as np
import torch

from trl_b200 import native

F64, F32 = torch.float64, torch.float32
THRESHOLD = {"f64": 1e-12, "f32": 1e-6}  # the solver's thresholds of the partial reorthogonalisation


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # the operator of the headline workload (96^3 anisotropic Laplacian), applied once
        # per Lanczos step
        dict(name="spmm_stencil96_f64_b8", kind="spmm", matrix="stencil3d", nx=96, ny=96, nz=96, dtype="f64", bs=8, nb=1),
        # long rows (81 entries): the elasticity operator at full size
        dict(name="spmm_elast64_f64_b8", kind="spmm", matrix="elast", m=64, dtype="f64", bs=8, nb=1),
        # irregular rows and random columns: the Zipf pattern in FP32 at the widest block
        dict(name="spmm_zipf524k_f32_b16", kind="spmm", matrix="zipf", n=524_288, dtype="f32", bs=16, nb=1),
        # one degree of the Chebyshev filter: six kept blocks, three-term, FP64
        dict(name="filter_stencil96_f64_b8x6", kind="spmm", matrix="stencil3d", nx=96, ny=96, nz=96, dtype="f64", bs=8, nb=6),
        # a Lanczos step in the middle of a cycle, partial reorthogonalisation (the default)
        dict(name="step_stencil96_f64_b8", kind="step", matrix="stencil3d", nx=96, ny=96, nz=96, dtype="f64", bs=8, nblk=24, reorth="partial"),
        # the same step where the basis is projected out (after a restart, or always)
        dict(name="step_full_stencil96_f64_b8", kind="step", matrix="stencil3d", nx=96, ny=96, nz=96, dtype="f64", bs=8, nblk=40, reorth="full"),
        # the FP32 phase of a mixed solve, projected, on an irregular matrix of odd size
        dict(name="step_full_zipf100k_f32_b16", kind="step", matrix="zipf", n=100_003, dtype="f32", bs=16, nblk=20, reorth="full"),
        # the restart rotation of the headline workload: 48 blocks into 5
        dict(name="rotate_884k_f64_b8_48to5", kind="rotate", n=884_736, dtype="f64", bs=8, m=48, k=5),
        # projected eigenproblems of a restart: the headline's, and a large one of block size 16
        dict(name="eigen_n384_b8", kind="eigen", bs=8, nblk=48, nev=32),
        dict(name="eigen_n512_b16", kind="eigen", bs=16, nblk=32, nev=100),
        # backward: the gradient of 16 eigenvalues over a 512^2 diffusion grid
        dict(name="adjoint_diff512_k16", kind="adjoint", m=512, k=16),
        # a whole restart cycle on a small problem, where launches and latency count
        dict(name="cycle_laplace128_f64_b4", kind="cycle", nx=128, ny=128, dtype="f64", bs=4, nblk=40, nev=10),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_matrix(rng, lo, hi):
    """A matrix of about lo to hi rows."""
    n = _log(rng, lo, hi)
    what = rng.choice(("stencil3d", "stencil3d", "stencil2d", "elast", "zipf"))
    if what == "stencil3d":
        nx, ny = (max(4, int(n ** (1 / 3) * rng.uniform(0.7, 1.3))) for _ in range(2))
        return dict(matrix=what, nx=nx, ny=ny, nz=max(4, min(n // (nx * ny), 2 * nx)))
    if what == "stencil2d":
        nx = max(8, int(n ** 0.5 * rng.uniform(0.7, 1.4)))
        return dict(matrix=what, nx=nx, ny=max(8, n // nx))
    if what == "elast":
        return dict(matrix=what, m=max(6, min(48, round((n / 3) ** (1 / 3)))))
    return dict(matrix=what, n=min(n, 400_000) | 1)


def draw(rng):
    kind = rng.choice(("spmm", "spmm", "step", "step", "rotate", "eigen", "adjoint", "cycle"))
    if kind == "spmm":
        return dict(kind=kind, **_draw_matrix(rng, 2_000, 900_000), dtype=rng.choice(("f64", "f32")), bs=rng.choice((1, 2, 4, 8, 8, 16)), nb=rng.choice((1, 1, 1, 2, 3, 5, 6)))
    if kind == "step":
        c = dict(kind=kind, **_draw_matrix(rng, 4_000, 600_000), dtype=rng.choice(("f64", "f32")), bs=rng.choice((2, 4, 8, 8, 16)), reorth=rng.choice(("partial", "full")))
        n = _rows(c)
        c["nblk"] = max(2, min(rng.randint(3, 47), n // (8 * c["bs"]), 200_000_000 // (n * c["bs"])))
        return c
    if kind == "rotate":
        bs, m = rng.choice((1, 2, 4, 8, 8, 16)), rng.randint(8, 48)
        return dict(kind=kind, n=min(_log(rng, 3_000, 900_000), 330_000_000 // (m * bs)) | 1, dtype=rng.choice(("f64", "f32")), bs=bs, m=m, k=rng.randint(1, max(1, m // 4)))
    if kind == "eigen":
        bs = rng.choice((1, 2, 4, 8, 8, 16))
        nblk = max(6, min(_log(rng, 40, 520) // bs, 120))
        return dict(kind=kind, bs=bs, nblk=nblk, nev=rng.randint(bs, min(100, max(bs, bs * (nblk // 4)))))
    if kind == "adjoint":
        return dict(kind=kind, m=_log(rng, 17, 512), k=rng.randint(1, 32))
    bs = rng.choice((1, 2, 4, 8))
    nx = rng.randint(24, 128)
    return dict(kind=kind, nx=nx, ny=rng.randint(24, 128), dtype="f64", bs=bs, nblk=rng.randint(8, 40 if bs < 8 else 24), nev=2 * bs)


# ---------------------------------------------------------------- matrices (CSR on the GPU)
def _rows(c):
    what = c["matrix"]
    return c["nx"] * c["ny"] * c["nz"] if what == "stencil3d" else c["nx"] * c["ny"] if what == "stencil2d" else 3 * c["m"] ** 3 if what == "elast" else c["n"]


def _entries(c):
    """Stored entries (the Zipf pattern: their expected number)."""
    what = c["matrix"]
    if what == "stencil3d":
        x, y, z = c["nx"], c["ny"], c["nz"]
        return 7 * x * y * z - 2 * (x * y + y * z + x * z)
    if what == "stencil2d":
        return 5 * c["nx"] * c["ny"] - 2 * (c["nx"] + c["ny"])
    if what == "elast":
        return 9 * (3 * c["m"] - 2) ** 3
    k = np.arange(1, 513)
    return int(2 * c["n"] * (k ** -0.5).sum() / (k ** -1.5).sum())


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _pointers(counts):
    p = torch.zeros(counts.numel() + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(counts, 0, out=p[1:])
    return p.to(torch.int32)


def _stencil(shape, weights):
    """Dirichlet stencil, first axis fastest; weights: the diagonal's and one per axis."""
    n = math.prod(shape)
    i = torch.arange(n, device="cuda")
    strides = [math.prod(shape[:a]) for a in range(len(shape))]
    cols, vals, ok = [i], [weights[0]], [torch.ones_like(i, dtype=torch.bool)]
    for a, s in enumerate(strides):
        at = (i // s) % shape[a]
        cols, vals = [i - s] + cols + [i + s], [-weights[1 + a]] + vals + [-weights[1 + a]]
        ok = [at > 0] + ok + [at < shape[a] - 1]
    ok = torch.stack(ok, 1)
    v = torch.tensor(vals, dtype=F64, device="cuda").expand(n, -1)
    return _pointers(ok.sum(1)), torch.stack(cols, 1)[ok].to(torch.int32), v[ok]


def _elast(m, g):
    """27-point coupling of m^3 nodes with 3 x 3 blocks, diagonally dominant (values: each
    entry its own draw)."""
    i = torch.arange(m ** 3, device="cuda")
    x, y, z = i % m, (i // m) % m, i // (m * m)
    cols, ok = [], []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                cols.append(i + dx + m * (dy + m * dz))
                ok.append((x + dx >= 0) & (x + dx < m) & (y + dy >= 0) & (y + dy < m) & (z + dz >= 0) & (z + dz < m))
    ok = torch.stack(ok, 1)
    scale = 10.0 ** torch.empty(m ** 3, 27, dtype=F64, device="cuda").uniform_(-3.0, 0.0, generator=g)
    vals = torch.randn(m ** 3, 3, 27, 3, dtype=F64, device="cuda", generator=g) * scale[:, None, :, None]
    every = ok[:, None, :, None].expand(-1, 3, -1, 3)
    own = torch.eye(3, dtype=torch.bool, device="cuda")
    vals[:, :, 13, :] = torch.where(own, 0.0, vals[:, :, 13, :])
    total = (vals.abs() * every).sum((2, 3))
    vals[:, :, 13, :] += torch.where(own, 1.05 * total[:, :, None], 0.0)
    c = (3 * torch.stack(cols, 1)[:, None, :, None] + torch.arange(3, device="cuda")).expand(-1, 3, -1, -1)
    return _pointers((3 * ok.sum(1)).repeat_interleave(3)), c[every].to(torch.int32), vals[every]


def _zipf(n, g):
    """Symmetric pattern: Zipf(1.5) out-degrees of at most 512, uniform columns, mirrored."""
    cdf = torch.cumsum(torch.arange(1, 513, dtype=F64, device="cuda") ** -1.5, 0)
    deg = torch.searchsorted(cdf, torch.rand(n, dtype=F64, device="cuda", generator=g) * cdf[-1]).clamp(max=511) + 1
    r = torch.repeat_interleave(torch.arange(n, device="cuda"), deg)
    c = torch.randint(0, n, (r.numel(),), device="cuda", generator=g)
    key = torch.unique(torch.minimum(r, c) * n + torch.maximum(r, c))
    r, c = key // n, key % n
    v = torch.randn(r.numel(), dtype=F64, device="cuda", generator=g)
    off = r != c
    r, c, v = torch.cat([r, c[off]]), torch.cat([c, r[off]]), torch.cat([v, v[off]])
    order = torch.argsort(r * n + c)
    return _pointers(torch.bincount(r, minlength=n)), c[order].to(torch.int32), v[order]


def _diffusion(m, g):
    """5-point diffusion on an m x m grid with log-normal edge conductivities."""
    k = [torch.exp(torch.randn(m, m + 1, dtype=F64, device="cuda", generator=g)) for _ in range(2)]
    kx, ky = k[0], k[1].t()
    rp, ci, _ = _stencil((m, m), (1.0, 1.0, 1.0))
    left, right, low, high = kx[:, :-1], kx[:, 1:], ky[:-1], ky[1:]
    i = torch.arange(m * m, device="cuda")
    x, y = i % m, i // m
    ok = torch.stack([y > 0, x > 0, x >= 0, x < m - 1, y < m - 1], 1)
    v = torch.stack([-low.reshape(-1), -left.reshape(-1), (left + right + low + high).reshape(-1), -right.reshape(-1), -high.reshape(-1)], 1)
    return rp, ci, v[ok]


def _matrix(c, g):
    what = c["matrix"]
    if what == "stencil3d":
        return _stencil((c["nx"], c["ny"], c["nz"]), (222.0, 1.0, 10.0, 100.0))
    if what == "stencil2d":
        return _stencil((c["nx"], c["ny"]), (4.0, 1.0, 1.0))
    return _elast(c["m"], g) if what == "elast" else _zipf(c["n"], g)


def _csr(arrays, dtype):
    rp, ci, va = arrays
    va = va.to(dtype)
    return native.DeviceCSRTensors(rp, ci, va, native.trl_csr(rp.numel() - 1, ci.numel(), rp.data_ptr(), ci.data_ptr(), va.data_ptr(), native.TRL_F64 if dtype == F64 else native.TRL_F32))


def _product(arrays, X, dtype=F64):
    """A X in 64 bits, with A's values as stored in `dtype`."""
    rp, ci, va = arrays
    n = rp.numel() - 1
    return torch.sparse_csr_tensor(rp, ci, va.to(dtype).to(F64), size=(n, n)) @ X.to(F64)


# ---------------------------------------------------------------- plain Lanczos in 64 bits
def _cholqr(W):
    """Orthonormal Q and upper triangular R with W = Q R (Cholesky-QR, twice)."""
    total = torch.eye(W.shape[1], dtype=F64, device="cuda")
    for _ in range(2):
        R = torch.linalg.cholesky(W.t() @ W).t()
        W = torch.linalg.solve_triangular(R, W, upper=True, left=False)
        total = R @ total
    return W, total


def _against(V, W):
    """W less its components along the blocks V (nblk, n, bs)."""
    for _ in range(2):
        W = W - torch.einsum("jnb,jbc->nc", V, torch.matmul(V.transpose(1, 2), W))
    return W


def _basis(arrays, V, dtype):
    """Lanczos from V[0] through all blocks of V (64 bits, fully orthogonalised). Returns the
    diagonal blocks and the factors R of each step."""
    D, R = [], []
    for i in range(V.shape[0] - 1):
        W = _product(arrays, V[i], dtype)
        if i:
            W -= V[i - 1] @ R[-1].t()
        D.append(V[i].t() @ W)
        W -= V[i] @ D[-1]
        V[i + 1], r = _cholqr(_against(V[: i + 1], W))
        R.append(r)
    return D, R


def _start_block(n, bs, g):
    return _cholqr(torch.randn(n, bs, dtype=F64, device="cuda", generator=g))[0]


def _sketch_weights(count, bs):
    """One fixed sequence of N(0, 1/bs) coefficients, whatever the seed."""
    w = np.random.default_rng(5).standard_normal((count, bs, bs)) / math.sqrt(bs)
    return torch.from_numpy(w).cuda()


# ---------------------------------------------------------------- projected matrices
def _projected(c, seed):
    """A thick-restart matrix: kept Ritz values, their coupling to the next block, and the
    block-tridiagonal rest; beta: the last step's factor."""
    rng = np.random.default_rng(seed)
    bs, nblk = c["bs"], c["nblk"]
    N, kr = bs * nblk, min(c["nev"] // bs + 1, nblk - 2)
    T = np.zeros((N, N))
    k = kr * bs
    T[:k, :k] = np.diag(440.0 + 4.0 * (np.arange(k)[::-1] + rng.uniform(0.1, 0.9, k)) / k)
    for b in range(kr, nblk):
        s = slice(b * bs, (b + 1) * bs)
        D = rng.standard_normal((bs, bs)) * (8.0 / math.sqrt(bs)) + np.eye(bs) * 110.0
        T[s, s] = D + D.T
        if b + 1 < nblk:
            T[(b + 1) * bs:(b + 2) * bs, s] = np.triu(rng.standard_normal((bs, bs)) * (20.0 / math.sqrt(bs)) + np.eye(bs) * 60.0)
    T[k:k + bs, :k] = rng.standard_normal((bs, k)) * 10.0 ** rng.uniform(-4.0, -1.0, k)
    T = np.tril(T) + np.tril(T, -1).T
    beta = np.triu(rng.standard_normal((bs, bs)) * 5.0 + np.eye(bs) * 40.0)
    return T, beta


def _kept(c):
    return min(c["bs"] * c["nblk"], (c["nev"] // c["bs"] + 1) * c["bs"])


def _signed(Y):
    """Eigenvectors in block layout, each column's sign such that its entries' sum is positive."""
    return Y * Y.sum((0, 2), keepdim=True).sign()


# ---------------------------------------------------------------- the program's side
_program = {}


def _handle():
    """One handle on a stream of the program's own, which is torch's current stream too."""
    if not _program:
        torch.cuda.set_stream(torch.cuda.Stream())
        _program["handle"] = native.Handle(0)
    return _program["handle"]


def _dtype(c):
    return F64 if c["dtype"] == "f64" else F32


def _adjoint_inputs(c, seed):
    """Eigenvectors, eigenvalues (with a few close pairs) and weights."""
    g, rng = _generator(seed), np.random.default_rng(seed)
    k = c["k"]
    X = torch.randn(c["m"] ** 2, k, dtype=F64, device="cuda", generator=g) / c["m"]
    lam = np.sort(rng.uniform(1.0, 40.0, k))
    lam[2::5] = lam[1::5][: lam[2::5].size]
    return _diffusion(c["m"], g), X, lam, rng.uniform(0.0, 1.0, k)


def _spmm_inputs(c, seed):
    g = _generator(seed)
    A = _matrix(c, g)
    shape = (c["nb"], _rows(c), c["bs"])
    X = torch.randn(shape, device="cuda", dtype=_dtype(c), generator=g)
    W = torch.randn(shape, device="cuda", dtype=_dtype(c), generator=g) if c["nb"] > 1 else None
    return A, X, W


def _step_inputs(c, seed):
    g = _generator(seed)
    A, n, bs, nblk = _matrix(c, g), _rows(c), c["bs"], c["nblk"]
    V = torch.empty((nblk, n, bs), dtype=F64, device="cuda")
    V[0] = _start_block(n, bs, g)
    _, R = _basis(A, V, _dtype(c))
    S = torch.einsum("jnb,jbc->nc", V, _sketch_weights(nblk, bs))
    return A, V.to(_dtype(c)), R[-1].contiguous(), S.to(_dtype(c))


def _rotate_inputs(c, seed):
    g = _generator(seed)
    V = torch.randn(c["m"], c["n"], c["bs"], dtype=_dtype(c), device="cuda", generator=g)
    q = torch.linalg.qr(torch.randn(c["m"] * c["bs"], c["m"] * c["bs"], dtype=F64, device="cuda", generator=g))[0]
    Y = q.reshape(c["m"], c["bs"], c["m"], c["bs"]).transpose(1, 2).contiguous()
    return V, Y


def prepare(case, seed):
    h, c = _handle(), case
    kind, bs = c["kind"], c.get("bs")
    if kind == "spmm":
        A, X, W = _spmm_inputs(c, seed)
        csr = _csr(A, _dtype(c))
        if c["nb"] == 1:
            X = X[0]
        return dict(c=c, h=h, op=h.prepare(csr, bs), X=X, Y=torch.empty_like(X), W=W)
    if kind == "step":
        A, V, B, S = _step_inputs(c, seed)
        nblk, n = V.shape[:2]
        basis = torch.empty((nblk + 1, n, bs), dtype=V.dtype, device="cuda")
        basis[:nblk] = V
        small = torch.zeros((4, bs, bs), dtype=F64, device="cuda")
        return dict(c=c, h=h, op=h.prepare(_csr(A, _dtype(c)), bs), V=basis, B=B, S=S, T=small[0], G=small[1], R=small[2], pair=torch.zeros(1, dtype=torch.int32, device="cuda"))
    if kind == "rotate":
        V, Y = _rotate_inputs(c, seed)
        return dict(c=c, h=h, V=V, Y=Y, W=torch.empty((c["k"],) + V.shape[1:], dtype=V.dtype, device="cuda"))
    if kind == "eigen":
        T, beta = _projected(c, seed)
        T = T.reshape(c["nblk"], bs, c["nblk"], bs).transpose(0, 2, 1, 3)
        return dict(c=c, h=h, T=torch.from_numpy(np.ascontiguousarray(T)).cuda(), beta=torch.from_numpy(beta).cuda())
    if kind == "adjoint":
        K, X, lam, w = _adjoint_inputs(c, seed)
        n = c["m"] ** 2
        i = torch.arange(n + 1, dtype=torch.int32, device="cuda")
        D = (i, i[:n].clone(), torch.ones(n, dtype=F64, device="cuda"))
        return dict(c=c, h=h, K=_csr(K, F64), D=_csr(D, F64), X=X, lam=lam, w=w, gK=torch.empty(K[1].numel(), dtype=F64, device="cuda"), gM=torch.empty(n, dtype=F64, device="cuda"))
    n, nblk = c["nx"] * c["ny"], c["nblk"]
    A = _stencil((c["nx"], c["ny"]), (4.0, 1.0, 1.0))
    V = torch.zeros((nblk + 1, n, bs), dtype=F64, device="cuda")
    V[0] = _start_block(n, bs, _generator(seed))
    return dict(c=c, h=h, op=h.prepare(_csr(A, F64), bs), V=V, S=torch.zeros((n, bs), dtype=F64, device="cuda"), G=torch.zeros((bs, bs), dtype=F64, device="cuda"),
                beta=torch.zeros((bs, bs), dtype=F64, device="cuda"), weights=_sketch_weights(nblk, bs), T=torch.zeros((nblk, nblk, bs, bs), dtype=F64, device="cuda"),
                pair=torch.zeros(1, dtype=torch.int32, device="cuda"))


def run(state):
    s, c, h = state, state["c"], state["h"]
    kind = c["kind"]
    if kind == "spmm":
        if c["nb"] == 1:
            s["op"].spmm(s["X"], s["Y"])
        else:
            s["op"].spmm(s["X"], s["Y"], 0.75, -1.25, 0.5, s["W"])
        return s["Y"]
    if kind == "step":
        V, nblk = s["V"], c["nblk"]
        v, W = V[nblk - 1], V[nblk]
        s["op"].spmm(v, W)
        h.bv_mult(native.TRL_SUBTRACT_TRANSPOSE, V[nblk - 2], s["B"], W)
        h.block_dot(V[nblk - 1:nblk], W, s["T"])
        h.bv_mult(native.TRL_SUBTRACT, v, s["T"], W)
        if c["reorth"] == "partial":
            h.project_out_sketch(V[:nblk], W, s["S"], THRESHOLD[c["dtype"]], s["G"], pair_state=s["pair"])
        else:
            h.project_out(V[:nblk], W, native.TRL_CGS_IFNEEDED, s["G"])
        h.cholqr_gram(W, 2, s["R"], s["G"])
        return [W, s["T"], s["R"]]
    if kind == "rotate":
        h.block_rotate(s["V"], s["Y"], c["k"], s["W"])
        return s["W"]
    if kind == "eigen":
        _, Y, evals, nconv = h.small_eigen_partial(s["T"], s["beta"], c["nev"], 1e-6, _kept(c))
        return [evals, _signed(Y), nconv]
    if kind == "adjoint":
        h.eigen_adjoint(s["K"], s["X"], s["lam"], s["w"], s["gK"], kind=0)
        h.eigen_adjoint(s["D"], s["X"], s["lam"], s["w"], s["gM"], kind=1)
        return [s["gK"], s["gM"]]
    V, T, S, weights = s["V"], s["T"], s["S"], s["weights"]
    nblk = c["nblk"]
    s["pair"].zero_()
    for i in range(nblk):
        W = V[i + 1]
        s["op"].spmm(V[i], W)
        if i:
            h.bv_mult(native.TRL_SUBTRACT_TRANSPOSE, V[i - 1], T[i, i - 1], W)
        h.block_dot(V[i:i + 1], W, T[i, i])
        h.bv_mult(native.TRL_SUBTRACT, V[i], T[i, i], W)
        if i:
            h.bv_mult(native.TRL_MULT_ADD, V[i], weights[i], S)
        else:
            h.bv_mult(native.TRL_MULT, V[0], weights[0], S)
        h.project_out_sketch(V[: i + 1], W, S, THRESHOLD["f64"], s["G"], pair_state=s["pair"])
        h.cholqr_gram(W, 2, T[i + 1, i] if i + 1 < nblk else s["beta"], s["G"])
    _, _, evals, nconv = h.small_eigen_partial(T, s["beta"], c["nev"], 1e-8, _kept(c))
    return [V, T, evals, nconv]


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    c = case
    kind, es, bs = c["kind"], 8 if c.get("dtype", "f64") == "f64" else 4, c.get("bs", 1)
    if kind in ("spmm", "step"):
        n, nnz = _rows(c), _entries(c)
        a, block = nnz * (es + 4.0) + 4.0 * (n + 1), float(n) * bs * es
        if kind == "spmm":
            return dict(bytes=a + c["nb"] * (2 if c["nb"] == 1 else 3) * block, flops=2.0 * nnz * bs * c["nb"])
        # the matrix, the blocks read (the last two and the sketch, or the basis) and the new one
        partial = c["reorth"] == "partial"
        blocks = 4 if partial else c["nblk"] + 1
        return dict(bytes=a + blocks * block, flops=2.0 * nnz * bs + 2.0 * n * bs * bs * (9 if partial else 2 * c["nblk"] + 8))
    if kind == "rotate":
        return dict(bytes=(c["m"] + c["k"]) * float(c["n"]) * bs * es, flops=2.0 * c["n"] * c["m"] * c["k"] * bs * bs)
    if kind == "eigen":
        N = bs * c["nblk"]
        return dict(bytes=16.0 * N * N, flops=4.0 / 3.0 * N ** 3 + 4.0 * N * N * _kept(c))
    if kind == "adjoint":
        n, k = c["m"] ** 2, c["k"]
        nnz = 5 * n - 4 * c["m"]
        return dict(bytes=8.0 * n * k + 12.0 * nnz + 4.0 * (n + 1) + 16.0 * n, flops=3.0 * k * (nnz + n))
    n, m = c["nx"] * c["ny"], c["nblk"]
    nnz = 5 * n - 2 * (c["nx"] + c["ny"])
    N = m * bs
    return dict(bytes=12.0 * nnz + 8.0 * n * bs * (m + 1) + 8.0 * N * N, flops=m * (2.0 * nnz * bs + 18.0 * n * bs * bs) + 4.0 / 3.0 * N ** 3)


# ---------------------------------------------------------------- the same in plain 64 bits
def exact(case, seed):
    _handle()
    c = case
    kind, bs = c["kind"], c.get("bs")
    if kind == "spmm":
        A, X, W = _spmm_inputs(c, seed)
        Y = torch.stack([_product(A, x, _dtype(c)) for x in X])
        return Y[0] if W is None else 0.75 * Y - 1.25 * X.to(F64) + 0.5 * W.to(F64)
    if kind == "step":
        A, V, B, _ = _step_inputs(c, seed)
        dtype, V = _dtype(c), V.to(F64)
        W = _product(A, V[-1], dtype) - V[-2] @ B.t()
        T = V[-1].t() @ W
        W -= V[-1] @ T
        if c["reorth"] == "full":
            W -= torch.einsum("jnb,jbc->nc", V, torch.matmul(V.transpose(1, 2), W))
        W, R = _cholqr(W)
        return [W, T, R]
    if kind == "rotate":
        V, Y = _rotate_inputs(c, seed)
        return torch.stack([sum(V[i].to(F64) @ Y[i, j] for i in range(c["m"])) for j in range(c["k"])])
    if kind in ("eigen", "cycle"):
        N = bs * c["nblk"]
        if kind == "eigen":
            T = torch.from_numpy(_projected(c, seed)[0]).cuda()
        else:
            A = _stencil((c["nx"], c["ny"]), (4.0, 1.0, 1.0))
            V = torch.empty((c["nblk"] + 1, c["nx"] * c["ny"], bs), dtype=F64, device="cuda")
            V[0] = _start_block(V.shape[1], bs, _generator(seed))
            D, R = _basis(A, V, F64)
            blocks = torch.zeros((c["nblk"], c["nblk"], bs, bs), dtype=F64, device="cuda")
            for i in range(c["nblk"]):
                blocks[i, i] = D[i]
                if i + 1 < c["nblk"]:
                    blocks[i + 1, i] = R[i]
            T = blocks.transpose(1, 2).reshape(N, N)
        w, Y = torch.linalg.eigh(T)
        order = torch.argsort(w.abs(), descending=True)
        w = w[order].cpu().numpy()
        if kind == "cycle":
            return [V, blocks, w, None]
        Y = Y[:, order].clone()
        Y[:, _kept(c):] = 0.0
        return [w, _signed(Y.reshape(c["nblk"], bs, c["nblk"], bs).transpose(1, 2)), None]
    (rp, ci, _), X, lam, w = _adjoint_inputs(c, seed)
    group = np.concatenate([[0], np.cumsum(np.diff(lam) > 1e-8 * lam.max())])
    mean = np.bincount(group, w) / np.bincount(group)
    w = torch.from_numpy(mean[group]).cuda()
    lam = torch.from_numpy(lam).cuda()
    r = torch.repeat_interleave(torch.arange(c["m"] ** 2, device="cuda"), (rp[1:] - rp[:-1]).long())
    return [(w * X[r] * X[ci.long()]).sum(1), -(w * lam * X * X).sum(1)]
