"""The prepared SpMM of operators with long rows (16 or more slots per slice), whose warps take their
slices from a counter: every residue of the row lengths modulo the 8 slots of a group, empty rows,
fewer slices than warps, rows of one window only, and a last window with missing slices; the counter
starts at zero again in every call, and two handles may use one operator at the same time.
Bit for bit the CSR kernel's per-row walk (trl_cuda_spmm_blocks), and the oracle to the
tolerances of test_sell_gpu.py."""
import functools

import numpy as np
import pytest
import torch

from trl_b200 import native
from trl_b200 import problems as P

from test_kernels_gpu import BS, DT, as_dt, dev
from test_sell_gpu import _mag

pytestmark = pytest.mark.gpu


def _rows(deg, seed):
    rng = np.random.default_rng(seed)
    n = deg.size
    cols = np.concatenate([rng.choice(n, size=d, replace=False) for d in deg])
    return P._from_coo(n, np.repeat(np.arange(n), deg), cols, rng.standard_normal(cols.size))


def _patterns():
    n = 9000  # three windows, the last one incomplete
    skewed = 17 + np.arange(n) % 9
    skewed[::501] = 700
    skewed[5::13] = 0
    return [("residues", _rows(16 + np.arange(997) % 41, 1)), ("skewed", _rows(skewed, 2)), ("one_slice", _rows(np.full(31, 31), 3))]


PATTERNS = _patterns()


@pytest.mark.parametrize("bs", BS)
@pytest.mark.parametrize("dtype", DT)
@pytest.mark.parametrize("case", PATTERNS, ids=lambda c: c[0])
def test_long_rows(cuda_handle, bs, dtype, case):
    A = case[1]
    rng = np.random.default_rng(bs)
    Ad = native.DeviceCSRTensors.from_host(A, dtype)
    op = cuda_handle.prepare(Ad, bs)
    X = as_dt(rng.standard_normal((A.n, bs)), dtype)
    W = as_dt(rng.standard_normal((A.n, bs)), dtype)
    Xd, Wd = dev(X, dtype), dev(W, dtype)
    ref = torch.empty((2, A.n, bs), dtype=dtype, device="cuda")
    cuda_handle.spmm_blocks(Ad, torch.stack([Xd, Xd]), ref, -0.5, 2.0, 0.25, torch.stack([Wd, Wd]))
    for _ in range(3):
        Y = torch.full((A.n, bs), float("nan"), dtype=dtype, device="cuda")
        op.spmm(Xd, Y, -0.5, 2.0, 0.25, Wd)
        assert torch.equal(Y, ref[0])
    vals = A.values.astype(np.float32).astype(np.float64) if dtype == torch.float32 else A.values
    host = -0.5 * P.CSRMatrix(A.n, A.rowptr, A.colind, vals).matmat(X) + 2.0 * X + 0.25 * W
    scale = 0.5 * _mag(A, vals, X) + 2.0 * np.abs(X).max() + 0.25 * np.abs(W).max()
    assert np.abs(Y.double().cpu().numpy() - host).max() <= (1e-12 if dtype == torch.float64 else 2e-6) * scale
    op.close()


def test_one_operator_on_two_handles(cuda_handle):
    A = PATTERNS[1][1]
    op = cuda_handle.prepare(native.DeviceCSRTensors.from_host(A), 8)
    X = torch.randn((A.n, 8), dtype=torch.float64, device="cuda")
    ref = torch.empty_like(X)
    op.spmm(X, ref)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    handles = [native.Handle(0, s) for s in streams]
    out = [[torch.full_like(X, float("nan")) for _ in range(20)] for _ in handles]
    torch.cuda.synchronize()
    for k in range(20):
        for h, o in zip(handles, out):
            h.check(h.lib.trl_cuda_op_spmm(h.h, op.op, X.data_ptr(), o[k].data_ptr(), 1, 1.0, 0.0, 0.0, None))
    torch.cuda.synchronize()
    assert all(torch.equal(y, ref) for o in out for y in o)
    op.close()


@pytest.mark.parametrize("dtype", DT)
def test_first_call_of_a_handle_inside_a_capture(cuda_handle, dtype):
    """A prepared product allocates nothing, so it may be the first thing a handle does inside a stream
    capture; the graph may be replayed."""
    A = PATTERNS[1][1]
    Ad = native.DeviceCSRTensors.from_host(A, dtype)
    op = cuda_handle.prepare(Ad, 4)
    X = dev(np.random.default_rng(0).standard_normal((A.n, 4)).astype(np.float32), dtype)
    ref, Y = torch.empty_like(X), torch.empty_like(X)
    op.spmm(X, ref)
    cuda_handle.sync()
    s = torch.cuda.Stream()
    h = native.Handle(0, stream=s)
    try:
        h.sync()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            h.check(h.lib.trl_cuda_op_spmm(h.h, op.op, X.data_ptr(), Y.data_ptr(), 1, 1.0, 0.0, 0.0, None))
        for _ in range(3):
            Y.fill_(float("nan"))
            torch.cuda.synchronize()
            g.replay()
            torch.cuda.synchronize()
            assert torch.equal(Y, ref)
        del g
    finally:
        torch.cuda.synchronize()
        h.close()
        op.close()


@functools.lru_cache(None)
def _with_counter(kind):
    """Slices enough and long enough that their warps take them from the counter: rows of one length nearly, and
    a skewed pattern whose longest slices come first."""
    n, base = (20000, 420) if kind == "even" else (40000, 152)
    deg = base + np.arange(n) % 9
    if kind == "skewed":
        deg[::1501] = 1500
        deg[7::1013] = 0
    row = np.repeat(np.arange(n), deg)
    col = (row + 7 * (np.arange(row.size) - np.repeat(np.cumsum(deg) - deg, deg))) % n
    return P._from_coo(n, row, col, np.random.default_rng(n).standard_normal(row.size))


@pytest.mark.parametrize("bs", BS)
@pytest.mark.parametrize("dtype", DT)
@pytest.mark.parametrize("kind", ["even", "skewed"])
def test_slices_from_the_counter(cuda_handle, bs, dtype, kind):
    A = _with_counter(kind)
    Ad = native.DeviceCSRTensors.from_host(A, dtype)
    op = cuda_handle.prepare(Ad, bs)
    X, W = (dev(as_dt(np.random.default_rng(s).standard_normal((A.n, bs)), dtype), dtype) for s in (1, 2))
    ref = torch.empty((2, A.n, bs), dtype=dtype, device="cuda")
    cuda_handle.spmm_blocks(Ad, torch.stack([X, X]), ref, -0.5, 2.0, 0.25, torch.stack([W, W]))
    for _ in range(3):
        Y = torch.full((A.n, bs), float("nan"), dtype=dtype, device="cuda")
        op.spmm(X, Y, -0.5, 2.0, 0.25, W)
        assert torch.equal(Y, ref[0])
    op.close()


def test_counters_of_two_handles_and_of_replays(cuda_handle, monkeypatch):
    monkeypatch.setitem(globals(), "PATTERNS", [None, ("skewed", _with_counter("skewed"))])
    test_one_operator_on_two_handles(cuda_handle)
    test_first_call_of_a_handle_inside_a_capture(cuda_handle, torch.float64)


def test_captured_products_of_one_handle_beside_one_another():
    """Two graphs captured from one handle, replayed on two streams at once, and the handle's own calls."""
    A = _with_counter("skewed")
    s = torch.cuda.Stream()
    h = native.Handle(0, stream=s)
    try:
        Ad = native.DeviceCSRTensors.from_host(A)  # on torch's stream; read on the handle's until the next synchronisation
        torch.cuda.synchronize()
        op = h.prepare(Ad, 16)
        h.sync()
        X = torch.randn((3, A.n, 16), dtype=torch.float64, device="cuda")
        Y, ref = torch.empty_like(X), torch.empty_like(X)
        torch.cuda.synchronize()
        for x, y in zip(X, ref):
            op.spmm(x, y)
        torch.cuda.synchronize()
        graphs = [torch.cuda.CUDAGraph() for _ in range(2)]
        for g, x, y in zip(graphs, X, Y):
            with torch.cuda.graph(g, stream=s):
                op.spmm(x, y)
        streams = [torch.cuda.Stream() for _ in range(2)]
        for _ in range(20):
            Y.fill_(float("nan"))
            torch.cuda.synchronize()
            for g, t in zip(graphs, streams):
                with torch.cuda.stream(t):
                    g.replay()
            op.spmm(X[2], Y[2])
            torch.cuda.synchronize()
            assert torch.equal(Y, ref)
        del graphs
        op.close()
    finally:
        torch.cuda.synchronize()
        h.close()
