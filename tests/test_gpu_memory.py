"""Solves where memory is short: what makes a solve faster is left out, the solve runs.

A fixture leaves a few MB of device memory free; each test asks for an optional table that
is larger than that on a system whose solve needs no further memory.  Every kernel of
the path has run once before, so that none is loaded under pressure.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


@pytest.fixture(scope="module")
def env():
    import torch

    import hpccg_b200 as hp
    return torch, hp


@pytest.fixture
def leave(env):
    """leave(n): fills the device but for at most n MB (driver allocations of 2 MB and more);
    leave.free() and the end of the test give all of it back."""
    torch, _ = env
    cu = ctypes.CDLL("libcuda.so.1")
    cu.cuMemAlloc_v2.argtypes = [ctypes.POINTER(ctypes.c_uint64), ctypes.c_size_t]
    cu.cuMemFree_v2.argtypes = [ctypes.c_uint64]
    held = []

    def fill(mb):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        size = torch.cuda.mem_get_info()[0]
        while (over := torch.cuda.mem_get_info()[0] - mb * MB) > 0:
            size = max(2 * MB, min(size, over) // (2 * MB) * 2 * MB)
            ptr = ctypes.c_uint64()
            if cu.cuMemAlloc_v2(ctypes.byref(ptr), size) == 0:
                held.append(ptr.value)
            else:
                assert size > 2 * MB, "could not fill the device"
                size //= 2

    def free():
        torch.cuda.synchronize()
        while held:
            assert cu.cuMemFree_v2(held.pop()) == 0

    fill.free = free
    yield fill
    free()


def _cg(torch, M, b, n=6):
    x = torch.zeros_like(b)
    it, normr, hist, st = M.cg_device(b, x, n, 0.0)
    assert st == 0 and it == n
    return np.asarray(hist), x


def test_row_patterns_are_optional(env, leave):
    """27M rows: codes of 54 MB.  CG on AUTO equals the explicit ELL's (dot products may be
    associated differently: 1e-12 of the residual, and of the solution's scale)."""
    torch, hp = env
    small = hp.Matrix.generated(96, 96, 160)
    M = hp.Matrix.generated(300, 300, 300)
    b = torch.rand(M.nrow, dtype=torch.float64, device="cuda")
    for W in (small, M):
        W.set_spmv(hp.SPMV_ELL)
        want = _cg(torch, W, b[:W.nrow])
    small.set_spmv(hp.SPMV_AUTO)
    _cg(torch, small, b[:small.nrow])
    x = torch.zeros_like(b)
    leave(40)
    M.set_spmv(hp.SPMV_AUTO)
    it, normr, hist, st = M.cg_device(b, x, 6, 0.0)
    assert st == hp.HPCCG_OK and it == 6
    assert (np.abs(hist - want[0]) <= 1e-12 * want[0]).all()
    xh, wh = x.cpu().numpy(), want[1].cpu().numpy()
    assert np.abs(xh - wh).max() <= 1e-12 * np.abs(wh).max() + 1e-12


def test_batch_row_patterns_are_optional(env, leave):
    """The same for a stored batch: FP64 on the stacked ELL, bit for bit the patterns' result."""
    torch, hp = env
    sizes = [(160, 128, 128)] * 10
    out = []
    for short in (False, True):
        B = hp.Batch.generated(sizes)
        b = torch.arange(B.stacked_rows, dtype=torch.float64, device="cuda") % 7 - 3
        x = torch.zeros_like(b)
        if short:
            leave(30)
        iters, relres, _, st = B.solve(b, x, hp.PREC_FP64, 1e-6, 100)
        assert st == hp.HPCCG_OK
        out.append((x.cpu().numpy(), iters))
        B.close()
    assert np.array_equal(out[0][1], out[1][1]) and np.array_equal(out[0][0], out[1][0])


def test_one_kernel_cg_buffers_are_optional(env, leave):
    """The one-kernel CG's second p takes 8.3 MB here; without it the graph of the same rows
    runs, whose dot products are associated differently (the bars of test_one_kernel_cg).
    With memory again the one kernel runs: the same context, the result of a fresh one."""
    torch, hp = env
    rows, cols, vals = hp.generate_matrix(101, 101, 102)[:3]
    big = hp.Matrix.from_csr(*hp.generate_matrix(110, 100, 100)[:3])  # the graph of the pattern rows
    fresh, M = (hp.Matrix.from_csr(rows, cols, vals) for _ in range(2))
    b = torch.rand(big.nrow, dtype=torch.float64, device="cuda")
    _cg(torch, big, b)
    want = _cg(torch, fresh, b[:M.nrow])
    y, x = torch.empty_like(want[1]), torch.zeros_like(want[1])
    M.spmv(want[1], y)  # finds the patterns
    leave(6)
    for _ in range(2):  # a second solve finds the buffers missing again
        x.zero_()
        it, normr, hist, st = M.cg_device(b[:M.nrow], x, 6, 0.0)
        assert st == hp.HPCCG_OK and it == 6
        assert (np.abs(hist - want[0]) <= 1e-12 * want[0]).all()
        assert np.abs(x.cpu().numpy() - want[1].cpu().numpy()).max() <= 1e-10
    leave.free()
    again = _cg(torch, M, b[:M.nrow])
    assert np.array_equal(again[0], want[0]) and torch.equal(again[1], want[1])


def test_batch_tiles_are_optional(env, leave):
    """The tiled FP32 iteration's second p takes 105 MB; without it the column walks run, and
    every system meets the target by a residual formed here in FP64."""
    torch, hp = env
    sizes = [(160, 128, 128)] * 10
    warm = hp.Batch.generated([(1, 1, 300), (2, 1, 50)])  # shapes the tiles do not suit
    B = hp.Batch.generated(sizes)
    b = torch.arange(B.stacked_rows, dtype=torch.float64, device="cuda") % 7 - 3
    x, r = torch.zeros_like(b), torch.zeros_like(b)
    for W in (warm, B):
        W.set_spmv(hp.SPMV_STENCIL)
    warm.solve(b[:warm.stacked_rows], x[:warm.stacked_rows].zero_(), hp.PREC_FP32, 1e-6, 100)
    x.zero_()
    leave(40)
    iters, relres, _, st = B.solve(b, x, hp.PREC_FP32, 1e-6, 200)
    leave.free()
    assert st == hp.HPCCG_OK
    B.spmv(x, r)
    for s, o in enumerate(B.offsets):
        v = slice(int(o), int(o + B.nrows[s]))
        rel = float(torch.linalg.vector_norm(b[v] - r[v]) / torch.linalg.vector_norm(b[v]))
        assert rel <= 1e-6 * (1 + 1e-6) and relres[s] == pytest.approx(rel, rel=1e-6)
    want = x.clone()
    B.solve(b, x.zero_(), hp.PREC_FP32, 1e-6, 200)  # the same form again
    assert torch.equal(x, want)
