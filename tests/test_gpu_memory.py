"""Solves where memory is short: what makes a solve faster is left out, the solve runs.

A fixture leaves a few MB of device memory free; each test asks for an optional table that
is larger than that on a system whose solve needs no further memory.  Every kernel of
the path has run once before, so that none is loaded under pressure.
"""
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
    """leave(n): fills the device but for at most n MB; freed after the test."""
    torch, _ = env
    held = []

    def fill(mb):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        for _ in range(1000):
            free = torch.cuda.mem_get_info()[0]
            if free <= mb * MB:
                return
            held.append(torch.empty(max(2 * MB, (free - mb * MB) // (2 * MB) * 2 * MB), dtype=torch.uint8, device="cuda"))
        raise AssertionError("could not fill the device")

    yield fill
    held.clear()
    torch.cuda.empty_cache()


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
