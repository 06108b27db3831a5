"""Row patterns of a stored matrix (HPCCG_SPMV_AUTO) against the ELL kernels.

The CG of small systems in one kernel is compared with the graph of the explicit
ELL kernel: the rows are the same, the dot products associated differently.

The pattern form adds the same terms in the same order, so FP64 products, fused
dots and CG runs, and the low-precision products, must equal the explicit ELL
kernel's bit for bit (the low-precision ELL kernel sums in the same order too).
"""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env():
    import torch

    import hpccg_b200 as hp
    return torch, hp


def _products(torch, hp, M, kind, x):
    """FP64 and low-precision products and a CG run with one row kernel."""
    M.set_spmv(kind)
    n = M.nrow
    dx = torch.from_numpy(x).cuda()
    y = torch.full((n,), 7.0, dtype=torch.float64, device="cuda")
    M.spmv(dx, y)
    out = [y.cpu().numpy()]
    xf = dx.float()
    for prec in (hp.PREC_FP32, hp.PREC_BF16):
        yf = torch.full((n,), 7.0, dtype=torch.float32, device="cuda")
        M.spmv_lowp(prec, xf, yf)
        out.append(yf.cpu().numpy())
    return out


@pytest.mark.parametrize("nx,ny,nz", [(3, 3, 3), (5, 4, 7), (32, 16, 9), (33, 17, 5), (34, 6, 33), (64, 18, 20), (97, 3, 40)])
@pytest.mark.parametrize("known_grid", [False, True])
def test_patterns_equal_ell_on_grids(env, nx, ny, nz, known_grid):
    torch, hp = env
    A, x0, b, _ = oracle.generate_matrix(nx, ny, nz)
    M = hp.Matrix.generated(nx, ny, nz) if known_grid else hp.Matrix.from_csr(A.rowindex, A.colindex, A.values)
    x = np.random.default_rng(nx).uniform(-1, 1, A.nrow)
    got, want = _products(torch, hp, M, hp.SPMV_AUTO, x), _products(torch, hp, M, hp.SPMV_ELL, x)
    assert np.array_equal(want[0], oracle.spmv(A, x))
    for g, w in zip(got, want):
        assert np.array_equal(g, w)


@pytest.mark.parametrize("nx,ny,nz", [(128, 128, 112), (130, 132, 90), (151, 131, 97), (161, 160, 160)])
def test_box_walks_equal_ell(env, nx, ny, nz):
    """Grids large enough for the walks: tiles (whole and partial) by TMA and by plain
    loads, one line and two lines a thread.  CG runs its graph at these sizes: the
    same sums in the same order, so the same bits."""
    torch, hp = env
    M = hp.Matrix.generated(nx, ny, nz)
    x = np.random.default_rng(nx).uniform(-1, 1, M.nrow)
    got, want = _products(torch, hp, M, hp.SPMV_AUTO, x), _products(torch, hp, M, hp.SPMV_ELL, x)
    for g, w in zip(got, want):
        assert np.array_equal(g, w)
    b = torch.from_numpy(x).cuda()
    runs = []
    for kind in (hp.SPMV_AUTO, hp.SPMV_ELL):
        M.set_spmv(kind)
        d = torch.full_like(b, 0.5)
        it, normr, hist, st = M.cg_device(b, d, 7, 0.0)
        runs.append((it, normr, hist, st, d.cpu().numpy()))
    for g, w in zip(*runs):
        assert np.array_equal(g, w)


def _mixed_rows(rng, n, npat):
    """A CSR of n rows with npat patterns of up to 27 entries (one of them full)."""
    pats = []
    for k in range(npat):
        w = 27 if k < 3 else int(rng.integers(0, 28))
        lo, hi = ((0, 41) if k == 0 else (-40, 1) if k == 1 else (-40, 41))
        off = np.sort(rng.choice(np.arange(lo, hi), w, replace=False))
        val = rng.choice([0.0, -0.0, 1.5, -2.0, 1e300, 5e-324, 0.1], w) + 0.0 * off
        pats.append((off, val))
    which = rng.integers(0, npat, n)
    which[:40], which[-40:] = 0, 1  # columns stay inside
    cols = [pats[p][0] + i + 1 for i, p in enumerate(which)]
    rowindex = np.concatenate([[1], 1 + np.cumsum([len(c) for c in cols])]).astype(np.int32)
    return rowindex, np.concatenate(cols).astype(np.int32), np.concatenate([pats[p][1] for p in which])


@pytest.mark.parametrize("nx,ny,nz", [(80, 80, 90), (96, 96, 96), (104, 104, 64), (131, 97, 60)])
def test_box_walks_equal_ell_one_block_an_sm(env, nx, ny, nz):
    """Grids whose walk has one block to two per SM, above the one-kernel CG's limit."""
    test_box_walks_equal_ell(env, nx, ny, nz)


@pytest.mark.parametrize("n,npat", [(100, 3), (1000, 32), (5001, 31), (5001, 33), (20000, 400)])
def test_patterns_of_other_matrices(env, n, npat):
    """Matrices that are no stencil, up to and beyond the number of patterns kept
    (more: the ELL kernels run); infinities reach the same rows as in the ELL."""
    torch, hp = env
    rng = np.random.default_rng(n + npat)
    M = hp.Matrix.from_csr(*_mixed_rows(rng, n, npat))
    x = rng.uniform(-1, 1, n)
    x[n // 2] = np.inf
    got, want = _products(torch, hp, M, hp.SPMV_AUTO, x), _products(torch, hp, M, hp.SPMV_ELL, x)
    for g, w in zip(got, want):
        assert np.array_equal(g, w, equal_nan=True)


@pytest.mark.parametrize("nx,ny,nz", [(3, 3, 3), (4, 4, 16), (16, 16, 17), (37, 32, 32), (19, 31, 65), (37, 64, 32),
                                      (43, 43, 41), (101, 101, 102), (102, 102, 101)])
def test_one_kernel_cg(env, nx, ny, nz):
    """Row counts around one row a thread in blocks of 256 and 512, several rows a
    thread, and the largest system of the one-kernel form (and one beyond it).
    FP64 dots of n terms differ by n 2^-53 of their terms at most; the bars are the
    history bars of the CG tests (1e-12 of the residual, of the first one once it
    has fallen by 1e8) and 1e-10 for x."""
    torch, hp = env
    M = hp.Matrix.generated(nx, ny, nz)
    n = M.nrow
    xs = torch.from_numpy(np.random.default_rng(n).uniform(-1, 1, n)).cuda()
    b = torch.empty_like(xs)
    M.spmv(xs, b)
    for max_iter, tol in ((0, 0.0), (1, 0.0), (12, 0.0), (200, 1e-9)):
        runs = []
        for kind in (hp.SPMV_AUTO, hp.SPMV_ELL):
            M.set_spmv(kind)
            x = torch.full_like(b, 0.25)
            it, normr, hist, st = M.cg_device(b, x, max_iter, tol * float(torch.linalg.vector_norm(b)))
            runs.append((it, normr, hist, st, x.cpu().numpy()))
        (i0, n0, h0, s0, x0), (i1, n1, h1, s1, x1) = runs
        assert (i0, s0) == (i1, s1)
        band = np.where(h1 >= 1e-8 * h1[0], h1, h1[0]) * 1e-12
        assert (np.abs(h0 - h1) <= band).all() and abs(n0 - n1) <= band[-1]
        assert np.abs(x0 - x1).max() <= 1e-10


def test_mixed_graph_follows_the_grid(env):
    """A CSR solved in mixed precision before and after its grid is declared: the second solve
    runs the box walk (the first one's graph holds the gathers), with the same bits."""
    torch, hp = env
    from torch.profiler import ProfilerActivity, profile

    nx, ny, nz = 96, 96, 96
    M = hp.Matrix.from_csr(*hp.generate_matrix(nx, ny, nz)[:3])
    b = torch.from_numpy(np.random.default_rng(4).uniform(-1, 1, M.nrow)).cuda()
    for prec in (hp.PREC_FP32, hp.PREC_BF16):
        runs = []
        for grid in (False, True):
            if grid:
                M.set_geometry(nx, ny, nz)
            with profile(activities=[ProfilerActivity.CUDA], acc_events=True) as prof:
                x = torch.zeros_like(b)
                info, st = M.solve_mixed_device(b, x, prec, 1e-8)
                torch.cuda.synchronize()
            assert st == hp.HPCCG_OK
            inner = {e.key for e in prof.key_averages() if "k_mp_spmv_dot" in e.key}
            if not inner:
                pytest.skip("the profiler reports no kernels here")
            assert all(("StratLpBox" if grid else "StratLpPattern") in k for k in inner), inner
            runs.append((info.outer_iters, x))
        M.close()
        M = hp.Matrix.from_csr(*hp.generate_matrix(nx, ny, nz)[:3])
        assert float((runs[0][1] - runs[1][1]).abs().max()) <= 1e-6
