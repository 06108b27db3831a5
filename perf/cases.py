"""The solver and network calls whose speed is measured, over the sizes they are used at.

Each case is one call (or one short sequence of calls) of the public Python interface
(hpccg_b200 / hpccg_b200.learned) on a workload of the kinds that the driver, the bench
and the tests run: FP64 CG on a stored matrix, FP64 CG with the matrix-free operator,
mixed precision on both, batches of uneven systems, the U-Net forward and backward, the
network-preconditioned solve, and the op-level calls.  Right-hand sides are b = A x* with
x* uniform in [-1, 1), so x* is the exact solution.
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "hpccg-f90_b200"))

import hpccg_b200 as hp  # noqa: E402
from hpccg_b200 import learned  # noqa: E402


def listed():
    return [
        # The driver's own run: a CSR from the host generator, 150 iterations at tolerance 0,
        # b and x in host memory.  Small enough that launches and latency are what counts.
        dict(name="cg_host_32", kind="cg_host", nx=32, ny=32, nz=32, max_iter=150, tol=0.0),
        # The plain FP64 CG at 128^3, 500 iterations (2.1M rows, 55M nonzeros), device arrays.
        dict(name="cg_stored_128", kind="cg_stored", nx=128, ny=128, nz=128, max_iter=500, tol=0.0),
        # An uploaded CSR with odd edges, solved to a tolerance: no grid is declared.
        dict(name="cg_csr_97x75x61", kind="cg_csr", nx=97, ny=75, nz=61, max_iter=500, tol=1e-10),
        # FP64 CG with the matrix-free operator on a large uneven grid.
        dict(name="cg_free_256x192x160", kind="cg_free", nx=256, ny=192, nz=160, max_iter=500, tol=1e-10),
        # The headline solve: FP32 matrix-free inner CG inside FP64 refinement at 256^3.
        dict(name="mixed_free_256", kind="mixed_free", nx=256, ny=256, nz=256, precision=1, tol=1e-8),
        # BF16 values of a stored matrix inside FP64 refinement, odd edges.
        dict(name="mixed_stored_150x131x97", kind="mixed_stored", nx=150, ny=131, nz=97, precision=2, tol=1e-8),
        # 64 independent systems, edges uniform in [16, 96]: matrix-free FP32 with refinement.
        dict(name="batch_free_64", kind="batch_free", nsys=64, lo=16, hi=96, sizes=7, precision=1, tol=1e-8),
        # The same kind of batch with fewer systems on the stacked stored matrix, FP64.
        dict(name="batch_stored_32", kind="batch_stored", nsys=32, lo=16, hi=64, sizes=11, precision=0, tol=1e-8),
        # One application of the network on the benchmark's grid.
        dict(name="unet_forward_256", kind="forward", nx=256, ny=256, nz=256, nb=1),
        # One training step's loss and gradient, at the training loop's own size and batch.
        dict(name="unet_grad_64x4", kind="grad", nx=64, ny=64, nz=64, nb=4),
        # The learned solve: FP64 refinement around the network-preconditioned FP32 flexible CG.
        dict(name="learned_128", kind="learned", nx=128, ny=128, nz=128, tol=1e-8),
        # The op-level calls a host program makes when it drives its own iteration.
        dict(name="ops_24", kind="ops", nx=24, ny=24, nz=24),
    ]


def draw(rng):
    def edge(lo, hi, step=1):
        return step * max(1, round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step))

    def grid(lo, hi, step=1):
        return dict(nx=edge(lo, hi, step), ny=edge(lo, hi, step), nz=edge(lo, hi, step))

    kind = rng.choice(["cg_host", "cg_stored", "cg_csr", "cg_free", "mixed_free", "mixed_stored", "batch_free",
                       "batch_stored", "forward", "grad", "learned", "ops"])
    tol = rng.choice([1e-6, 1e-8, 1e-10])
    if kind == "cg_host":
        return dict(kind=kind, **grid(16, 64), max_iter=150, tol=tol)
    if kind in ("cg_stored", "cg_csr"):
        return dict(kind=kind, **grid(16, 128), max_iter=500, tol=tol)
    if kind == "cg_free":
        return dict(kind=kind, **grid(16, 200), max_iter=500, tol=tol)
    if kind == "mixed_free":
        return dict(kind=kind, **grid(16, 256), precision=1, tol=tol)
    if kind == "mixed_stored":
        return dict(kind=kind, **grid(16, 150), precision=rng.choice([1, 2]), tol=tol)
    if kind in ("batch_free", "batch_stored"):
        lo = edge(8, 32)
        return dict(kind=kind, nsys=edge(4, 64), lo=lo, hi=lo + edge(4, 48), sizes=rng.randrange(1 << 20),
                    precision=rng.choice([0, 1]), tol=tol)
    if kind == "forward":
        return dict(kind=kind, **grid(16, 256, 8), nb=1)
    if kind == "grad":
        return dict(kind=kind, **grid(16, 64, 8), nb=rng.randint(1, 4))
    if kind == "learned":
        return dict(kind=kind, **grid(32, 128, 8), tol=1e-8)
    return dict(kind=kind, **grid(4, 160))


# ---- inputs -------------------------------------------------------------------------------


def _uniform(n, seed, dtype=torch.float64):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.rand(n, generator=g, device="cuda", dtype=dtype) * 2 - 1


def _box3(v, d):
    s = v.clone()
    n = v.shape[d]
    if n > 1:
        s.narrow(d, 1, n - 1).add_(v.narrow(d, 0, n - 1))
        s.narrow(d, 0, n - 1).add_(v.narrow(d, 1, n - 1))
    return s


def _apply(x, nx, ny, nz):
    """The 27-point operator in plain torch: 28 x - (sum over the 3x3x3 neighbourhood)."""
    v = x.reshape(nz, ny, nx)
    return (28 * v - _box3(_box3(_box3(v, 2), 1), 0)).reshape(-1)


def _sizes(case):
    return hp.batch_sizes(case["sizes"], case["nsys"], case["lo"], case["hi"])


def _multilevel_weights(net, seed):
    """Weights of a network that sums the residual averaged to every level (an additive
    multilevel preconditioner), the other channels as a fresh network has them: what a
    program that loads a trained network has in hand."""
    layers = [(1, 0)] + [(16, 1)] * 7 + [(32, 2), (16, 1), (32, 2), (16, 1), (32, 2)]
    scale = {8: (1.0, 1.0), 10: (1.0, 1.0), 12: (1.0, 1.0)}  # decoder joins: own level, level below
    rng = np.random.RandomState(seed % (1 << 31))
    out = []
    for i, (cin, _) in enumerate(layers):
        w = (rng.uniform(-1, 1, (27, cin, 16)) * math.sqrt(6.0 / (27 * cin))).astype(np.float32)
        w[:, :, :2] = 0
        c = np.zeros((cin, 2), np.float32)  # channels 0 and 1: the positive and the negative part
        if i == 0:
            c[0] = (1, -1)
        else:
            for g, s in enumerate(scale.get(i, (1.0,))):
                c[16 * g:16 * g + 2] = np.array([[s, -s], [-s, s]], np.float32)
        w[13, :, :2] = c
        out += [w.reshape(-1), np.zeros(16, np.float32)]
    proj = np.zeros(17, np.float32)
    proj[:2] = (1 / 27, -1 / 27)
    net.set_params(np.concatenate(out + [proj]))


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case)
    if kind in ("batch_free", "batch_stored"):
        sizes = _sizes(case)
        B = hp.Batch.generated(sizes)
        if kind == "batch_free":
            B.set_spmv(hp.SPMV_STENCIL)
        b = torch.zeros(B.stacked_rows, dtype=torch.float64, device="cuda")
        for i, (nx, ny, nz) in enumerate(sizes.tolist()):
            n, o = nx * ny * nz, int(B.offsets[i])
            b[o:o + n] = _apply(_uniform(n, seed * 1000 + i), nx, ny, nz)
        s.update(B=B, b=b, x=torch.zeros_like(b))
        return s
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    if kind in ("forward", "grad"):
        net = hp.Unet(seed + 1)
        s.update(net=net, inp=_uniform(n * case["nb"], seed, torch.float32))
        if kind == "grad":
            net.set_loss(1)  # the loss of the training loop
            s.update(tgt=0.1 * _uniform(n * case["nb"], seed + 17, torch.float32))
        else:
            s.update(out=torch.empty_like(s["inp"]))
        return s
    if kind in ("cg_host", "cg_csr"):
        rowindex, colindex, values = hp.generate_matrix(nx, ny, nz)[:3]
        s["M"] = hp.Matrix.from_csr(rowindex, colindex, values)
    else:
        s["M"] = hp.Matrix.generated(nx, ny, nz)
    if kind in ("cg_free", "mixed_free", "learned"):
        s["M"].set_spmv(hp.SPMV_STENCIL)
    xs = _uniform(n, seed)
    if kind == "ops":
        s.update(x=xs, y=torch.empty_like(xs), w=torch.empty_like(xs))
        return s
    b = _apply(xs, nx, ny, nz)
    s.update(b=b, bnorm=float(torch.linalg.vector_norm(b)), x=torch.zeros_like(b))
    if kind == "cg_host":
        s.update(b=b.cpu().numpy())
    if kind == "learned":
        s["net"] = hp.Unet(1)
        _multilevel_weights(s["net"], 3)
    return s


# ---- one pass -----------------------------------------------------------------------------


def run(s):
    kind = s["kind"]
    if kind == "cg_host":
        x, niters, _, hist, _ = s["M"].cg(s["b"], np.zeros_like(s["b"]), s["max_iter"], s["tol"] * s["bnorm"])
        return {"x": x, "hist": hist, "niters": niters}
    if kind in ("cg_stored", "cg_csr", "cg_free"):
        s["x"].zero_()
        niters, _, hist, _ = s["M"].cg_device(s["b"], s["x"], s["max_iter"], s["tol"] * s["bnorm"])
        return {"x": s["x"], "hist": hist, "niters": niters}
    if kind in ("mixed_free", "mixed_stored"):
        s["x"].zero_()
        info, _ = s["M"].solve_mixed_device(s["b"], s["x"], s["precision"], s["tol"])
        return {"x": s["x"], "cycles": int(info.outer_iters)}
    if kind in ("batch_free", "batch_stored"):
        s["x"].zero_()
        s["B"].solve(s["b"], s["x"], s["precision"], s["tol"])
        return {"x": s["x"]}
    if kind == "forward":
        s["net"].forward(s["inp"], s["out"], s["nx"], s["ny"], s["nz"], s["nb"])
        return {"out": s["out"]}
    if kind == "grad":
        loss, grad = s["net"].loss_grad(s["inp"], s["tgt"], s["nx"], s["ny"], s["nz"], s["nb"], want_grad=True)
        return {"loss": np.float32(loss), "grad": grad}
    if kind == "learned":
        s["x"].zero_()
        learned.solve_mixed_fcg(s["M"], s["net"], (s["nx"], s["ny"], s["nz"]), s["b"], s["x"], s["tol"])
        return {"x": s["x"]}
    s["M"].spmv(s["x"], s["y"])
    dot = s["M"].ddot(s["x"], s["y"])
    s["M"].waxpby(1.0, s["x"], -0.5, s["y"], s["w"])
    return {"y": s["y"], "dot": dot, "w": s["w"]}


# ---- what a pass cannot do without ----------------------------------------------------------


def _iterations(nx, ny, nz, tol):
    """About the CG iterations of the 27-point operator on these grids for a random x*."""
    return max(10, int(math.log10(1.0 / tol) * 5.5))


def work(case):
    kind = case["kind"]
    if kind in ("batch_free", "batch_stored"):
        sizes = _sizes(case).astype(np.int64)
        n = int(sizes.prod(axis=1).sum())
        nnz = int((3 * sizes - 2).prod(axis=1).sum())
        stored = 12 * nnz if kind == "batch_stored" else 0
        return {"bytes": stored + 24 * n, "flops": _iterations(1, 1, 1, case["tol"]) * (2 * nnz + 10 * n)}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    nnz = (3 * nx - 2) * (3 * ny - 2) * (3 * nz - 2)
    if kind in ("forward", "grad"):
        v = n * case["nb"]
        flops = 0
        for lvl, convs in enumerate(((1, 16, 32), (16, 16, 32, 16), (16, 16, 32, 16), (16, 16))):
            flops += sum(2 * 27 * c * 16 for c in convs) * (v >> (3 * lvl))
        flops += 2 * 16 * v
        if kind == "grad":  # the input and the weight gradients cost a forward each
            return {"bytes": 8 * v, "flops": 3 * flops}
        return {"bytes": 8 * v, "flops": flops}
    if kind == "ops":
        return {"bytes": 12 * nnz + 24 * n, "flops": 2 * nnz + 5 * n}
    stored = kind in ("cg_host", "cg_stored", "cg_csr", "mixed_stored")
    if case["tol"] == 0.0:
        iters = case["max_iter"]
    else:
        iters = _iterations(nx, ny, nz, case["tol"])
    return {"bytes": (12 * nnz if stored else 0) + 24 * n, "flops": iters * (2 * nnz + 10 * n)}


# ---- the same in 64 bits, in plain torch ----------------------------------------------------


def _split(params):
    """[(W [27, cin, 16], bias [16])] per layer and the projection's 17 numbers."""
    cins = [1] + [16] * 7 + [32, 16, 32, 16, 32]
    out, o = [], 0
    for cin in cins:
        w = params[o:o + 27 * cin * 16].reshape(27, cin, 16)
        o += 27 * cin * 16
        out.append((w, params[o:o + 16]))
        o += 16
    return out, params[o:o + 17]


def _conv(x, wb):
    """3x3x3 convolution of [b, z, y, x, cin] with zeros outside the grid, then ReLU."""
    w, bias = wb
    _, nz, ny, nx, _ = x.shape
    p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
    y = bias
    for t in range(27):
        z0, y0, x0 = t // 9, t // 3 % 3, t % 3
        y = y + p[:, z0:z0 + nz, y0:y0 + ny, x0:x0 + nx] @ w[t]
    return torch.relu(y)


def _pool(x):
    b, nz, ny, nx, c = x.shape
    return x.reshape(b, nz // 2, 2, ny // 2, 2, nx // 2, 2, c).mean(dim=(2, 4, 6))


def _up(x):
    return x.repeat_interleave(2, 1).repeat_interleave(2, 2).repeat_interleave(2, 3)


def _network(params, x):
    L, proj = _split(params)
    e1 = _conv(_conv(x, L[0]), L[1])
    e2 = _conv(_conv(_pool(e1), L[2]), L[3])
    e3 = _conv(_conv(_pool(e2), L[4]), L[5])
    e4 = _conv(_conv(_pool(e3), L[6]), L[7])
    c3 = _conv(_conv(torch.cat([e3, _up(e4)], -1), L[8]), L[9])
    c2 = _conv(_conv(torch.cat([e2, _up(c3)], -1), L[10]), L[11])
    c1 = _conv(torch.cat([e1, _up(c2)], -1), L[12])
    return c1 @ proj[:16] + proj[16]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("batch_free", "batch_stored"):
        B = []
        for i, (nx, ny, nz) in enumerate(_sizes(case).tolist()):
            n = nx * ny * nz
            B.append(torch.nn.functional.pad(_uniform(n, seed * 1000 + i), (0, -n % 512)))
        return {"x": torch.cat(B)}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    if kind in ("forward", "grad"):
        shape = (case["nb"], nz, ny, nx, 1)
        params = torch.from_numpy(hp.Unet(seed + 1).get_params()).cuda().double()
        inp = _uniform(n * case["nb"], seed, torch.float32).double().reshape(shape)
        if kind == "forward":
            with torch.no_grad():
                return {"out": _network(params, inp).reshape(-1)}
        params.requires_grad_(True)
        tgt = (0.1 * _uniform(n * case["nb"], seed + 17, torch.float32)).double().reshape(shape[:4])
        d = tgt - _network(params, inp)
        ad = 28 * d - _box3(_box3(_box3(d, 3), 2), 1)
        loss = (d * ad).mean()
        (grad,) = torch.autograd.grad(loss, params)
        return {"loss": loss.detach(), "grad": grad}
    xs = _uniform(n, seed)
    if kind == "ops":
        y = _apply(xs, nx, ny, nz)
        return {"y": y, "dot": float(xs @ y), "w": xs - 0.5 * y}
    return {"x": xs, "hist": None, "niters": None, "cycles": None}
