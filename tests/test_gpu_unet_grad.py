"""Weight and bias gradients of every layer against 64-bit sums of the same terms.

The network's weights are scaled permutations at the centre tap and its biases positive, so
every convolution is exact in FP32 and the oracle repeats the whole pass with the
kernels' own roundings (BF16 activations and masked gradients, FP32 sums of the loss, the
resampling and the skips).  What remains is the sum of each gradient over the voxels.

Bars: an accumulator takes at most eight MMAs between two drains, each a truncating sum in
FP32 that loses up to 4 units of 2^-24 of the terms' magnitudes, the drains and the
first layer's chains add at most 16 FP32 sums, and the result is rounded: 50 2^-24 of
sum |x dY| for any element; and 1e-6 of the norm of those sums for a layer, as the
roundings do not add up all in one direction.
"""
import numpy as np
import pytest

import unet_oracle as uo

pytestmark = pytest.mark.gpu
F = np.float32


@pytest.fixture(scope="module")
def env():
    import torch

    import hpccg_b200 as hp
    return torch, hp


def _exact_params(rng):
    off, n = uo.offsets()
    p = np.zeros(n, F)
    for l, (cin, _) in enumerate(uo.LAYERS):
        W = np.zeros((27, cin, 16), F)
        if cin == 1:
            W[13, 0] = 2.0 ** -rng.integers(0, 3, 16)
        else:
            for g in range(cin // 16):
                W[13, 16 * g + rng.permutation(16), np.arange(16)] = 0.5 if cin == 32 else 1.0
        p[off[l]:off[l] + W.size] = W.reshape(-1)
        p[off[l] + W.size:off[l + 1]] = rng.integers(1, 17, 16) / 32
    p[off[-1]:] = rng.choice([-1, 1], 17) * 2.0 ** -rng.integers(0, 3, 17)
    return p


def _sum8(d):
    """The eight fine children of each coarse voxel, added in FP32 in the order z, y, x."""
    s = np.zeros((d.shape[0], d.shape[1] // 2, d.shape[2] // 2, d.shape[3] // 2, 16), F)
    for k in range(8):
        s = s + d[:, k >> 2::2, (k >> 1) & 1::2, k & 1::2]
    return s


def _gradients(x, dy):
    """dW [27][cin][16] and dbias in FP64; the terms are those of voxels inside the grid."""
    x, dy = x.astype(np.float64), dy.astype(np.float64)
    out = np.zeros((27, x.shape[-1], 16))
    for t in range(27):
        xs, ds = [slice(None)], [slice(None)]
        for o, n in zip((t // 9 - 1, t // 3 % 3 - 1, t % 3 - 1), x.shape[1:4]):
            xs.append(slice(max(0, o), n + min(0, o)))
            ds.append(slice(max(0, -o), n + min(0, -o)))
        out[t] = x[tuple(xs)].reshape(-1, x.shape[-1]).T @ dy[tuple(ds)].reshape(-1, 16)
    return np.concatenate([out.reshape(-1), dy.reshape(-1, 16).sum(0)])


def _layers(params, r, tgt):
    """[(x, dY)] of the 13 layers, in the kernels' roundings."""
    Ws, bs, proj = uo.unpack(params.astype(np.float64))
    bf = uo.bf16_round

    def conv(l, *xs):
        pre = uo.conv3(np.concatenate(xs, -1).astype(np.float64), Ws[l], bs[l])
        assert np.array_equal(pre.astype(F), pre, equal_nan=True)  # exact in FP32
        return bf(np.nan_to_num(np.maximum(pre, 0), nan=0.0, posinf=np.inf))

    def pool(a):
        return bf(_sum8(a) * F(0.125))

    e1a = conv(0, r[..., None])
    e1b = conv(1, e1a)
    d1 = pool(e1b)
    e2a = conv(2, d1)
    e2b = conv(3, e2a)
    d2 = pool(e2b)
    e3a = conv(4, d2)
    e3b = conv(5, e3a)
    d3 = pool(e3b)
    e4a = conv(6, d3)
    e4b = conv(7, e4a)
    u3 = uo.up(e4b)
    c3a = conv(8, e3b, u3)
    c3b = conv(9, c3a)
    u2 = uo.up(c3b)
    c2a = conv(10, e2b, u2)
    c2b = conv(11, c2a)
    u1 = uo.up(c2b)
    c1 = conv(12, e1b, u1)
    out = c1.astype(np.float64) @ proj[:16] + proj[16]
    assert np.array_equal(out.astype(F), out)
    dout = (F(2) / F(out.size)) * (out.astype(F) - tgt)

    def mask(d, act):
        return bf(np.where(act > 0, d, 0))

    def back(l, d):
        dx = uo.conv3(d.astype(np.float64), Ws[l][::-1].transpose(0, 2, 1))
        assert np.array_equal(dx.astype(F), dx, equal_nan=True)
        return dx.astype(F)

    def skip(fine, coarse, act):  # the gradient of a skip tensor and of the pooled one below it
        return mask(fine + F(0.125) * uo.up(coarse), act)

    L = [None] * 13
    L[12] = (np.concatenate([e1b, u1], -1), mask(dout[..., None] * proj[:16].astype(F), c1))
    g = back(12, L[12][1])
    L[11] = (c2a, mask(_sum8(g[..., 16:]), c2b))
    L[10] = (np.concatenate([e2b, u2], -1), mask(back(11, L[11][1]), c2a))
    g2 = back(10, L[10][1])
    L[9] = (c3a, mask(_sum8(g2[..., 16:]), c3b))
    L[8] = (np.concatenate([e3b, u3], -1), mask(back(9, L[9][1]), c3a))
    g3 = back(8, L[8][1])
    L[7] = (e4a, mask(_sum8(g3[..., 16:]), e4b))
    L[6] = (d3, mask(back(7, L[7][1]), e4a))
    L[5] = (e3a, skip(g3[..., :16], back(6, L[6][1]), e3b))
    L[4] = (d2, mask(back(5, L[5][1]), e3a))
    L[3] = (e2a, skip(g2[..., :16], back(4, L[4][1]), e2b))
    L[2] = (d1, mask(back(3, L[3][1]), e2a))
    L[1] = (e1a, skip(g[..., :16], back(2, L[2][1]), e1b))
    L[0] = (r[..., None], mask(back(1, L[1][1]), e1a))
    return L


def _run(env, nx, ny, nz, nb, seed, poke=None):
    """Gradients of a random input and target; poke(r, tgt) changes them first.
    Yields (layer, device's, 64-bit, sum of magnitudes)."""
    torch, hp = env
    rng = np.random.default_rng(seed)
    net = hp.Unet(1)
    p = _exact_params(rng)
    net.set_params(p)
    r = (rng.integers(8, 256, (nb, nz, ny, nx)) / 64).astype(F)  # whole numbers of BF16
    tgt = rng.normal(0, 4, r.shape).astype(F)
    if poke:
        poke(r, tgt)
    with np.errstate(invalid="ignore", over="ignore"):
        L = _layers(p, r, tgt)
        want = [_gradients(*l) for l in L]
        mag = [_gradients(np.abs(x), np.abs(d)) for x, d in L]
    _, g = net.loss_grad(torch.from_numpy(r).cuda(), torch.from_numpy(tgt).cuda(), nx, ny, nz, nb, want_grad=True)
    off, _ = uo.offsets()
    for l in range(13):
        yield l, g[off[l]:off[l + 1]].astype(np.float64), want[l], mag[l]


SHAPES = [(16, 16, 16, 1), (24, 16, 40, 2), (136, 24, 8, 1), (40, 72, 16, 3), (64, 64, 64, 1)]


@pytest.mark.parametrize("nx,ny,nz,nb", SHAPES)
def test_every_layers_gradient_sums(env, nx, ny, nz, nb):
    for l, got, want, mag in _run(env, nx, ny, nz, nb, nx + nz):
        err = np.abs(got - want)
        assert (err <= 50 * 2.0 ** -24 * mag).all(), (l, (err / mag).max())
        assert np.linalg.norm(err) <= 1e-6 * np.linalg.norm(mag), l


@pytest.mark.parametrize("nx,ny,nz,nb", SHAPES[:4])
@pytest.mark.parametrize("last", [False, True])
@pytest.mark.parametrize("what", ["input", "target"])
def test_gradients_with_a_non_finite_corner(env, nx, ny, nz, nb, last, what):
    """An infinite input or target at a corner of a grid reaches the sums that have a term of
    it: taps that leave the grid there keep their finite sums, the others are what the
    64-bit sums are."""
    at = (nb - 1, nz - 1, ny - 1, nx - 1) if last else (0, 0, 0, 0)

    def poke(r, tgt):
        (r if what == "input" else tgt)[at] = np.inf

    seen = 0
    for l, got, want, mag in _run(env, nx, ny, nz, nb, nx + nz, poke):
        bad = ~np.isfinite(want)
        seen += bad.sum()
        assert np.array_equal(got[bad], want[bad], equal_nan=True), l
        assert (np.abs(got[~bad] - want[~bad]) <= 50 * 2.0 ** -24 * mag[~bad]).all(), l
    assert seen
