"""The rounding rates that every bound of the tensor path is charged with, element by element: |computed - exact| against
rate * sum |a||b| plus the share of fp16's exponent range, for the contraction on fp16 pairs (nyb200_umma16.cu) and for the
convolutions (nyb200_convwin.cu; transposed ones whose im2col products are the faster form: nyb200_umma.cu).  Products are taken through point_vjp_batched on networks of one layer: the
gradients of K rows are rows * W (a transposed convolution), the values with unit rows are the forward product.  Operands:
normal with rows of very different size, one sign (the largest accumulators), alternating (the most cancellation), and rows
of a few huge values among tiny ones (the exponent range)."""
import numpy as np
import pytest
import torch
import torch.nn.functional as F

from ny_b200 import Conv2d, Network

pytestmark = pytest.mark.gpu
U23, U24, SPLIT = 2.0 ** -23, 2.0 ** -24, 0.75 * 2.0 ** -20
KINDS = ("normal", "positive", "alternating", "range")


@pytest.fixture(scope="module")
def eng():
    from ny_b200 import B200Engine, engine

    e = B200Engine(0)
    e.set_path(engine.PATH_TF32X3)
    yield e
    e.close()


def _rows(g, m, k, kind):
    a = g.standard_normal((m, k)).astype(np.float32)
    if kind == "normal":
        a *= np.exp2(np.round(g.uniform(-30, 30, (m, 1)))).astype(np.float32)
    elif kind == "range":          # 2^30 between neighbours: the small ones lie below fp16's range beside the large ones
        a *= np.exp2(np.where(g.random((m, k)) < 0.03, 0.0, g.uniform(-45, -20, (m, k)))).astype(np.float32)
    else:
        a = (g.random((m, k)) + 0.5).astype(np.float32)
        if kind == "alternating":
            a[:, ::2] *= -1
    return a


def _weights(g, shape, kind):
    w = g.standard_normal(shape).astype(np.float32) if kind in ("normal", "range") else (g.random(shape) + 0.5).astype(np.float32)
    if kind == "range":            # as far as a layer may span and keep its fp16 pairs
        w *= np.exp2(np.round(g.uniform(-22, 0, shape))).astype(np.float32)
        w = np.where(np.abs(w) < np.abs(w).max() * 2.0 ** -26, np.abs(w).max() * np.float32(2.0 ** -26), w).astype(np.float32)
    return w


def _f16_rate(K):
    chunks, steps = (K + 63) // 64, min(4, (K + 15) // 16)
    lo = (chunks + 63) // 64
    hi = max(lo, min(64, chunks // 8))
    adds = max((chunks + n - 1) // n + (n if n > 1 else 0) for n in (lo, hi))
    return SPLIT + steps * U23 * (1 + 2 * 2.0 ** -10 * 1.001) + adds * U24


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("m,k,n", [(1, 1, 1), (5, 7, 3), (130, 15, 17), (64, 50, 50), (128, 64, 64), (129, 65, 130), (300, 256, 256),
                                   (1000, 10, 256), (513, 256, 784), (40, 1024, 33), (130, 4100, 20), (2000, 512, 512)])
def test_contraction_on_fp16_pairs(eng, m, k, n, kind):
    g = np.random.Generator(np.random.PCG64([m, k, n, KINDS.index(kind)]))
    a, w = _rows(g, m, k, kind), _weights(g, (k, n), kind)
    nid = eng.register_network(Network([w], [None]))
    got = eng.point_vjp_batched(nid, a, masks=np.zeros((m, k), np.float32)).astype(np.float64)
    eng.release_network(nid)
    a64, w64 = a.astype(np.float64), w.astype(np.float64)
    mag = np.abs(a64) @ np.abs(w64)
    # 2^-50 of a chunk's largest for every element of it that is too small beside it
    pad = -k % 64
    cm = np.abs(np.pad(a64, ((0, 0), (0, pad)))).reshape(m, -1, 64).max(axis=2)
    cw = np.abs(np.pad(w64, ((0, pad), (0, 0)))).reshape(-1, 64, n).sum(axis=1)
    bound = _f16_rate(k) * mag + 2.0 ** -50 * (cm @ cw)
    err = np.abs(got - a64 @ w64)
    assert np.all(err <= bound), float((err / bound).max())


# in (c, h, w), (channels, kernel, stride, padding): planes around the 8 x 16 tile, every tap parity, 16 / 32 / 64-channel pixels
CONVS = [((1, 5, 5), (1, 1, 1, 0)), ((16, 17, 9), (33, 3, 1, 1)), ((15, 16, 8), (17, 3, 2, 1)),
         ((4, 15, 31), (31, 5, 3, 2)), ((64, 9, 10), (65, 3, 1, 1)), ((66, 12, 20), (130, 3, 2, 1)), ((5, 12, 12), (20, 7, 1, 3)),
         # ... and where the transposed form takes windows too
         ((3, 32, 32), (16, 4, 2, 1)), ((7, 16, 8), (16, 3, 1, 1)), ((24, 17, 9), (15, 3, 1, 1)), ((56, 17, 9), (31, 3, 1, 0)), ((130, 10, 9), (65, 3, 1, 1)),
         ((5, 30, 30), (15, 3, 2, 1)), ((9, 31, 17), (16, 5, 3, 2)), ((20, 12, 12), (20, 7, 1, 3)), ((64, 16, 16), (64, 3, 2, 1))]


def _window(ic, oc, kh, kw, s, pad, kind):
    """(products of a MAIN chain, all products, chains) of a window convolution, as nyb200_convwin.cu lays it out."""
    cin = oc if kind == "transposed" else ic
    cp = 16 if cin <= 16 else 32 if cin <= 32 else (cin + 63) // 64 * 64
    ks, nchunk = min(cp, 64) * 2 // 32, max(1, cp // 64)
    if kind == "transposed":       # the union of the stride parities' windows
        def span(k):
            lo, hi = 1 << 30, -(1 << 30)
            for p in range(s):
                k0 = (p + pad) % s
                q, n = (p + pad - k0) // s, (k - k0 + s - 1) // s if k0 < k else 0
                if n:
                    lo, hi = min(lo, q - (n - 1)), max(hi, q)
            return hi - lo + 1
        taps = [span(kh) * span(kw)]
    else:
        taps = [((kh - ry + s - 1) // s) * ((kw - rx + s - 1) // s) for ry in range(min(s, kh)) for rx in range(min(s, kw))]
    tpc = max(1, 4 // ks)
    return tpc * ks, sum(taps) * nchunk * ks, sum(nchunk * ((t + tpc - 1) // tpc) for t in taps)


def _win_rate(*geom):
    chain, steps, chains = _window(*geom)
    return (SPLIT + chain * U23 + 2 * steps * U23 * 2.0 ** -10 + (chains + 1) * U24) * 1.000001


def _transposed_rate(ic, oc, k, s, p, oh, ow, h, w):
    tiles = -(-(-(-h // s)) // 16) * -(-(-(-w // s)) // 8)
    steps = _window(ic, oc, k, k, s, p, "transposed")[1]
    if oh * ow * ic * k * k >= 650 * steps * tiles:
        return _win_rate(ic, oc, k, k, s, p, "transposed"), True
    stages = (oc + 31) // 32                  # im2col products on TF32 pairs: K = oc, and the cast of the sum over the taps
    cs = 2 if stages >= 8 else 1
    cross = 8 * U23 * (cs - 1 + 2.0 ** -10)
    return (SPLIT + min(cs, stages) * 4 * U23 + cross + -(-stages // cs) * U24 + 5.97e-8) * 1.000001, False


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("chw,conv", CONVS)
def test_convolution_windows(eng, chw, conv, kind):
    (c, h, w), (oc, k, s, p) = chw, conv
    g = np.random.Generator(np.random.PCG64([c, h, oc, k, KINDS.index(kind)]))
    wt = _weights(g, (oc, c, k, k), kind)
    layer = Conv2d(wt, np.zeros(oc, np.float32), (s, s), (p, p), (h, w))
    nid = eng.register_network(Network([layer], [None]))
    n0, n1 = c * h * w, oc * layer.oh * layer.ow
    t = torch.from_numpy(wt).double()
    zero = np.zeros((1, n1), np.float32)

    def transposed(a, wt):
        extra = [(h + 2 * p - k) % s, (w + 2 * p - k) % s]     # rows and columns that no output reads
        return F.conv_transpose2d(torch.from_numpy(a).reshape(-1, oc, layer.oh, layer.ow), wt, None, s, p, extra).reshape(len(a), -1).numpy()

    m = 37
    a = _rows(g, m, n1, kind)
    got = eng.point_vjp_batched(nid, a, masks=zero.repeat(m, 0)).astype(np.float64)
    a64 = a.astype(np.float64)
    rest = transposed(np.ones((1, n1)), t.abs())
    rate, window = _transposed_rate(c, oc, k, s, p, layer.oh, layer.ow, h, w)
    assert window == (CONVS.index((chw, conv)) >= 7)
    bound = rate * transposed(np.abs(a64), t.abs()) + (2.0 ** -48 * np.abs(a64).max(axis=1, keepdims=True) + 1e-37) * rest
    err = np.abs(got - transposed(a64, t))
    assert np.all(err <= bound), float((err / np.maximum(bound, 1e-300)).max())

    # forward: one point in every row, the unit rows read its outputs
    x = _rows(g, 1, n0, kind)
    unit = np.zeros((min(n1, 600), n1), np.float32)
    at = g.permutation(n1)[: len(unit)]
    unit[np.arange(len(unit)), at] = 1.0
    _, val = eng.point_vjp_batched(nid, unit, x=x.repeat(len(unit), 0))
    eng.release_network(nid)
    xi = torch.from_numpy(x.astype(np.float64)).reshape(1, c, h, w)
    want, mag, ones = (F.conv2d(i, j, None, s, p).reshape(-1).numpy()[at] for i, j in ((xi, t), (xi.abs(), t.abs()), (torch.ones_like(xi), t.abs())))
    bound = _win_rate(c, oc, k, k, s, p, "forward") * mag + (2.0 ** -48 * np.abs(x).max() + 1e-37) * ones + U24 * np.abs(want)
    err = np.abs(val.astype(np.float64) - want)
    assert np.all(err <= bound), float((err / np.maximum(bound, 1e-300)).max())
