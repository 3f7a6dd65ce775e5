"""Convolutions as windows over an image on the tensor cores, at the edges of their tiling: planes around the 8 x 16
pixel tile, one tile and many, kernels and strides in every parity, channel counts around the 16/32/64-byte pixel rows and
the 64-channel chunks, more columns than one block.  References: the binary64 path and the binary64 forward pass."""
import numpy as np
import pytest
import torch
import torch.nn.functional as F

from ny_b200 import workloads as W

pytestmark = pytest.mark.gpu

# in (c, h, w), convolutions (channels, kernel, stride, padding)
NETS = [
    ((1, 5, 5), ((1, 1, 1, 0), (2, 3, 1, 1))),
    ((3, 16, 8), ((15, 3, 1, 1), (17, 3, 2, 1))),
    ((2, 17, 9), ((16, 4, 2, 1), (33, 3, 1, 0))),
    ((4, 15, 31), ((31, 5, 3, 2), (5, 2, 2, 0))),
    ((16, 9, 10), ((64, 3, 1, 1), (65, 3, 2, 1))),
    ((7, 13, 20), ((66, 4, 4, 0), (130, 3, 1, 1))),
    ((5, 12, 12), ((8, 1, 2, 0), (20, 7, 1, 3))),
    # the backward pass takes windows where an im2col product space is large beside a tile's products (the others above it does
    # not): the same edges with more input channels
    ((40, 17, 9), ((16, 3, 1, 1),)),
    ((130, 10, 9), ((65, 3, 1, 1),)),
    ((9, 31, 17), ((16, 5, 3, 2),)),
    ((20, 12, 12), ((20, 7, 1, 3),)),
    ((64, 16, 16), ((64, 3, 1, 1), (64, 3, 2, 1))),
]


@pytest.mark.parametrize("in_chw,convs", NETS)
def test_window_convolutions_match_binary64(in_chw, convs):
    from ny_b200 import B200Engine, engine

    wl = W.config_cnn(seed=61, eps=0.02, n_fix=3, in_chw=in_chw, convs=convs, fcs=(11, 4))
    D, out = 67, {}
    g = np.random.Generator(np.random.PCG64(5))
    x0 = (wl.in_lo + g.random((D, len(wl.in_lo)), dtype=np.float32) * (wl.in_hi - wl.in_lo)).astype(np.float32)
    for path in (engine.PATH_TF32X3, engine.PATH_F64):
        eng = B200Engine(0)
        eng.set_path(path)
        eng.set_refine_tolerance(3e38)   # nothing is evaluated again in binary64
        nid = eng.register_network(wl.net)
        pl, pu = eng.ibp_forward_gpu(nid, wl.in_lo, wl.in_hi)
        splits, ns = W.draw_domains(wl, pl[0], pu[0], D)
        lo, hi, inf = eng.bab_bound_batch(nid, wl.spec, wl.in_lo, wl.in_hi, pl[0], pu[0], splits, ns, mode=0)
        best, bx, _ = eng.pgd_attack(nid, wl.spec, wl.in_lo, wl.in_hi, x0, 0, 0.01)
        stepped = eng.pgd_attack(nid, wl.spec, wl.in_lo, wl.in_hi, x0, 1, 0.01)[0]
        out[path] = (pl[0], pu[0], lo, hi, inf, best, stepped)
        eng.close()
    tl, tu, tlo, thi, tinf, tbest, tstep = out[engine.PATH_TF32X3]
    fl, fu, flo, fhi, finf, fbest, fstep = out[engine.PATH_F64]
    mag = np.maximum(np.abs(fl), np.abs(fu)).max()
    assert np.all(np.abs(tl - fl) <= 1e-5 * mag) and np.all(np.abs(tu - fu) <= 1e-5 * mag)
    ok = ~finf.astype(bool)
    assert np.array_equal(tinf, finf) and ok.any()
    scale = max(np.abs(flo[ok]).max(), np.abs(fhi[ok]).max())
    # every rounding is charged: the bounds are the wider ones, up to the slopes' own rounding, and close
    assert np.all(np.abs(tlo - flo)[ok] <= 1e-4 * scale) and np.all(np.abs(thi - fhi)[ok] <= 1e-4 * scale)
    want = (W.forward(wl.net, x0) @ wl.spec.astype(np.float64).T).min(axis=1)
    assert np.allclose(tbest, want, rtol=1e-5, atol=2e-6 * np.abs(want).max())
    assert np.allclose(tstep, fstep, rtol=1e-4, atol=1e-4 * np.abs(want).max())


# (input channels, output channels, kernel, stride, padding).  From 64 channels on a pixel's high and low parts are tiles of their own
# in one ring, which holds low and high ones in turn where the number of slots is odd: 3 slots, forward and back, back on two chunks of
# channels and on three (5), forward on four chunks, then 4 to 8 forward, and the union of a stride's parities back (3).
RINGS = [(64, 64, (3, 3), 1, 1), (64, 128, (3, 3), 1, 1), (64, 192, (3, 3), 1, 1), (256, 16, (3, 3), 1, 1), (64, 16, (5, 5), 1, 2),
         (64, 16, (4, 4), 1, 1), (64, 32, (3, 3), 1, 1), (64, 16, (4, 3), 1, 1), (64, 16, (3, 3), 1, 1), (64, 64, (4, 4), 2, 1)]
# Tiles of one or two chains, of which the accumulators hold several: 64, 32 and 16 columns, one and two tiles in the ring.
RINGS += [(16, 64, (1, 1), 1, 0), (16, 32, (2, 2), 1, 0), (16, 16, (1, 1), 1, 0), (32, 64, (2, 2), 1, 0), (64, 64, (1, 1), 1, 0), (64, 32, (1, 1), 1, 0),
          (64, 16, (1, 2), 1, 0)]


@pytest.mark.parametrize("ring", RINGS)
def test_a_ring_of_many_tiles(ring):
    """Every tile of a long launch is multiplied from its own data: values and gradients of one layer over about seven tiles a
    CTA, twice with the same bits, against binary64 with the products' rounding rate (at most 2.5e-6 of the sum of
    magnitudes, win_eps).  A tile taken for another one is off by that sum's order itself."""
    from ny_b200 import B200Engine, Conv2d, Network, engine

    ic, oc, (kh, kw), s, pad = ring
    g = np.random.default_rng(ic + oc + kh)
    h, w = 48 * s, 24 * s
    wt = g.standard_normal((oc, ic, kh, kw)).astype(np.float32)
    layer = Conv2d(wt, np.zeros(oc, np.float32), (s, s), (pad, pad), (h, w))
    rows = max(37, 5000 // (9 * max(4, (oc + 15) // 16)))
    n1 = oc * layer.oh * layer.ow
    x = g.standard_normal((rows, ic * h * w), dtype=np.float32)
    spec = np.copysign(g.random((rows, n1), dtype=np.float32) + np.float32(0.5), g.random((rows, n1), dtype=np.float32) - np.float32(0.5))
    eng = B200Engine(0)
    eng.set_path(engine.PATH_TF32X3)
    nid = eng.register_network(Network([layer], [None]))
    grads, values = eng.point_vjp_batched(nid, spec, x=x)
    for _ in range(3):
        again = eng.point_vjp_batched(nid, spec, x=x)
        assert np.array_equal(again[0], grads) and np.array_equal(again[1], values)
    eng.close()
    dev = "cuda:0"
    t = torch.from_numpy(wt).to(dev).double()
    extra = [(h + 2 * pad - kh) % s, (w + 2 * pad - kw) % s]
    for r0 in range(0, rows, 16):
        a = torch.from_numpy(spec[r0:r0 + 16]).to(dev).double().reshape(-1, oc, layer.oh, layer.ow)
        xi = torch.from_numpy(x[r0:r0 + 16]).to(dev).double().reshape(-1, ic, h, w)
        got = torch.from_numpy(grads[r0:r0 + 16]).to(dev).double().reshape(xi.shape)
        err = (got - F.conv_transpose2d(a, t, None, s, pad, extra)).abs()
        assert (err <= 3e-6 * F.conv_transpose2d(a.abs(), t.abs(), None, s, pad, extra)).all()
        val = (a * F.conv2d(xi, t, None, s, pad)).flatten(1).sum(1).cpu().numpy()
        mag = (a.abs() * F.conv2d(xi.abs(), t.abs(), None, s, pad)).flatten(1).sum(1).cpu().numpy()
        assert np.all(np.abs(values[r0:r0 + 16] - val) <= 3e-6 * mag)
