"""Relaxation between convolutions straight into the next one's operand: the whole bound on the tensor path, with the
re-evaluation off, against binary64 contractions, whose pass goes layer by layer, over the forms the layers' rule
accepts and refuses: channel counts at the edges of a warp's share and of the padding, odd images, strides, pixel-major
and planar sources, identity branches that join and that are kept, more rows than a block holds, large multipliers.

Slopes are given, so no tie decides a line; the bounds then differ by the tensor products' roundings, which are charged.
A window layer's rate is at most 2.5e-6 of a row's sum of magnitudes (win_eps), an im2col one's 3e-6, and up to six layers
charge it: 2e-5 of that sum on either end.  The sum is taken as ten times the domain's largest bound (these networks' rows
cancel no further) and what its multipliers add: each times the largest magnitude of the neuron it stands at."""
import numpy as np
import pytest
import torch
import torch.nn.functional as F

from ny_b200 import SPLIT_DTYPE
from ny_b200 import workloads as W
from test_gpu_rates import _f16_rate, _transposed_rate

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    from ny_b200 import B200Engine

    e = B200Engine(0)
    yield e
    e.close()


def _conv(g, ci, co, k, s, p, hw):
    from ny_b200 import Conv2d

    return Conv2d((g.standard_normal((co, ci, k, k)) * np.sqrt(2.0 / (ci * k * k))).astype(np.float32),
                  (g.standard_normal(co) * 0.1).astype(np.float32), (s, s), (p, p), hw)


def _net(chw, convs, skips, n_out, seed):
    from ny_b200 import Network

    g = np.random.default_rng(seed)
    c, h, w = chw
    layers = []
    for co, k, s, p in convs:
        layers.append(_conv(g, c, co, k, s, p, (h, w)))
        c, h, w = co, layers[-1].oh, layers[-1].ow
    n = c * h * w
    fc = (g.standard_normal((n_out, n)) * np.sqrt(2.0 / n)).astype(np.float32)
    return Network(layers + [fc], [None] * len(layers) + [(g.standard_normal(n_out) * 0.1).astype(np.float32)], skips)


K3 = (3, 1, 1)   # kernel, stride, padding
CASES = [
    # image, convolutions, identity branches, specification rows, domains, multipliers
    ((3, 12, 10), [(12, *K3), (20, 4, 2, 1)], {}, 1, 70, 1.0),
    ((2, 9, 7), [(16, *K3), (33, *K3), (36, *K3)], {}, 3, 70, 1.0),          # 33 channels: no image of that layer
    ((3, 7, 9), [(64, *K3), (96, *K3), (64, *K3)], {}, 4, 66, 1.0),          # 96 channels: padded to 128
    ((3, 8, 8), [(160, *K3), (32, *K3), (128, *K3)], {}, 2, 64, 1.0),        # 160: too many for a block
    ((3, 8, 8), [(16, *K3)] * 5, {2: 0, 4: 2}, 9, 70, 1.0),                  # stem by im2col, branches kept and joined
    ((3, 16, 16), [(64, *K3)] * 5, {2: 0, 4: 2}, 5, 64, 1.0),
    ((3, 8, 8), [(16, *K3)] * 5, {2: 0, 4: 0}, 2, 70, 1.0),                  # two branches join one layer: not in one pass
    ((3, 8, 8), [(16, *K3)] * 5, {3: 0, 4: 1}, 2, 70, 1.0),                  # overlapping branches
    ((3, 13, 11), [(16, 4, 2, 1), (32, 4, 2, 1)], {}, 40, 20, 1.0),          # 80 rows a domain; few domains
    ((3, 16, 12), [(8, 4, 2, 1), (16, 4, 2, 1), (24, 3, 3, 0)], {}, 6, 66, 80.0),
]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_rows_through_images_agree_with_binary64(eng, case):
    from ny_b200 import engine

    chw, convs, skips, S, D, scale = CASES[case]
    net = _net(chw, convs, skips, S + 1, 90 + case)
    g = np.random.default_rng(190 + case)
    n0 = int(net.dims[0])
    x = g.uniform(0, 1, n0).astype(np.float32)
    lo, hi = (x - 0.02).astype(np.float32), (x + 0.02).astype(np.float32)
    spec = W.margin_spec(S + 1, 0)[:S]
    nid = eng.register_network(net)
    pl, pu = eng.ibp_forward_gpu(nid, lo, hi)
    rl, ru = pl[0], pu[0]
    offs = np.concatenate([[0], np.cumsum(net.dims[1:-1])])
    unstable = np.flatnonzero((rl[:offs[-1]] < 0) & (ru[:offs[-1]] > 0))
    n = 6
    edges = np.linspace(0, len(unstable), n + 1).astype(np.int64)
    pick = unstable[edges[:-1] + (g.random((D, n)) * (edges[1:] - edges[:-1])).astype(np.int64)]
    relu = np.searchsorted(offs, pick, side="right") - 1
    sp = np.zeros((D, n), SPLIT_DTYPE)
    sp["relu"], sp["neuron"] = relu, pick - offs[relu]
    sp["sign"] = np.where(g.random((D, n)) < 0.5, 1, -1)
    sp["beta"] = scale * g.random((D, n), dtype=np.float32)
    ns = np.full(D, n, np.int32)
    alpha = g.random((D, net.n_pre), dtype=np.float32)
    out = {}
    eng.set_refine_tolerance(0.0)
    for path in (engine.PATH_TF32X3, engine.PATH_F64):
        eng.set_path(path)
        out[path] = eng.bab_bound_batch(nid, spec, lo, hi, rl, ru, sp, ns, 1, alpha)
    eng.set_refine_tolerance(5e-5)
    eng.set_path(engine.PATH_AUTO)
    eng.release_network(nid)
    (l, u, inf), (fl, fu, finf) = out[engine.PATH_TF32X3], out[engine.PATH_F64]
    assert np.array_equal(inf, finf)
    fin = np.isfinite(fl) & np.isfinite(fu)          # large multipliers empty a row: repaired to infinities
    assert np.array_equal(np.isfinite(l) & np.isfinite(u), fin) and fin.mean() > 0.9
    size = np.where(fin, np.maximum(np.abs(fl), np.abs(fu)), 0.0).max(axis=1, keepdims=True)
    total = 10.0 * size + (sp["beta"] * np.maximum(np.abs(rl), np.abs(ru))[pick]).sum(axis=1, keepdims=True)
    for got, want in ((l, fl), (u, fu)):
        off = np.abs(got - want)
        assert (off <= 2e-5 * total)[fin].all()
        assert np.median((off / size)[fin]) <= 1e-4


def _exact(net, spec, lo, hi, rl, ru, sp, alpha):
    """Bounds of the same lines in plain binary64, and per row what the layers' rounding rates charge: each layer's rate times the
    sum of |coefficient| q, q its weights' magnitudes times its inputs'; and the sum of q alone."""
    D, S, L = len(sp), len(spec), len(net.weights)
    offs = np.concatenate([[0], np.cumsum(net.dims[1:])])
    code, beta = np.zeros((D, offs[-1])), np.zeros((D, offs[-1]))
    at = offs[sp["relu"]] + sp["neuron"]
    np.put_along_axis(code, at, sp["sign"].astype(float), 1)
    np.put_along_axis(beta, at, (sp["sign"] * sp["beta"]).astype(float), 1)
    t = lambda x: torch.from_numpy(np.ascontiguousarray(x)).to("cuda:0").double()
    code, beta, l, u, al = t(code), t(beta), t(rl).expand(D, -1), t(ru).expand(D, -1), t(alpha)
    l, u = torch.where(code > 0, l.clamp(min=0), l), torch.where(code < 0, u.clamp(max=0), u)
    on, off = (code > 0) | (l >= 0), (code < 0) | ((code <= 0) & (u <= 0))
    us = torch.where(on, 1.0, torch.where(off, 0.0, u / (u - l).clamp(min=1e-8)))
    ls, ui = torch.where(on, 1.0, torch.where(off, 0.0, al)), torch.where(on | off, 0.0, -us * l)

    def forward(k, z):
        w = net.weights[k]
        if k == L - 1:
            return z @ t(w).abs().T
        return F.conv2d(z.reshape(-1, w.ic, w.ih, w.iw), t(w.weight).abs(), None, (w.sh, w.sw), (w.ph, w.pw)).flatten(1)

    def back(k, a):
        w = net.weights[k]
        if k == L - 1:
            return a @ t(w)
        pad = [(n + 2 * p - kk) % s for n, p, kk, s in ((w.ih, w.ph, w.weight.shape[2], w.sh), (w.iw, w.pw, w.weight.shape[3], w.sw))]
        return F.conv_transpose2d(a.reshape(-1, w.oc, w.oh, w.ow), t(w.weight), None, (w.sh, w.sw), (w.ph, w.pw), pad).flatten(1)

    xl, xu = t(lo), t(hi)
    z = [torch.maximum(xl.abs(), xu.abs()).expand(D, -1)] + [torch.where(code < 0, 0.0, u.clamp(min=0))[:, offs[k]:offs[k + 1]] for k in range(L - 1)]
    a = t(np.concatenate([spec, spec])).repeat(D, 1)
    upper = (torch.arange(2 * S, device=a.device) >= S).repeat(D)[:, None]
    sign, rows = torch.where(upper, 1.0, -1.0), lambda x: x.repeat_interleave(2 * S, 0)
    const, charge, floor, kept = torch.zeros(len(a), device=a.device).double(), 0.0, 0.0, {}
    for k in range(L - 1, -1, -1):
        b = net.biases[k] if k == L - 1 else np.repeat(net.weights[k].bias, net.weights[k].oh * net.weights[k].ow)
        q = rows(forward(k, z[k]))
        w = net.weights[k]
        rate = _f16_rate(net.dims[L]) if k == L - 1 else _transposed_rate(w.ic, w.oc, w.weight.shape[2], w.sh, w.ph, w.oh, w.ow, w.ih, w.iw)[0]
        const, charge, floor = const + a @ t(b), charge + rate * (a.abs() * q).sum(1), floor + q.sum(1)
        if k in net.skips:
            kept[net.skips[k]] = kept.get(net.skips[k], 0.0) + a
        a = back(k, a)
        if k:
            j = slice(offs[k - 1], offs[k])
            a = a + kept.get(k - 1, 0.0)
            line = (a > 0) == upper        # the upper line, or the lower one
            const = const + torch.where(line, a * rows(ui[:, j]), 0.0).sum(1)
            a = torch.where(line, a * rows(us[:, j]), a * rows(ls[:, j])) + sign * rows(beta[:, j])
    take = (a >= 0) == upper
    bound = (const + torch.where(take, a * xu, a * xl).sum(1)).reshape(D, 2, S).cpu().numpy()
    return bound[:, 0], bound[:, 1], charge.reshape(D, 2, S).cpu().numpy(), floor.reshape(D, 2, S).cpu().numpy()


@pytest.mark.parametrize("scale", [1.0, 5e-32])
@pytest.mark.parametrize("case", range(len(CASES)))
def test_every_rounding_is_charged_outwards(eng, case, scale):
    """A lower bound lies below the same lines' bound in plain binary64, an upper one above it, by what the layers charge, each at its
    products' rate (window, im2col, fully connected): a twentieth is left for the actual roundings, which are a tenth of
    their rates, and a quarter on top for the lines' own charges; rows of tiny coefficients, whose scale ends near fp32's,
    add the share of the exponent range (1.1e-37 of the weights' and inputs' magnitudes).  A layer whose charge is lost, or
    charged to the wrong side, falls short."""
    from ny_b200 import engine

    chw, convs, skips, S, D, mult = CASES[case]
    net = _net(chw, convs, skips, S + 1, 90 + case)
    g = np.random.default_rng(290 + case)
    x = g.uniform(0, 1, int(net.dims[0])).astype(np.float32)
    lo, hi = (x - 0.02).astype(np.float32), (x + 0.02).astype(np.float32)
    spec = (W.margin_spec(S + 1, 0)[:S] * np.float32(scale)).astype(np.float32)
    nid = eng.register_network(net)
    pl, pu = eng.ibp_forward_gpu(nid, lo, hi)
    offs = np.concatenate([[0], np.cumsum(net.dims[1:-1])])
    unstable = np.flatnonzero((pl[0, :offs[-1]] < 0) & (pu[0, :offs[-1]] > 0))
    edges = np.linspace(0, len(unstable), 5).astype(np.int64)
    pick = unstable[edges[:-1] + (g.random((D, 4)) * (edges[1:] - edges[:-1])).astype(np.int64)]
    relu = np.searchsorted(offs, pick, side="right") - 1
    sp = np.zeros((D, 4), SPLIT_DTYPE)
    sp["relu"], sp["neuron"] = relu, pick - offs[relu]
    sp["sign"] = np.where(g.random((D, 4)) < 0.5, 1, -1)
    sp["beta"] = np.float32(scale * min(mult, 2.0)) * g.random((D, 4), dtype=np.float32)
    alpha = g.random((D, net.n_pre), dtype=np.float32)
    eng.set_refine_tolerance(0.0)
    eng.set_path(engine.PATH_TF32X3)
    got_l, got_u, inf = eng.bab_bound_batch(nid, spec, lo, hi, pl[0], pu[0], sp, np.full(D, 4, np.int32), 0, alpha)   # the inherited intervals as they are
    eng.set_refine_tolerance(5e-5)
    eng.set_path(engine.PATH_AUTO)
    eng.release_network(nid)
    want_l, want_u, charge, floor = _exact(net, spec, lo, hi, pl[0], pu[0], sp, alpha)
    assert not inf.any() and np.isfinite(got_l).all() and np.isfinite(got_u).all()
    for short, c, f in ((want_l - got_l, charge[:, 0], floor[:, 0]), (got_u - want_u, charge[:, 1], floor[:, 1])):
        assert (short >= 0.95 * c).all(), (short / c).min()
        assert (short <= 1.25 * c + 1.1e-37 * f).all(), (short / c).max()
