"""Which lower line an unstable neuron takes (slope 1 where u > -l, else 0) is a step function of its interval: a rounding
that decides a tie the other way moves single bounds by up to a percent.  The interval pass of a batch of 64 domains and
more is made of TF32 pairs whose bits every release keeps, so the choices are the same ones: their digests over whole
batches are recorded in tests/golden/slopes.json (numpy seeds, inherited bounds too wide to count, so that the intervals
are the device's alone)."""
import hashlib
import json
import os

import numpy as np
import pytest

from ny_b200 import SPLIT_DTYPE
from ny_b200 import workloads as W

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "slopes.json")

NETS = {
    "mlp-784-8x256": (lambda: W.make_mlp([784] + [256] * 8 + [10], 43), 0.02, 4096),
    "mlp-100-4x130": (lambda: W.make_mlp([100] + [130] * 4 + [5], 42), 0.03, 2000),
    "mlp-300-3x512": (lambda: W.make_mlp([300] + [512] * 3 + [10], 46), 0.015, 777),
    "cnn-3x32x32": (lambda: W.make_cnn(44, (3, 32, 32), ((16, 4, 2, 1), (32, 4, 2, 1)), (100, 10)), 2.0 / 255.0, 1024),
    "resnet-3x16x16": (lambda: W.make_resnet(45, (3, 16, 16), 16, 2, 10), 2.0 / 255.0, 300),
}


def evaluate(name, refine, path=None):
    """Bounds of the batch, then u > -l of every hidden neuron of every domain (False where it is not unstable) and the
    unstable ones."""
    from ny_b200 import B200Engine

    make, eps, D = NETS[name]
    net = make()
    g = np.random.Generator(np.random.PCG64(D))
    x0 = g.random(net.dims[0], dtype=np.float32)
    lo, hi = x0 - np.float32(eps), x0 + np.float32(eps)
    wide = np.full(net.n_pre, 1e30, np.float32)
    n_hidden, offs = sum(net.dims[1:-1]), np.concatenate([[0], np.cumsum(net.dims[1:-1])])
    edges = np.linspace(0, n_hidden, 7).astype(np.int64)      # one split from each sixth: no neuron twice
    pick = edges[:-1] + (g.random((D, 6)) * np.diff(edges)).astype(np.int64)
    sp = np.zeros((D, 6), SPLIT_DTYPE)
    sp["relu"] = np.searchsorted(offs, pick, side="right") - 1
    sp["neuron"] = pick - offs[sp["relu"]]
    sp["sign"] = np.where(g.random((D, 6)) < 0.5, 1, -1)
    eng = B200Engine(0)
    if path is not None:
        eng.set_path(path)
    eng.set_refine_tolerance(refine)
    nid = eng.register_network(net)
    eng.batch_upload(nid, W.margin_spec(net.dims[-1], 0)[:2], lo, hi, -wide, wide, sp, np.full(D, 6, np.int32), 1)
    eng.batch_run()
    bounds = eng.batch_download()
    l, u = eng.batch_download_pre_bounds()
    eng.close()
    l, u = l[:, :n_hidden], u[:, :n_hidden]
    unstable = (l < 0) & (u > 0)
    return bounds, (u > -l) & unstable, unstable


def digest(up, unstable):
    return {"unstable": int(unstable.sum()), "slope_1": int(up.sum()), "sha256": hashlib.sha256(np.packbits(up).tobytes()).hexdigest()}


@pytest.mark.parametrize("name", list(NETS))
def test_slopes_are_the_recorded_ones(name):
    with open(GOLDEN) as f:
        assert digest(*evaluate(name, 0.0)[1:]) == json.load(f)[name]   # 0: the tensor path's intervals in every domain


@pytest.mark.parametrize("name", list(NETS))
def test_bounds_of_the_two_paths_differ_beyond_their_roundings_only_at_a_tie(name):
    """Domains whose neurons all take the same line on the tensor path and in binary64 agree to 1e-4 of their bounds (1 % of
    the domain's largest where a row cancels); a tie may be decided either way, and such domains are few."""
    from ny_b200 import engine

    (tl, tu, ti), tup, _ = evaluate(name, 5e-5)
    (fl, fu, fi), fup, _ = evaluate(name, 5e-5, engine.PATH_F64)
    assert np.array_equal(ti, fi)
    feas = fi == 0
    got, want = np.concatenate([tl, tu], 1), np.concatenate([fl, fu], 1)
    den = np.maximum(np.abs(want), 1e-2 * np.abs(want).max(axis=1, keepdims=True))
    off = feas & (np.abs(got - want) > 1e-4 * den).any(axis=1)
    tie = (tup != fup).any(axis=1)
    assert not np.any(off & ~tie), np.flatnonzero(off & ~tie)[:5]


def test_interval_convolution_in_slices_is_that_of_smaller_batches():
    """A convolution's product space is bounded: 340 domains of 13 MB each take two slices, and every domain's interval ends
    are bit for bit those of a batch that fits into one."""
    from ny_b200 import B200Engine

    net = W.make_cnn(46, (3, 16, 16), ((64, 3, 1, 1), (128, 5, 1, 2)), (4,))
    g = np.random.Generator(np.random.PCG64(1))
    D, x0 = 340, g.random(net.dims[0], dtype=np.float32)
    lo = (x0 - g.random((D, net.dims[0]), dtype=np.float32) * np.float32(0.02)).astype(np.float32)
    hi = (x0 + np.float32(0.02)).astype(np.float32)[None].repeat(D, 0)
    wide = np.full(net.n_pre, 1e30, np.float32)
    eng = B200Engine(0)
    eng.set_refine_tolerance(0.0)
    nid = eng.register_network(net)

    def ends(a, b):
        eng.batch_upload(nid, W.margin_spec(4, 0)[:1], lo[a:b], hi[a:b], -wide, wide, np.zeros((b - a, 0), SPLIT_DTYPE), np.zeros(b - a, np.int32), 1)
        eng.batch_run()
        eng.batch_download()
        return eng.batch_download_pre_bounds()

    whole, first, last = ends(0, D), ends(0, 200), ends(200, D)
    for i in range(2):
        assert np.array_equal(whole[i][:200], first[i]) and np.array_equal(whole[i][200:], last[i])
    eng.close()


def test_interval_convolution_of_more_domains_than_a_grid_has_rows():
    from ny_b200 import B200Engine

    net = W.make_cnn(47, (1, 4, 4), ((2, 3, 1, 1), (3, 3, 1, 1)), (2,))
    g = np.random.Generator(np.random.PCG64(2))
    D = 65600
    lo = g.random((D, 16), dtype=np.float32)
    hi = lo + np.float32(0.05)
    wide = np.full(net.n_pre, 1e30, np.float32)
    eng = B200Engine(0)
    eng.set_refine_tolerance(0.0)
    nid = eng.register_network(net)

    def bounds(a, b):
        return eng.bab_bound_batch(nid, W.margin_spec(2, 0), lo[a:b], hi[a:b], -wide, wide, np.zeros((b - a, 0), SPLIT_DTYPE), np.zeros(b - a, np.int32))

    whole, last = bounds(0, D), bounds(D - 200, D)
    for i in range(2):
        assert np.all(np.isfinite(whole[i])) and np.allclose(whole[i][-200:], last[i], rtol=1e-5, atol=1e-5)
    eng.close()
