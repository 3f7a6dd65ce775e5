"""Rounding charges of the upper lines' intercepts.  The fused chain sums them in fp32 and charges each sum through the coefficients
behind the relaxation (|a intercept| <= |a slope| max|z|).  Lines that do not keep to that are charged all the same: neurons whose
width lies below the relaxation's smallest, where the slope is u / 1e-8 and the intercept close to u, and tables of the caller's."""
from fractions import Fraction

import numpy as np
import pytest

from ny_b200 import SPLIT_DTYPE, Network
from ny_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _net(width, n_out, seed):
    """The last layer's weights have 10 significant bits, so that their products with unit rows are exact on every path."""
    g = np.random.default_rng(seed)
    net = W.make_mlp([6, width, width, n_out], seed)
    last = (g.integers(512, 1024, (n_out, width)) / 1024.0 * g.choice([-1, 1], (n_out, width))).astype(np.float32)
    ws = [*net.weights[:-1], last]
    return Network(ws, [np.zeros(w.shape[0], np.float32) for w in ws])


def test_intercepts_of_the_smallest_widths_are_charged():
    from ny_b200 import B200Engine, engine

    width, n_out, D = 64, 9, 70
    net = _net(width, n_out, 3)
    u = np.float32(2.0 ** -40)
    rl = np.concatenate([np.full(width, -1, np.float32), np.full(width, -u, np.float32), np.full(n_out, -10, np.float32)])
    ru = np.concatenate([np.full(width, -0.5, np.float32), np.full(width, u, np.float32), np.full(n_out, 10, np.float32)])
    eng = B200Engine(0)
    eng.set_path(engine.PATH_TF32X3)
    eng.set_refine_tolerance(1e30)
    nid = eng.register_network(net)
    x = np.zeros(6, np.float32)
    lo, hi, _ = eng.bab_bound_batch(nid, np.eye(n_out, dtype=np.float32), x, x + 1, rl, ru, np.zeros((D, 0), SPLIT_DTYPE),
                                    np.zeros(D, np.int32), 0)
    # the first hidden layer is inactive, so the bounds are the intercepts' sums and their charges: with slope u / 1e-8 the
    # intercept is u (1 - slope), rounded up
    icp = float(u) * (1 - float(u) / 1e-8)
    a = net.weights[-1].astype(np.float64)
    mine = np.stack([np.minimum(a, 0), np.maximum(a, 0)]).sum(axis=2) * icp      # lower and upper rows
    eps = 0.75 * 2.0 ** -20 + 4 * 2.0 ** -23           # the first product's rounding: operand split, accumulation (less than charged)
    charge = eps * np.abs(a).sum(axis=1) * float(u) + 16 * 2.0 ** -24 * np.abs(mine)
    slack = 2.0 ** -22 * np.abs(mine)                  # fp32 result, the intercepts' directed rounding
    assert np.all(lo <= mine[0] - charge[0] + slack[0]) and np.all(hi >= mine[1] + charge[1] - slack[1])
    assert np.all(lo >= mine[0] - 4 * charge[0] - slack[0]) and np.all(hi <= mine[1] + 4 * charge[1] + slack[1])
    eng.close()


@pytest.mark.parametrize("width,rows", [(64, 9), (260, 9), (260, 1)])
def test_lines_of_the_caller_with_steep_intercepts_are_charged(width, rows):
    """Constant upper lines (slope 0): nothing is left of the coefficients that the intercepts' sums could be charged through."""
    from ny_b200 import B200Engine, engine

    D = 700 if width > 256 else 70
    net = _net(width, rows, width + rows)
    zero, half = np.zeros(width, np.float32), np.full(width, 0.5, np.float32)
    # a sum of 1 and seven terms of 2^-25: one behind the other in fp32 they are all lost
    icp = np.full(width, 0.75, np.float32)
    icp[:8] = [2.0, *[2.0 ** -24] * 7]
    w = net.weights
    w[-1][:, 8:] = 0
    w[-1][:, :8] = np.where(np.arange(rows) % 2, 0.5, -0.5)[:, None]
    layers = [("linear", w[2], net.biases[2]), ("act", zero, zero, None, icp), ("linear", w[1], net.biases[1]), ("act", zero, zero, None, half),
              ("linear", w[0], net.biases[0])]
    small = np.full(width, 1e-30, np.float32)
    one = {"layers": layers, "lo": np.zeros(6, np.float32), "hi": np.ones(6, np.float32), "node_abs": [small, small], "beta_signed": [zero, zero]}
    eng = B200Engine(0)
    eng.set_path(engine.PATH_TF32X3)
    eng.set_refine_tolerance(1e30)
    lo, hi = eng.crown_resnet_beta_batched([one] * D, np.eye(rows, dtype=np.float32))
    assert (lo == lo[0]).all() and (hi == hi[0]).all()
    for s in range(rows):
        terms = [Fraction(float(a)) * Fraction(float(i)) for a, i in zip(w[2][s], icp)]
        below, above = sum(t for t in terms if t < 0), sum(t for t in terms if t > 0)
        assert Fraction(float(lo[0, s])) <= below and Fraction(float(hi[0, s])) >= above
        assert float(lo[0, s]) >= float(below) * (1 + 1e-6) - 1e-30 and float(hi[0, s]) <= float(above) * (1 + 1e-6) + 1e-30
    eng.close()
