"""Slopes that cross the bus beside the interval pass (one-call bounds of large batches) give the bounds of slopes that were
uploaded before it, bit for bit: fully connected and convolutional networks, widths that leave the rows unpadded, infinite
and NaN slopes, split neurons among them; and the branching pick over rows whose last neurons are not a whole group of four
is the first largest width."""
import numpy as np
import pytest

from ny_b200 import SPLIT_DTYPE
from ny_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", ["wide", "ragged", "chain", "cnn", "few"])
def test_late_slopes_are_the_uploaded_ones(case):
    from ny_b200 import B200Engine

    g = np.random.default_rng(17)
    net, D = {"wide": (W.make_mlp([20, 300, 300, 300, 4], 3), 400), "ragged": (W.make_mlp([20, 301, 299, 203, 4], 4), 400),
              "chain": (W.make_mlp([20, 256, 256, 256, 4], 5), 500), "cnn": (W.make_cnn(6, (3, 16, 16), ((16, 4, 2, 1), (32, 4, 2, 1)), (50, 4)), 200),
              "few": (W.make_cnn(7, (3, 28, 28), ((16, 3, 1, 1), (16, 4, 2, 1)), (40, 4)), 40)}[case]
    n0 = int(net.dims[0])
    x = g.uniform(0, 1, n0).astype(np.float32)
    lo, hi = x - np.float32(0.03), x + np.float32(0.03)
    spec = W.margin_spec(4, 1)
    eng = B200Engine(0)
    nid = eng.register_network(net)
    pl, pu = eng.ibp_forward_gpu(nid, lo, hi)
    rl, ru = pl[0], pu[0]
    offs = np.concatenate([[0], np.cumsum(net.dims[1:-1])])
    unstable = np.flatnonzero((rl[:offs[-1]] < 0) & (ru[:offs[-1]] > 0))
    pick = g.choice(unstable, (D, 3))
    pick.sort(axis=1)
    sp = np.zeros((D, 3), SPLIT_DTYPE)
    relu = np.searchsorted(offs, pick, side="right") - 1
    sp["relu"], sp["neuron"] = relu, pick - offs[relu]
    sp["sign"] = np.where(pick % 2 == 0, 1, -1)       # (a neuron picked twice has one sign)
    sp["beta"] = 0.5
    ns = np.full(D, 3, np.int32)
    alpha = g.uniform(-0.2, 1.2, (D, net.n_pre)).astype(np.float32)
    alpha[::7, ::5] = np.nan
    alpha[::9, ::4] = np.inf
    assert alpha.nbytes >= 1 << 20
    args = (nid, spec, lo, hi, rl, ru, sp, ns, 1, alpha)
    once = eng.bab_bound_batch(*args)
    again = eng.bab_bound_batch(*args)                # the second call's interval pass beside the first one's buffers
    eng.batch_upload(*args)
    eng.batch_run()
    want = eng.batch_download()
    for a, b, c in zip(once, again, want):
        assert np.array_equal(a, c) and np.array_equal(b, c)
    eng.close()


def test_a_given_up_call_leaves_its_batch_resident():
    from ny_b200 import B200Engine, EngineError, engine

    g = np.random.default_rng(23)
    net, D = W.make_mlp([20, 300, 300, 300, 4], 3), 400
    x = g.uniform(0, 1, 20).astype(np.float32)
    lo, hi = x - np.float32(0.03), x + np.float32(0.03)
    spec = W.margin_spec(4, 1)
    eng = B200Engine(0)
    nid = eng.register_network(net)
    pl, pu = eng.ibp_forward_gpu(nid, lo, hi)
    alpha = g.uniform(0, 1, (D, net.n_pre)).astype(np.float32)
    assert alpha.nbytes >= 1 << 20
    args = (nid, spec, lo, hi, pl[0], pu[0], np.zeros((D, 0), SPLIT_DTYPE), np.zeros(D, np.int32), 1, alpha)
    want = eng.bab_bound_batch(*args)
    eng.bab_bound_batch(*args[:-1], np.zeros_like(alpha))   # other slopes in the batch's place
    eng.set_deadline(0.0)
    with pytest.raises(EngineError) as ei:
        eng.bab_bound_batch(*args)
    assert ei.value.code == engine.DEADLINE and "deadline" in str(ei.value)
    eng.set_deadline(None)
    eng.batch_run()
    for a, b in zip(eng.batch_download(), want):
        assert np.array_equal(a, b)
    eng.close()


@pytest.mark.parametrize("widths", [(5, 6), (64, 66), (130, 127), (301, 3)])
def test_branching_picks_the_first_widest(widths):
    from ny_b200 import B200Engine

    eng = B200Engine(0)
    net = W.make_mlp([6, *widths, 3], 9)
    g = np.random.default_rng(widths[0])
    x = g.uniform(-1, 1, 6).astype(np.float32)
    lo, hi = x - np.float32(0.3), x + np.float32(0.3)
    nid = eng.register_network(net)
    pl, pu = eng.ibp_forward_gpu(nid, lo, hi)
    rl, ru = pl[0], pu[0]
    hidden = sum(widths)
    ties = (rl[:hidden] < 0) & (ru[:hidden] > 0)
    rl, ru = rl.copy(), ru.copy()
    rl[:hidden][ties] = np.maximum(rl[:hidden][ties], -0.25)   # many equal widths
    ru[:hidden][ties] = np.minimum(ru[:hidden][ties], 0.25)
    D = 70
    eng.batch_upload(nid, W.margin_spec(3, 0), lo, hi, rl, ru, np.zeros((D, 0), SPLIT_DTYPE), np.zeros(D, np.int32), 0)
    eng.batch_run()
    relu, neuron, width = eng.batch_select_branch()[:3]
    w = np.where((rl[:hidden] < 0) & (ru[:hidden] > 0), ru[:hidden] - rl[:hidden], -1).astype(np.float32)
    i = int(np.argmax(w))
    r = 0 if i < widths[0] else 1
    assert (np.asarray(relu) == r).all() and (np.asarray(neuron) == i - r * widths[0]).all() and np.allclose(width, w[i])
    eng.close()
