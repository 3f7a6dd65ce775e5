"""The adjoint step takes two neurons a thread on even places and one elsewhere, several domains of a narrow layer to a block;
the relaxation by domains takes its rows three at a time: three Adam iterations on the tensor path against binary64, to the
1e-3 that a gradient component near zero allows (its sign decides a step)."""
import numpy as np
import pytest

from ny_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,rows,domains", [(31, 3, 70), (66, 1, 130), (128, 9, 90), (258, 5, 66)])
def test_optimised_bounds_at_odd_and_narrow_widths(width, rows, domains):
    from ny_b200 import SPLIT_DTYPE, B200Engine, engine

    eng = B200Engine(0)
    net = W.make_mlp([20, width, width, rows + 1], 600 + width)
    g = np.random.default_rng(700 + width)
    x = g.uniform(0, 1, 20).astype(np.float32)
    lo, hi = x - np.float32(0.05), x + np.float32(0.05)
    cl, ch = np.repeat(lo[None], domains, 0), np.repeat(hi[None], domains, 0)
    ch[::2, 3] = x[3]
    cl[1::2, 3] = x[3]
    spec = W.margin_spec(rows + 1, 0)[:rows]
    nid = eng.register_network(net)
    pl, pu = eng.ibp_forward_gpu(nid, lo, hi)
    out = {}
    for path in (engine.PATH_TF32X3, engine.PATH_F64):
        eng.set_path(path)
        eng.batch_upload(nid, spec, cl, ch, pl[0], pu[0], np.zeros((domains, 0), SPLIT_DTYPE), np.zeros(domains, np.int32), 1)
        eng.batch_optimize(3, 0.1, 0.0)
        out[path] = eng.batch_download()[0]
    eng.close()
    got, want = out[engine.PATH_TF32X3], out[engine.PATH_F64]
    assert np.isfinite(want).all()
    assert (np.abs(got - want) <= 1e-3 * np.maximum(np.abs(want), 0.1 * np.abs(want).max(axis=1, keepdims=True))).all()


# 400 threads an SM for pairs of neurons: on 148 of them 59200 threads are the line
@pytest.mark.parametrize("width,rows,domains", [(64, 1, 1849), (64, 1, 1850), (258, 2, 460)])
def test_optimised_bounds_on_both_sides_of_the_line_for_pairs(width, rows, domains):
    test_optimised_bounds_at_odd_and_narrow_widths(width, rows, domains)


# with dual alpha 800 threads: 118400 threads are the line
@pytest.mark.parametrize("width,rows,domains", [(64, 1, 3699), (64, 1, 3700)])
def test_dual_slopes_on_both_sides_of_the_line_for_pairs(width, rows, domains):
    """Every other domain has one of two boxes: within a batch equal domains come out equal, and on the two paths within 1e-3."""
    from ny_b200 import SPLIT_DTYPE, B200Engine, engine

    eng = B200Engine(0)
    net = W.make_mlp([20, width, width, rows + 1], 81)
    g = np.random.default_rng(82)
    x = g.uniform(0, 1, 20).astype(np.float32)
    lo, hi = np.repeat((x - np.float32(0.05))[None], domains, 0), np.repeat((x + np.float32(0.05))[None], domains, 0)
    hi[::2, 3] = lo[1::2, 3] = x[3]
    nid = eng.register_network(net)
    pl, pu = eng.ibp_forward_gpu(nid, lo[0], (x + np.float32(0.05)))
    out = []
    for path in (engine.PATH_TF32X3, engine.PATH_F64):
        eng.set_path(path)
        eng.batch_upload(nid, W.margin_spec(rows + 1, 0)[:rows], lo, hi, pl[0], pu[0], np.zeros((domains, 0), SPLIT_DTYPE), np.zeros(domains, np.int32), 0)
        eng.batch_optimize(3, 0.1, 0.0, objective=2)
        lower, upper, _ = eng.batch_download()
        b = np.concatenate([lower, upper], 1)
        assert np.isfinite(b).all() and (np.ptp(b[::2], axis=0) <= 1e-3 * np.abs(b).max()).all() and (np.ptp(b[1::2], axis=0) <= 1e-3 * np.abs(b).max()).all()
        out.append(b)
    eng.close()
    assert (np.abs(out[0] - out[1]) <= 1e-3 * np.abs(out[1]).max()).all()
