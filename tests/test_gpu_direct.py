"""The direct binary64 evaluation of fully connected networks (one kernel per backward pass) at the edges of its tiling:
widths around the eight-column tiles and the groups of sixteen, one row group and many, several sweeps over a wide
layer, one box and several, with and without split lists."""
import numpy as np
import pytest

from ny_b200 import SPLIT_DTYPE
from ny_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    from ny_b200 import B200Engine

    e = B200Engine(0)
    yield e
    e.close()


@pytest.mark.parametrize("boxes", [1, 5, 160])
@pytest.mark.parametrize("dims", [[3, 1, 2], [1, 7, 9, 3], [16, 8, 8, 8, 4], [9, 17, 130, 33, 5], [40, 64, 65, 63, 10], [20, 520, 300, 6]])
def test_direct_crown_matches_the_oracle(eng, oracle, dims, boxes):
    if boxes > 5 and max(dims) > 130:
        pytest.skip("the oracle takes too long at this size")
    net = W.make_mlp(dims, 300 + sum(dims))
    g = np.random.Generator(np.random.PCG64(boxes))
    mid = g.uniform(-1, 1, (boxes, dims[0])).astype(np.float32)
    lo, hi = mid - np.float32(0.03), mid + np.float32(0.03)
    spec = W.margin_spec(dims[-1], 0)
    onet = oracle.Net(net.weights, net.biases).with_spec(spec)
    nid = eng.register_network(net)
    glo, ghi, gil, giu = eng.crown_bounds(nid, spec, lo if boxes > 1 else lo[0], hi if boxes > 1 else hi[0])
    for d in range(0, boxes, max(1, boxes // 5)):
        olo, ohi = oracle.crown(onet, lo[d], hi[d])
        scale = max(np.abs(olo).max(), np.abs(ohi).max())   # the oracle carries the reference's (looser) error matrices
        assert np.all(np.abs(glo[d] - olo) <= 2e-4 * scale) and np.all(np.abs(ghi[d] - ohi) <= 2e-4 * scale), d
    # every point's outputs lie inside the bounds, of the rows and of the intermediate layers
    x = lo[:, None, :] + g.random((boxes, 64, dims[0])) * (hi - lo)[:, None, :].astype(np.float64)
    y = W.forward(net, x.reshape(-1, dims[0])) @ spec.astype(np.float64).T
    y = y.reshape(boxes, 64, -1)
    assert np.all(y.min(axis=1) >= glo - 1e-12) and np.all(y.max(axis=1) <= ghi + 1e-12)
    assert np.all(gil <= giu)
    # no split anywhere: the split entry point returns the plain bounds bit for bit
    sp, ns = np.zeros((boxes, 1), SPLIT_DTYPE), np.zeros(boxes, np.int32)
    slo, shi, sil, siu, inf = eng.crown_bounds_split(nid, spec, lo, hi, sp, ns)
    assert np.array_equal(slo, glo) and np.array_equal(shi, ghi) and np.array_equal(sil, gil) and not inf.any()
    eng.release_network(nid)


@pytest.mark.parametrize("dims,D", [([5, 9, 3], 1), ([17, 33, 15, 4], 3), ([96, 64, 64, 64, 10], 63), ([784, 256, 256, 256, 10], 7),
                                    ([40, 520, 130, 6], 2), ([30, 100, 301, 100, 10], 33)])
def test_direct_bound_of_a_few_domains_matches_the_oracle(eng, oracle, dims, D):
    """Batches of fewer than 64 domains: interval pass and backward pass in one kernel each (clusters of CTAs per domain and
    per group of rows), at ragged widths and row counts, split multipliers included."""
    net = W.make_mlp(dims, 500 + sum(dims) + D)
    g = np.random.Generator(np.random.PCG64(D))
    x0 = g.uniform(0, 1, dims[0]).astype(np.float32)
    wl = W.Workload("", net, x0, x0 - np.float32(0.02), x0 + np.float32(0.02), W.margin_spec(dims[-1], 1), 3, 500 + D)
    onet = oracle.Net(net.weights, net.biases)
    rl, ru = oracle.ibp_forward(onet, wl.in_lo, wl.in_hi)
    nid = eng.register_network(net)
    splits, ns = W.draw_domains(wl, rl, ru, D)
    lo, hi, inf = eng.bab_bound_batch(nid, wl.spec, wl.in_lo, wl.in_hi, rl, ru, splits, ns)
    S = wl.spec.shape[0]
    rl2 = np.concatenate([rl, np.full(S, -np.inf, np.float32)])
    ru2 = np.concatenate([ru, np.full(S, np.inf, np.float32)])
    olo, ohi, oinf, _ = oracle.bab_bound_batch(onet.with_spec(wl.spec), wl.in_lo, wl.in_hi, rl2, ru2, splits, ns, 1)
    f = ~oinf.astype(bool)
    assert np.array_equal(inf.astype(bool), oinf.astype(bool))
    both, want = np.concatenate([lo, hi], 1)[f], np.concatenate([olo, ohi], 1)[f]
    scale = np.abs(want).max(axis=1, keepdims=True)
    assert np.all(np.abs(both - want) <= 1e-4 * np.maximum(np.abs(want), 1e-2 * scale))
    assert np.all(lo[f] <= olo[f] + 1e-6 * scale) and np.all(hi[f] >= ohi[f] - 1e-6 * scale)
    # the same domains one per box: nothing is shared between them
    lo2, hi2, _ = eng.bab_bound_batch(nid, wl.spec, np.repeat(wl.in_lo[None], D, 0), np.repeat(wl.in_hi[None], D, 0), rl, ru, splits, ns)
    assert np.all(np.abs(lo2[f] - lo[f]) <= 1e-6 * scale) and np.all(np.abs(hi2[f] - hi[f]) <= 1e-6 * scale)
    eng.release_network(nid)


@pytest.mark.parametrize("dims,D", [([20, 33, 64, 5], 12), ([96, 64, 64, 64, 10], 40)])
def test_path_and_fusion_select_the_form(dims, D):
    """The default takes a few domains, and plain CROWN, directly in binary64; PATH_TF32X3 keeps both on the tensor cores and
    PATH_F64 with fusion off takes one launch per layer.  All agree to the roundings they charge."""
    from ny_b200 import B200Engine, engine

    net = W.make_mlp(dims, 600 + D)
    g = np.random.Generator(np.random.PCG64(D))
    x0 = g.uniform(0, 1, dims[0]).astype(np.float32)
    lo, hi, wide = x0 - np.float32(0.02), x0 + np.float32(0.02), np.full(net.n_pre, 1e30, np.float32)
    spec = W.margin_spec(dims[-1], 0)
    e = B200Engine(0)
    e.set_refine_tolerance(0.0)
    nid = e.register_network(net)

    def both(path, fusion):
        e.set_path(path)
        e.set_fusion(fusion)
        for _ in range(2):     # the second time without preparing operands
            n0 = e.launch_count()
            b = e.bab_bound_batch(nid, spec, lo, hi, -wide, wide, np.zeros((D, 0), SPLIT_DTYPE), np.zeros(D, np.int32))
            n1 = e.launch_count()
            c = e.crown_bounds(nid, spec, lo, hi)
        return np.concatenate(b[:2], 1), np.concatenate(c[:2], 1), n1 - n0, e.launch_count() - n1

    auto = both(engine.PATH_AUTO, True)
    tensor = both(engine.PATH_TF32X3, True)
    layers = both(engine.PATH_F64, False)
    direct = both(engine.PATH_F64, True)
    assert auto[2] == direct[2] < min(tensor[2], layers[2]) and auto[3] == direct[3] < min(tensor[3], layers[3])
    assert np.array_equal(auto[0], direct[0]) and np.array_equal(auto[1], direct[1])
    assert not np.array_equal(auto[0], tensor[0]) and not np.array_equal(auto[1], tensor[1])
    for got in (auto, tensor, layers):
        for i in range(2):
            scale = np.abs(direct[i]).max()
            assert np.all(np.abs(got[i] - direct[i]) <= (5e-4 if got is tensor else 1e-5) * scale)
    e.close()


@pytest.mark.parametrize("dims,rows,D,direct", [
    ([30, 40, 40, 5], 4, 63, True), ([30, 40, 40, 5], 4, 64, False),                   # 64 domains and more: TF32 intervals
    ([784] + [256] * 8 + [10], 9, 63, True), ([20, 256, 256, 10], 9, 1, True),
    ([20, 400, 400, 5], 4, 39, True), ([20, 400, 400, 5], 4, 40, False),               # 5e7 products of the widest layer
    ([20, 257, 40, 5], 4, 63, True), ([20, 64, 512, 10], 9, 10, True), ([20, 64, 512, 10], 9, 11, False),
])
def test_which_batches_go_direct(dims, rows, D, direct):
    from ny_b200 import B200Engine, engine

    net = W.make_mlp(dims, 3)
    x0 = np.full(dims[0], 0.4, np.float32)
    wide = np.full(net.n_pre, 1e30, np.float32)
    e = B200Engine(0)
    e.set_refine_tolerance(0.0)
    nid = e.register_network(net)
    args = (W.margin_spec(dims[-1], 0)[:rows], x0 - np.float32(0.02), x0 + np.float32(0.02), -wide, wide, np.zeros((D, 0), SPLIT_DTYPE), np.zeros(D, np.int32))
    got = {}
    for path in (engine.PATH_AUTO, engine.PATH_F64, engine.PATH_TF32X3):
        e.set_path(path)
        got[path] = e.bab_bound_batch(nid, *args)
    same = [p for p in (engine.PATH_F64, engine.PATH_TF32X3) if np.array_equal(got[engine.PATH_AUTO][0], got[p][0])]
    assert same == [engine.PATH_F64 if direct else engine.PATH_TF32X3]
    e.close()
