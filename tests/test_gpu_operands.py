"""What a network's first calls build: one operand set per use, of what that use reads, and nothing a second time."""
import numpy as np
import pytest

from ny_b200 import SPLIT_DTYPE, Network
from ny_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _bound(eng, nid, net, D):
    g = np.random.Generator(np.random.PCG64(3))
    x0 = g.random(net.dims[0], dtype=np.float32)
    lo, hi = x0 - np.float32(0.01), x0 + np.float32(0.01)
    wide = np.full(net.n_pre, 1e30, np.float32)
    n0 = eng.launch_count()
    out = eng.bab_bound_batch(nid, W.margin_spec(net.dims[-1], 0), lo, hi, -wide, wide, np.zeros((D, 0), SPLIT_DTYPE), np.zeros(D, np.int32))
    return out, eng.launch_count() - n0


@pytest.mark.parametrize("dims", [[60, 64, 128, 32, 10], [30, 256, 256, 256, 256, 5], [10, 8, 3]])
def test_a_plain_bound_builds_what_it_reads(dims):
    from ny_b200 import B200Engine

    eng = B200Engine(0)
    eng.set_refine_tolerance(0.0)
    net, L = W.make_mlp(dims, 7), len(dims) - 1
    nid = eng.register_network(net)
    first, n1 = _bound(eng, nid, net, 200)
    again, n2 = _bound(eng, nid, net, 200)
    # interval operands and the chain's of L - 1 layers, and the first layer's for the contraction behind the chain
    assert n1 - n2 == 2 * (L - 1) + 1
    # the per-layer form reads the other layers' own operands; the first layer's is there
    eng.set_fusion(False)
    _, n3 = _bound(eng, nid, net, 200)
    _, n4 = _bound(eng, nid, net, 200)
    assert n3 - n4 == L - 1
    eng.set_fusion(True)
    third, n5 = _bound(eng, nid, net, 200)
    assert n5 == n2
    for a, b, c in zip(first, again, third):
        assert np.array_equal(a, b) and np.array_equal(a, c)
    eng.close()


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("where", ["first", "last"])
def test_weights_that_are_not_finite_are_refused(value, where):
    from ny_b200 import B200Engine, EngineError

    eng = B200Engine(0)
    net = W.make_mlp([70, 300, 257, 3], 5)
    w = [x.copy() for x in net.weights]
    if where == "first":
        w[0][0, 0] = value
    else:
        w[-1][-1, -1] = value
    with pytest.raises(EngineError):
        eng.register_network(Network(w, net.biases))
    nid = eng.register_network(net)
    out, _ = _bound(eng, nid, net, 70)
    assert np.all(out[0] <= out[1])
    eng.close()
