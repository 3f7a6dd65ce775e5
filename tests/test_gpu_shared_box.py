"""Re-evaluation of an optimised batch whose domains share one box: the first layer's charge weights exist once, in the first
domain's row, and the other rows hold what earlier calls or other programs left there.  A batch of huge boxes of their
own in front of it must change nothing."""
import numpy as np
import pytest

from ny_b200 import SPLIT_DTYPE
from ny_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("widths", [(32, 32, 32), (70, 41)])
@pytest.mark.parametrize("iterations", [1, 4])
def test_charges_of_a_shared_box_are_its_own(widths, iterations):
    from ny_b200 import B200Engine, engine

    net = W.make_mlp([24, *widths, 5], 3)
    g = np.random.default_rng(7)
    x = g.uniform(-1, 1, 24).astype(np.float32)
    lo, hi = x - np.float32(0.05), x + np.float32(0.05)
    spec, D = W.margin_spec(5, 1), 70
    none = (np.zeros((D, 0), SPLIT_DTYPE), np.zeros(D, np.int32))
    out = {}
    for before in (False, True):
        eng = B200Engine(0)
        eng.set_path(engine.PATH_TF32X3)
        nid = eng.register_network(net)
        pl, pu = eng.ibp_forward_gpu(nid, lo, hi)
        if before:
            big = np.full((D, 24), 1e12, np.float32)
            bl, bu = eng.ibp_forward_gpu(nid, -big[0], big[0])
            eng.bab_bound_batch(nid, spec, -big, big, bl[0], bu[0], *none, 1)
        eng.set_refine_tolerance(0.0)
        eng.batch_upload(nid, spec, lo, hi, pl[0], pu[0], *none, 1)
        eng.batch_optimize(iterations, 0.1, 0.0)
        fast = eng.batch_download()
        eng.set_refine_tolerance(1e-30)   # every domain is evaluated again in binary64
        eng.batch_upload(nid, spec, lo, hi, pl[0], pu[0], *none, 1)
        eng.batch_optimize(iterations, 0.1, 0.0)
        out[before] = eng.batch_download()
        assert eng.batch_refined() == D
        assert (out[before][0] >= fast[0]).all() and (out[before][0] > fast[0]).any()
        eng.close()
    for a, b in zip(out[False], out[True]):
        assert np.array_equal(a, b)
