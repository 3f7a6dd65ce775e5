"""Plain CROWN of many boxes, whose passes give a warp two groups of eight rows, against the same boxes a few at a time, whose
passes give it one: the arithmetic of a row is the same in both, up to the order of its binary64 sums, so bounds and
coefficients agree to a few fp32 steps.  Widths at the edges of the column tiles (two groups a warp from 41 on, and not where that
saves no wave of CTAs); rows that span boxes; a last group and a last warp that are not full."""
import numpy as np
import pytest

from ny_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_in,width,n_out,rows", [(3, 7, 2, 1), (5, 8, 5, 4), (2, 20, 3, 3), (12, 50, 5, 4), (70, 57, 5, 2), (9, 64, 4, 3), (5, 33, 7, 7), (4, 41, 3, 2), (6, 48, 5, 5)])
@pytest.mark.parametrize("per_sm", [20, 24])
def test_two_groups_a_warp_agree_with_one(n_in, width, n_out, rows, per_sm):
    from ny_b200 import B200Engine

    eng = B200Engine(0)
    D = -(-148 * per_sm * 8 // (2 * width)) + 3      # a little more than so many groups of eight rows an SM, not a whole number of warps
    net = W.make_mlp([n_in] + [width] * 3 + [n_out], 400 + width)
    g = np.random.default_rng(500 + width)
    mid = g.uniform(-0.5, 0.5, (D, n_in)).astype(np.float32)
    lo, hi = mid - np.float32(0.03), mid + np.float32(0.03)
    spec = g.standard_normal((rows, n_out)).astype(np.float32)
    nid = eng.register_network(net)
    many = eng.crown_bounds(nid, spec, lo, hi)
    many_a = eng.crown_input_coeffs(D, rows, n_in)
    few = [eng.crown_bounds(nid, spec, lo[i:i + 64], hi[i:i + 64]) for i in range(0, D, 64)]
    last_a = eng.crown_input_coeffs((D - 1) % 64 + 1, rows, n_in)
    for got, want in zip(many, (np.concatenate(x) for x in zip(*few))):
        assert np.isfinite(want).all()
        np.testing.assert_allclose(got, want, rtol=2e-6, atol=2e-6 * np.abs(want).max())
    for got, want in zip(many_a, last_a):
        np.testing.assert_allclose(got[-len(want):], want, rtol=2e-6, atol=1e-6 * np.abs(want).max())
    eng.close()
