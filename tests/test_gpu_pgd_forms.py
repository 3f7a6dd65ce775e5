"""Forward values and gradients of points through window convolutions whose split adds the bias and the ReLU of the layer
in front, or drops masked rows, against binary64 contractions: channel counts on both sides of the one-thread-a-pixel
split, odd images, layers without a bias, identity branches that join in between, a fully connected layer next to them.

A layer's products err by at most 2.5e-6 of a row's sum of magnitudes (win_eps); random signs make that a few 1e-7 of a
vector's norm, and at most six layers add up: 2e-5 of the norm leaves a factor of ten."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

K3 = (3, 1, 1)
CASES = [
    ((3, 12, 10), [(16, 4, 2, 1), (32, 4, 2, 1)], {}, True),
    ((1, 9, 7), [(5, *K3), (16, *K3), (17, *K3)], {}, True),
    ((3, 11, 13), [(33, *K3), (64, 3, 2, 1), (8, *K3)], {}, True),
    ((3, 8, 8), [(16, *K3)] * 4, {}, False),
    ((3, 8, 8), [(16, *K3)] * 5, {2: 0, 4: 2}, True),
    ((2, 16, 16), [(24, *K3)], {}, True),
]


@pytest.mark.parametrize("case", range(len(CASES)))
@pytest.mark.parametrize("rows", [3, 130])
def test_values_and_gradients_agree_with_binary64(case, rows):
    from ny_b200 import B200Engine, Conv2d, Network, engine

    (c, h, w), convs, skips, bias = CASES[case]
    g = np.random.default_rng(300 + case)
    layers = []
    for co, k, s, p in convs:
        b = (g.standard_normal(co) * 0.3).astype(np.float32) if bias else None
        layers.append(Conv2d((g.standard_normal((co, c, k, k)) * np.sqrt(2.0 / (c * k * k))).astype(np.float32), b, (s, s), (p, p), (h, w)))
        c, h, w = co, layers[-1].oh, layers[-1].ow
    n = c * h * w
    net = Network(layers + [(g.standard_normal((7, n)) * np.sqrt(2.0 / n)).astype(np.float32)], [None] * len(layers) + [np.zeros(7, np.float32)], skips)
    x = (g.uniform(-1, 1, (rows, int(net.dims[0]))) * 10.0 ** g.uniform(-2, 2, (rows, 1))).astype(np.float32)
    spec = g.standard_normal((rows, 7)).astype(np.float32)
    masks = (g.random((rows, net.n_pre)) < 0.6).astype(np.float32)
    out = {}
    for path in (engine.PATH_TF32X3, engine.PATH_F64):
        eng = B200Engine(0)
        eng.set_path(path)
        nid = eng.register_network(net)
        _, values = eng.point_vjp_batched(nid, spec, x=x)
        best, points, _ = eng.pgd_attack(nid, spec[:2], x.min(0), x.max(0), x, 0, 0.1)
        out[path] = (np.asarray(values, np.float64), np.asarray(eng.point_vjp_batched(nid, spec, masks=masks), np.float64), best, points)
        eng.close()
    (v, gr, best, points), (fv, fg, fbest, fpoints) = out[engine.PATH_TF32X3], out[engine.PATH_F64]
    assert np.linalg.norm(gr - fg) <= 2e-5 * np.linalg.norm(fg)
    row = np.linalg.norm(gr - fg, axis=1) / np.maximum(np.linalg.norm(fg, axis=1), 1e-30)
    assert row.max() <= 1e-4
    assert np.linalg.norm(v - fv) <= 2e-5 * np.linalg.norm(fv)
    assert np.array_equal(points, fpoints) and np.allclose(best, fbest, rtol=1e-6)   # (the same binary64 evaluation)
