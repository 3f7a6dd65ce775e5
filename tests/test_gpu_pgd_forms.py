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


@pytest.mark.parametrize("form", ["plain", "outside", "wide", "dead", "resnet"])
def test_a_step_follows_the_gradient(form):
    """One step of the attack on the tensor path against the same step in plain binary64: the point it keeps is the start, or the
    start moved against the gradient of its worst row and cut to the box, wherever the gradient's component is more than 1e-4
    of its largest (products err by 2e-5, above) and the two points' margins differ.  Points in the box and outside
    it; points of very different sizes, down to 1e-14, in a box of 1e6, on layers without bias; a channel that a bias of -1e30
    switches off; an identity branch."""
    import torch
    import torch.nn.functional as F

    from ny_b200 import B200Engine, Conv2d, Network, engine

    g = np.random.default_rng(17)
    c, h, w = 3, 12, 10
    convs, skips = ([(8, *K3), (8, *K3), (8, *K3), (16, 4, 2, 1)], {2: 0}) if form == "resnet" else ([(8, 4, 2, 1), (16, *K3), (24, *K3)], {})
    layers = []
    for i, (co, k, s, p) in enumerate(convs):
        b = (g.standard_normal(co) * 0.1).astype(np.float32)
        if form == "dead" and i < 2:
            b[3] = -1e30
        layers.append(Conv2d((g.standard_normal((co, c, k, k)) * np.sqrt(2.0 / (c * k * k))).astype(np.float32), None if form == "wide" else b, (s, s), (p, p), (h, w)))
        c, h, w = co, layers[-1].oh, layers[-1].ow
    n = c * h * w
    net = Network(layers + [(g.standard_normal((7, n)) * np.sqrt(2.0 / n)).astype(np.float32)], [None] * len(layers) + [np.zeros(7, np.float32)], skips)
    n0, rows, step = int(net.dims[0]), 130, np.float32(1e-3)
    x = g.uniform(-1, 1, (rows, n0))
    lo, hi = np.full(n0, -1.0, np.float32), np.full(n0, 1.0, np.float32)
    if form == "outside":
        x *= 1.1
    if form == "wide":
        x, lo, hi = x * 10.0 ** g.uniform(-14, 2, (rows, 1)), lo * np.float32(1e6), hi * np.float32(1e6)
    x = x.astype(np.float32)
    spec = g.standard_normal((5, 7)).astype(np.float32)
    eng = B200Engine(0)
    eng.set_path(engine.PATH_TF32X3)
    _, points, _ = eng.pgd_attack(eng.register_network(net), spec, lo, hi, x, 1, step)
    eng.close()

    t = lambda a: torch.from_numpy(np.asarray(a)).double()

    def margin(z):
        post, z = [], t(z) if isinstance(z, np.ndarray) else z
        for k, l in enumerate(layers):
            z = F.conv2d(z.reshape(-1, l.ic, l.ih, l.iw), t(l.weight), None if l.bias is None else t(l.bias), (l.sh, l.sw), (l.ph, l.pw)).flatten(1)
            z = torch.relu(z + post[skips[k]] if k in skips else z)
            post.append(z)
        return (z @ t(net.weights[-1]).T @ t(spec).T).min(1).values

    start = t(x).requires_grad_()
    m0 = margin(start)
    m0.sum().backward()
    grad, m0 = start.grad.numpy(), m0.detach().numpy()
    moved = np.clip(x - np.float32(10) * step * np.where(grad < 0, -1, 1).astype(np.float32), lo, hi)   # (the first moment's correction: 1 / 0.1)
    m1 = margin(moved).numpy()
    clear = np.abs(m1 - m0) > 1e-3 * np.maximum(np.abs(m0), np.abs(m1))
    better = clear & (m1 < m0)
    assert better.sum() > rows // 3
    sure = np.abs(grad) > 1e-4 * np.abs(grad).max(axis=1, keepdims=True)
    assert sure.mean() > 0.5
    assert np.array_equal(points[clear & ~better], x[clear & ~better])
    assert np.allclose(points[better][sure[better]], moved[better][sure[better]], rtol=1e-6, atol=1e-5 * step)   # (the step's own rounding)


# more than 64 channels: a thread of the split takes several groups of four pairs, the last one not whole
WIDE = [((2, 10, 9), [(66, *K3), (96, *K3), (130, *K3), (4, *K3)], {}, True), ((3, 8, 8), [(48, *K3), (20, *K3), (100, *K3), (3, *K3)], {}, False)]
CASES.extend(WIDE)


@pytest.mark.parametrize("case", range(len(CASES) - len(WIDE), len(CASES)))
@pytest.mark.parametrize("rows", [3, 130])
def test_values_and_gradients_of_many_channels_agree_with_binary64(case, rows):
    test_values_and_gradients_agree_with_binary64(case, rows)
