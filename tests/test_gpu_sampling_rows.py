"""Row sweep of the S^2 sampling where its window logic can go wrong: rows
that hold only stray points beside dense ones, whole circles near the poles,
columns that wrap, empty and tiny clouds; and both clouds of a registration
sampled in one set of launches against each sampled alone.  Nearest-point
indices must equal the brute-force search over the same projected points."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nat():
    from phaser_b200 import native
    native.load()
    return native


def polar(theta, phi, r):
    return np.stack([r * np.sin(theta) * np.cos(phi), r * np.sin(theta) * np.sin(phi), r * np.cos(theta)], 1)


def clouds(bw):
    rng = np.random.default_rng(bw)
    w = np.pi / (2 * bw)
    out = {}
    # a dense band whose outermost ring lies on a row edge, a few stray points in the next row
    th = np.concatenate([np.full(60 * bw, 0.5 * np.pi - 0.4 // w * w), rng.uniform(0.5 * np.pi - 0.3, 0.5 * np.pi + 0.4, 200 * bw)])
    stray = 0.5 * np.pi - 0.4 // w * w - 0.5 * w
    th = np.concatenate([th, np.full(3, stray)])
    out["stray"] = polar(th, rng.uniform(0, 2 * np.pi, len(th)), rng.uniform(1, 9, len(th)))
    out["poles"] = polar(np.concatenate([rng.uniform(0, 1.5 * w, 300), np.pi - rng.uniform(0, 0.5 * w, 300)]),
                         rng.uniform(0, 2 * np.pi, 600), np.full(600, 2.0))
    out["wrap"] = polar(rng.uniform(0.2, 3.0, 500), rng.normal(0.0, 0.5 * w, 500), rng.uniform(1, 3, 500))
    out["one"] = np.array([[1.0, 2.0, 0.5]])
    out["sphere"] = rng.standard_normal((2000, 3))
    return {k: np.concatenate([v, rng.uniform(0, 1, (len(v), 1))], 1).astype(np.float32) for k, v in out.items()}


@pytest.mark.parametrize("bw", [2, 3, 16, 33, 64])
def test_nearest_points_of_awkward_rows(nat, bw):
    c = nat.Context(spherical_bandwidth=bw, spatial_n_voxels=4)
    grid = O.dh_grid(bw)
    for name, xyzi in clouds(bw).items():
        pts, _ = O.project(xyzi)
        idx, _ = O.nn(grid, pts)
        c.sample_s2(xyzi, side=0)
        _, got = c.samples(0)
        bad = got != idx
        if bad.any():  # the projections of the two sides may differ in the last bit: equal distances up to it
            a = ((grid[bad] - pts[got[bad]]).astype(np.float64) ** 2).sum(1)
            b = ((grid[bad] - pts[idx[bad]]).astype(np.float64) ** 2).sum(1)
            assert np.all(np.sqrt(a) <= np.sqrt(b) + 3e-7), name
            assert bad.mean() < 0.01, name


def test_two_clouds_in_one_launch(nat):
    cl = clouds(16)
    names = list(cl)
    c = nat.Context(spherical_bandwidth=16, spatial_n_voxels=8, spatial_discretize_lower=-10, spatial_discretize_upper=10)
    for a, b in zip(names, names[1:] + names[:1]):
        alone = []
        for k in (a, b):
            c.sample_s2(cl[k], side=0)
            alone.append(c.samples(0))
        c.register_pair((cl[a], None), (cl[b], None))
        for side in (0, 1):
            v, i = c.samples(side)
            assert np.array_equal(i, alone[side][1]) and np.array_equal(v, alone[side][0]), (a, b, side)


def test_longitude_bound_is_an_upper_bound():
    """2 asin x <= 2 x (1 + 0.5708 x^2) (1 + 1e-5) on [0, 1], evaluated as the kernel does."""
    x2 = np.linspace(0, 1, 200001)
    x = np.sqrt(x2.astype(np.float32)).astype(np.float32)
    bound = 2 * x * (np.float32(0.5708) * x2.astype(np.float32) + 1) * np.float32(1 + 1e-5)
    assert np.all(bound.astype(np.float64) >= 2 * np.arcsin(np.sqrt(x2)))


def test_arc_sine_bound_is_an_upper_bound():
    """pi - 2 sqrt(1 - x) P(x) + 2e-4 >= 2 asin of the exact root on [0, 1], with x evaluated as the kernel does (float32,
    a root short of 2^-22)."""
    x2 = np.concatenate([np.linspace(0, 1, 200001), 1 - np.logspace(-12, -1, 20001)])
    f = np.float32
    x = np.sqrt(x2.astype(f) * f(1 + 1e-5)) * f(1 - 2.0 ** -22)
    p = ((f(-0.0187293) * x + f(0.0742610)) * x + f(-0.2121144)) * x + f(1.5707288)
    bound = f(3.14159265) - f(2) * (np.sqrt(np.maximum(f(1) - x, f(0))) * p) + f(2e-4)
    slack = bound.astype(np.float64) - 2 * np.arcsin(np.sqrt(x2))
    assert slack.min() >= 0 and slack.max() < 0.01


@pytest.mark.parametrize("bw", [5, 16, 40, 64])
@pytest.mark.parametrize("opening,n", [(60.0, 20000), (5.0, 20000), (0.3, 20000), (60.0, 300), (360.0, 40)])
def test_narrow_openings(nat, bw, opening, n):
    """Clouds seen through a narrow opening (windows of many and of few points, wide and far from the points)."""
    rng = np.random.default_rng(bw + n)
    a = 0.5 * np.deg2rad(opening)
    if opening < 360:
        v = np.stack([np.ones(n), np.tan(rng.uniform(-a, a, n)), np.tan(rng.uniform(-a, a, n))], 1) * rng.uniform(2, 9, (n, 1))
        v = v @ np.linalg.qr(rng.standard_normal((3, 3)))[0]
    else:
        v = rng.standard_normal((n, 3))
    xyzi = np.concatenate([v, rng.uniform(0, 1, (n, 1))], 1).astype(np.float32)
    c = nat.Context(spherical_bandwidth=bw, spatial_n_voxels=4)
    grid = O.dh_grid(bw)
    pts, _ = O.project(xyzi)
    idx, _ = O.nn(grid, pts)
    c.sample_s2(xyzi, side=0)
    _, got = c.samples(0)
    bad = got != idx
    if bad.any():  # as above: equal distances up to the projections' last bit
        a = ((grid[bad] - pts[got[bad]]).astype(np.float64) ** 2).sum(1)
        b = ((grid[bad] - pts[idx[bad]]).astype(np.float64) ** 2).sum(1)
        assert np.all(np.sqrt(a) <= np.sqrt(b) + 3e-7)
        assert bad.mean() < 0.01
