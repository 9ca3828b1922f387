"""The translation passes over voxelised clouds (row sums, x, z and inverse
passes) against the FP64 oracle at lengths where they can go wrong: the
shortest transforms, odd and prime lengths, prime factors at both ends of the
generic stage, the compile-time lengths and their neighbours, tiles with a
remainder; with one row and one slab filled, the rest nearly empty; two, three
and four channels; a cloud outside the grid.  The bar is the repository's
relative L2 of 1e-5 for correlation volumes."""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_parity import REL_L2, tie_masked_rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nat():
    from phaser_b200 import native
    native.load()
    return native


def cloud(rng, N, half, n=400):
    """Points at random, along one whole row (every y) and over one z slab."""
    edges = np.linspace(-half, half, N, dtype=np.float32)
    step = edges[1] - edges[0] if N > 1 else np.float32(half)
    p = rng.uniform(-half, half, (n, 3)).astype(np.float32)
    k = np.arange(N)
    row = np.stack([np.full(N, edges[N // 3]), edges[k], np.full(N, edges[N // 2])], 1) + 0.4 * step
    m = min(N * N // 2, 3000)
    slab = np.stack([edges[rng.integers(0, N, m)], edges[rng.integers(0, N, m)], np.full(m, edges[N // 4])], 1) + 0.4 * step
    xyz = np.concatenate([p, row, slab]).astype(np.float32)
    xyz = np.clip(xyz, -half, half)
    w = rng.uniform(0.1, 1.0, (len(xyz), 3)).astype(np.float32)
    return np.concatenate([xyz, w[:, :1]], 1), w[:, 1].copy(), w[:, 2].copy()


@pytest.mark.parametrize("N,channels", [(2, 3), (3, 2), (4, 4), (7, 3), (8, 2), (11, 3), (13, 4), (22, 3), (31, 2), (35, 3),
                                        (64, 4), (66, 3), (67, 3), (97, 2), (100, 3), (121, 3), (127, 2), (128, 2),
                                        (130, 3), (200, 2)])
def test_voxelised_translation_vs_oracle(nat, N, channels):
    rng = np.random.default_rng(1000 * N + channels)
    half = 10
    clouds = [cloud(rng, N, half) for _ in range(2)]
    c = nat.Context(spherical_bandwidth=2, spatial_n_voxels=N, spatial_discretize_lower=-half,
                    spatial_discretize_upper=half, flags=nat.PHGPU_FLAG_KEEP_VOLUMES)
    grids = []
    for side, (xyzi, refl, amb) in enumerate(clouds):
        args = (xyzi, refl if channels > 2 else None, amb if channels > 3 else None)
        c.voxelize(*args, side=side)
        grids.append(O.discretize(*args, N, -half, half).reshape(4, -1))
    c.spatial_correlate_voxelized()
    vox, peak, vol = c.spatial_result(volume=True)
    ref = O.spatial_correlation(grids[0], grids[1], N, laplace=True)
    err, _ = tie_masked_rel_l2(vol, ref, grids[0], grids[1], N)
    assert err <= REL_L2
    # the same grids again (they are kept), then a far cloud: everything zero, the first voxel wins
    c.spatial_correlate_voxelized()
    again = c.spatial_result(volume=True)
    assert again[0] == vox and np.array_equal(again[2], vol)
    far = clouds[1][0].copy()
    far[:, 2] += 1000.0 * half
    lin = O.voxel_index(far, N, -half, half)
    c.voxelize(far, clouds[1][1] if channels > 2 else None, clouds[1][2] if channels > 3 else None, side=1)
    c.spatial_correlate_voxelized()
    vox, peak, vol = c.spatial_result(volume=True)
    if (lin == 0xffffffff).all():
        assert vox == 0 and peak == 0.0 and not vol.any()


@pytest.mark.parametrize("N", [1, 2, 9, 64, 101, 169, 200])
def test_host_grids_translation_vs_oracle(nat, N):
    rng = np.random.default_rng(N)
    f, g = rng.standard_normal((2, 2, N ** 3))
    c = nat.Context(spherical_bandwidth=2, spatial_n_voxels=N, flags=nat.PHGPU_FLAG_KEEP_VOLUMES)
    c.spatial_correlate(list(f), list(g))
    _, _, vol = c.spatial_result(volume=True)
    ref = O.spatial_correlation(f, g, N, laplace=True)
    err, _ = tie_masked_rel_l2(vol, ref, f, g, N)
    assert err <= REL_L2


def test_fast_division_is_exact():
    """fast_div(x, ceil(2^32 / d)) == x // d over the passes' ranges (x d < 2^32)."""
    x = np.arange(1 << 18, dtype=np.uint64)
    for d in [*range(2, 130), 201, 255, 256, 257, 511, 512, 513, 1000, 1023, 1024]:
        mul = np.uint64(0xffffffff // d + 1)
        assert np.array_equal((x * mul) >> np.uint64(32), x // np.uint64(d)), d


def test_voxels_of_a_smaller_cloud_are_cleared(nat):
    """A context whose buffers grow between voxelisations, and one that goes from
    the voxelisation calls to whole registrations and back, must not keep voxels
    of an earlier cloud."""
    rng = np.random.default_rng(5)
    small, large = cloud(rng, 40, 10, n=5), cloud(rng, 40, 10, n=3000)
    kw = dict(spherical_bandwidth=8, spatial_n_voxels=40, spatial_discretize_lower=-10, spatial_discretize_upper=10,
              flags=nat.PHGPU_FLAG_KEEP_VOLUMES)

    def volume(c, a, b):
        c.voxelize(*a, side=0)
        c.voxelize(*b, side=1)
        c.spatial_correlate_voxelized()
        return c.spatial_result(volume=True)[2]

    fresh = volume(nat.Context(**kw), small, large)
    c = nat.Context(max_points=8, **kw)
    for a, b in ((small, small), (large, small), (small, large)):
        vol = volume(c, a, b)
    np.testing.assert_allclose(vol, fresh, rtol=0, atol=1e-6 * np.abs(fresh).max())
    c.register_pair(large[:2], small[:2])
    vol = volume(c, small, large)
    np.testing.assert_allclose(vol, fresh, rtol=0, atol=1e-6 * np.abs(fresh).max())


@pytest.mark.parametrize("first", [1, 511, 512, 513, 5000])
def test_voxels_are_cleared_by_points_and_by_rows(nat, first):
    """The next voxelisation clears the last one's voxels point by point below an eighth of the 16^3 voxels, its
    rows whole from there on; points outside the grid and a second cloud of another size in between."""
    rng = np.random.default_rng(first)
    N, half = 16, 10

    def points(n):
        xyzi = rng.uniform(-1.1 * half, 1.1 * half, (n, 4)).astype(np.float32)
        return xyzi, rng.uniform(0.1, 1.0, n).astype(np.float32)

    kw = dict(spherical_bandwidth=2, spatial_n_voxels=N, spatial_discretize_lower=-half, spatial_discretize_upper=half,
              flags=nat.PHGPU_FLAG_KEEP_VOLUMES)
    small, other = points(40), points(60)

    def volume(c):
        c.voxelize(*small, side=0)
        c.voxelize(*other, side=1)
        c.spatial_correlate_voxelized()
        return c.spatial_result(volume=True)[2]

    fresh = volume(nat.Context(**kw))
    c = nat.Context(max_points=6000, **kw)
    for n in (first, 600, first):
        for side in range(2):
            c.voxelize(*points(n), side=side)
    np.testing.assert_allclose(volume(c), fresh, rtol=0, atol=1e-6 * np.abs(fresh).max())


@pytest.mark.parametrize("N", [128, 200, 201, 320])
def test_full_rows_round_no_more_than_an_fft(nat, N):
    """Rows with a point in every voxel (slabs of them; one point a voxel, so the means are the values): the
    correlation of the voxelised clouds is no further from FP64 than that of the same grids handed in, whose rows
    take an FFT.  Bar: in a model of both sums in FP32 the rows' error is at most 1.05 times the FFT's at any length
    and number of voxels, so the volume's is at most 1.05 times plus the spread between draws (well under a tenth
    for N^3 values); one running sum over the row gives 1.3 (N = 128) to 1.9 (N = 320) times."""
    rng = np.random.default_rng(N)
    half = 10
    edges = np.linspace(-half, half, N, dtype=np.float32)
    at = np.clip(edges + 0.4 * (edges[1] - edges[0]), -half, half)
    c = nat.Context(spherical_bandwidth=2, spatial_n_voxels=N, spatial_discretize_lower=-half,
                    spatial_discretize_upper=half, spatial_fusion=nat.PHGPU_FUSION_NONE, flags=nat.PHGPU_FLAG_KEEP_VOLUMES,
                    max_points=3 * N * N)
    grids = []
    for side in range(2):
        z = rng.choice(N, 3, replace=False)
        xyz = np.stack(np.meshgrid(at, at, at[z], indexing="ij"), -1).reshape(-1, 3)
        xyzi = np.concatenate([xyz, rng.standard_normal((len(xyz), 1))], 1).astype(np.float32)
        lin = O.voxel_index(xyzi, N, -half, half)
        assert len(np.unique(lin)) == len(lin) and lin.max() < N ** 3
        g = np.zeros(N ** 3)
        g[lin] = xyzi[:, 3]
        grids.append(g)
        c.voxelize(xyzi, side=side)
    ax = (0, 1, 2)
    F, G = (np.fft.rfftn(g.reshape(N, N, N), axes=ax) for g in grids)
    ref = np.fft.irfftn(F * np.conj(G), (N, N, N), axes=ax).reshape(-1) * N ** 3

    def error(vol):
        return np.linalg.norm(vol - ref) / np.linalg.norm(ref)

    c.spatial_correlate_voxelized()
    rows = error(c.spatial_result(volume=True)[2])
    c.spatial_correlate([grids[0]], [grids[1]])
    fft = error(c.spatial_result(volume=True)[2])
    print(f"N {N}: sums {rows:.3g}, FFT {fft:.3g}")
    assert rows <= 1.2 * fft <= REL_L2


@pytest.mark.parametrize("N,channels", [(28, 1), (30, 2), (48, 3), (50, 4), (64, 3), (98, 2), (100, 3), (108, 4), (200, 1), (256, 1),
                                        (320, 1)])
def test_rows_around_the_density_limit(nat, N, channels):
    """Rows of 16 voxels (one sum), of 17 and of as many as are still summed in parts, of one more (transformed), full
    ones and ones with a gap at either end, in one slab: the correlation against FP64 at the bar for volumes, twice from kept grids, and again after a registration
    that clears them on the way."""
    rng = np.random.default_rng(N)
    half = 10
    edges = np.linspace(-half, half, N, dtype=np.float32)
    at = np.clip(edges + 0.4 * (edges[1] - edges[0]), -half, half)
    plain = channels == 1
    kw = dict(spherical_bandwidth=8, spatial_n_voxels=N, spatial_discretize_lower=-half, spatial_discretize_upper=half,
              spatial_fusion=nat.PHGPU_FUSION_NONE if plain else nat.PHGPU_FUSION_LAPLACE, flags=nat.PHGPU_FLAG_KEEP_VOLUMES)
    c = nat.Context(**kw)
    clouds, grids = [], []
    for side in range(2):
        cols = [np.arange(16), rng.choice(N, 16, replace=False), rng.choice(N, 17, replace=False), np.arange(N - 17, N),
                np.arange(N), np.arange(1, N), np.arange(N - 1), np.array([N // 2])]
        limit = min(max(N // 5, 16), 40)
        cols[4:4] = [rng.choice(N, min(limit + k, N), replace=False) for k in (0, 1)]
        xyz = np.concatenate([np.stack([np.full(len(y), at[(2 * i + side) % N]), at[y], np.full(len(y), at[N // 3 + side])], 1)
                              for i, y in enumerate(cols)])
        xyzi = np.concatenate([xyz, rng.uniform(0.1, 1.0, (len(xyz), 1))], 1).astype(np.float32)
        refl, amb = rng.uniform(0.1, 1.0, (2, len(xyzi))).astype(np.float32)
        clouds.append((xyzi, refl if channels > 2 else None, amb if channels > 3 else None))
        grids.append(O.discretize(*clouds[-1], N, -half, half).reshape(4, -1)[:1 if plain else 4])
        c.voxelize(*clouds[-1], side=side)
    if plain:
        ax = (0, 1, 2)
        F, G = (np.fft.rfftn(g.reshape(N, N, N), axes=ax) for g in grids)
        ref = np.fft.irfftn(F * np.conj(G), (N, N, N), axes=ax).reshape(-1) * N ** 3
    else:
        ref = O.spatial_correlation(grids[0], grids[1], N, laplace=True)

    def check():
        c.spatial_correlate_voxelized()
        vol = c.spatial_result(volume=True)[2]
        err = np.linalg.norm(vol - ref) / np.linalg.norm(ref) if plain else tie_masked_rel_l2(vol, ref, grids[0], grids[1], N)[0]
        assert err <= REL_L2
        return vol

    vol = check()
    assert np.array_equal(check(), vol)
    c.register_pair(clouds[0][:2], clouds[1][:2])
    for side in range(2):
        c.voxelize(*clouds[side], side=side)
    check()
