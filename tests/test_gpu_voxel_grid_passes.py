"""The voxel grid's radix passes around the cell counts where their number
changes, leaf lengths around the centroid's batches and clouds around the scan
kernels' limits: leaf order, counts and centroids equal the oracle's bit for bit."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(1, 1, 1), (16, 16, 1), (256, 256, 1), (256, 257, 1), (65536, 1, 1), (65537, 1, 1),
                                      (4096, 64, 3)])
def test_cell_counts_around_the_pass_limit(nx, ny, nz):
    from phaser_b200 import native
    rng = np.random.default_rng(nx + ny)
    n = 7000
    ijk = np.stack([rng.integers(0, d, n) for d in (nx, ny, nz)], 1)
    ijk[0] = 0
    ijk[1] = (nx - 1, ny - 1, nz - 1)
    x = np.concatenate([(ijk + rng.uniform(0.2, 0.8, (n, 3))), rng.uniform(0, 1, (n, 1))], 1).astype(np.float32)
    vg = native.VoxelGrid(8192)
    out, refl, _ = vg.filter(x, (1.0, 1.0, 1.0), 0, x[:, 3].copy())
    want, wrefl, _ = O.voxel_grid(x, (1.0, 1.0, 1.0), 0, x[:, 3].copy())
    assert np.array_equal(out, want) and np.array_equal(refl, wrefl)


def _both(x, leaf, min_points, vg):
    from phaser_b200 import native
    vg = vg or native.VoxelGrid(len(x))
    amb = (x[:, 0] * 3).copy()
    out, refl, ambient = vg.filter(x, (leaf,) * 3, min_points, x[:, 3].copy(), amb)
    want, wrefl, wamb = O.voxel_grid(x, (leaf,) * 3, min_points, x[:, 3].copy(), amb)
    for a, b in ((out, want), (refl, wrefl), (ambient, wamb)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("counts", [(1, 2, 3, 4, 5, 7, 8), (255, 256, 257, 258, 259), (511, 512, 513, 3000), (2047,), (2049, 31, 33)])
@pytest.mark.parametrize("min_points", [0, 5])
def test_leaf_lengths_around_the_batches(counts, min_points):
    """Leaves that end at, before and behind a group of four points, a batch and
    a tile, with non-finite points in between: the in-order float sums of every
    component are those of one thread."""
    rng = np.random.default_rng(sum(counts))
    ijk = np.repeat(np.arange(len(counts)), counts)
    x = rng.uniform(0.1, 0.9, (len(ijk), 4)).astype(np.float32)
    x[:, 0] += ijk
    x = x[rng.permutation(len(x))]
    bad = rng.uniform(0, 1, (len(x) // 3, 4)).astype(np.float32)
    bad[:, rng.integers(0, 3)] = np.nan
    x = np.insert(x, rng.integers(0, len(x) + 1, len(bad)), bad, axis=0)
    _both(x, 1.0, min_points, None)


@pytest.mark.parametrize("span", [(2, 2, 2), (200, 300, 270), (260, 300, 300), (2000, 1000, 1000)])
def test_one_to_four_passes(span):
    """Leaf indices of 3, 24, 25 and 31 bits: an odd and an even number of radix passes."""
    rng = np.random.default_rng(span[0])
    x = np.concatenate([rng.uniform(0, 1, (5000, 3)) * np.array(span), rng.uniform(0, 1, (5000, 1))], 1).astype(np.float32)
    _both(x, 1.0, 0, None)


def test_no_finite_point():
    _both(np.full((3000, 4), np.nan, np.float32), 0.5, 0, None)


@pytest.mark.parametrize("n", [192 * 1024, 192 * 1024 + 1, 4096 * 1024, 4096 * 1024 + 5])
def test_tiles_around_the_scan_kernels(n):
    """Blocks add up the tiles' counts themselves up to 192 tiles of 1024 items in the radix passes and 4096 in
    the compactions; scan kernels do beyond that."""
    rng = np.random.default_rng(1)
    x = (rng.integers(0, 400, (n, 4)) / np.float32(4)).astype(np.float32)
    _both(x, 4.0, 2, None)


@pytest.mark.parametrize("seed", [0, 1, 2])
def test_long_leaves_in_consecutive_batches(seed):
    """More leaves than the centroid's grid takes at a time (8 warps of 2368 blocks): blocks that have long leaves in
    one batch and, in other warps' places, in the next, with short ones between them."""
    rng = np.random.default_rng(seed)
    blocks, batch = 2368, 8 * 2368
    counts = rng.integers(1, 5, 2 * batch + 5000)
    lengths = np.array([129, 130, 895, 896, 897, 1793, 3000])
    for b in rng.choice(blocks, 60, replace=False):
        for turn in range(3):
            w = rng.choice(8, rng.integers(1, 4), replace=False)
            leaf = turn * batch + b + w * blocks
            leaf = leaf[leaf < len(counts)]
            counts[leaf] = rng.choice(lengths, len(leaf))
    ijk = rng.permutation(np.repeat(np.arange(len(counts)), counts))
    x = rng.uniform(0.1, 0.9, (len(ijk), 4)).astype(np.float32)
    x[:, 0] += ijk
    from phaser_b200 import native
    vg = native.VoxelGrid(len(x))
    for _ in range(3):
        _both(x, 1.0, 0, vg)
