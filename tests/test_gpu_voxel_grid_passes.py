"""The voxel grid's radix passes on both sides of the 2^16-cell line (the last
two passes are skipped below it): leaf order, counts and centroids equal the
oracle's bit for bit."""
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
