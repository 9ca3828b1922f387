"""The SO(3) angle transforms (alpha in place, packed gamma pairs with the
argmax) at lengths where they can go wrong: the shortest, prime factors in
both halves of the runtime plans, compile-time lengths and their neighbours,
a last tile with one pair of betas, zero padding.  Random signals against the
FP64 oracle at the repository's relative L2 of 1e-5, and the reported bin is
the first of the volume's largest values."""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_parity import REL_L2

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nat():
    from phaser_b200 import native
    native.load()
    return native


@pytest.mark.parametrize("bw,pad", [(2, 0), (3, 1), (8, 3), (11, 0), (13, 4), (16, 1), (17, 0), (32, 0), (32, 2), (19, 4),
                                    (33, 0), (37, 0), (50, 0)])
def test_rotation_volume_vs_oracle(nat, bw, pad):
    rng = np.random.default_rng(100 * bw + pad)
    f, g = rng.standard_normal((2, 1, 4 * bw * bw))
    c = nat.Context(spherical_bandwidth=bw, spherical_zero_padding=pad, spatial_n_voxels=4,
                    spherical_fusion=nat.PHGPU_FUSION_NONE, flags=nat.PHGPU_FLAG_KEEP_VOLUMES)
    c.sph_correlate(list(f), list(g))
    b, peak, vol = c.sph_result(volume=True)
    ref = O.spherical_correlation(f, g, bw, bw_out=bw + pad)
    ref = ref[0] if isinstance(ref, tuple) else ref
    assert np.linalg.norm(vol - ref.reshape(-1)) <= REL_L2 * np.linalg.norm(ref)
    assert b == int(np.argmax(vol)) and np.float32(peak) == np.float32(vol[b])


def test_equal_values_take_the_first_bin(nat):
    c = nat.Context(spherical_bandwidth=10, spatial_n_voxels=4, spherical_fusion=nat.PHGPU_FUSION_NONE,
                    flags=nat.PHGPU_FLAG_KEEP_VOLUMES)
    z = np.zeros((1, 400))
    c.sph_correlate(list(z), list(z))
    b, peak, vol = c.sph_result(volume=True)
    assert b == 0 and peak == 0.0 and not vol.any()


@pytest.mark.parametrize("bw", [8, 32, 37])
def test_undefined_volume_has_its_peak_at_the_first_bin(nat, bw):
    """One NaN sample makes every bin NaN: the reference's max_element then stays at the first one."""
    rng = np.random.default_rng(bw)
    f, g = rng.standard_normal((2, 1, 4 * bw * bw))
    f[0, 5] = np.nan
    c = nat.Context(spherical_bandwidth=bw, spatial_n_voxels=4, spherical_fusion=nat.PHGPU_FUSION_NONE,
                    flags=nat.PHGPU_FLAG_KEEP_VOLUMES)
    c.sph_correlate(list(f), list(g))
    b, peak, vol = c.sph_result(volume=True)
    assert np.isnan(vol).all()
    assert b == O.argmax(vol) == 0 and np.isnan(peak)


@pytest.mark.parametrize("pad", [871, 873, 878])
def test_longest_transforms(nat, pad):
    """Lengths 1746 = 2 9 97, 1750 and 1760, the longest whose tiles fit (22 GB of spectra).  The correlation of two
    signals of bandwidth 2 is a trigonometric polynomial of degree 1 per angle, its square z^2 of degree 2 with
    |d^2 z^2| <= 4 max z^2: grids of spacing h <= 2 pi / 804 miss its maximum by at most 3 * 4 / 2 (h / 2)^2 = 9.2e-5
    of it, and the transforms add 1e-5."""
    rng = np.random.default_rng(9)
    f, g = rng.standard_normal((2, 1, 16))
    peaks = []
    for p in (400, pad):
        c = nat.Context(spherical_bandwidth=2, spherical_zero_padding=p, spatial_n_voxels=4,
                        spherical_fusion=nat.PHGPU_FUSION_NONE)
        c.sph_correlate(list(f), list(g))
        peaks.append(c.sph_result()[1])
        c.close()
    assert abs(peaks[1] - peaks[0]) <= 1.2e-4 * peaks[0]
