"""The Wigner synthesis at the lengths where its rule changes the betas per
thread (2, 4, 5 or 7), with an odd and an even number of degrees, a last thread
with fewer betas, and several rounds of betas a thread.  Random signals against
the FP64 oracle at the repository's relative L2 of 1e-5."""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_parity import REL_L2

pytestmark = pytest.mark.gpu


def _volumes(bw, pad, ref_pad):
    from phaser_b200 import native as nat
    rng = np.random.default_rng(100 * bw + pad)
    f, g = rng.standard_normal((2, 1, 4 * bw * bw))
    c = nat.Context(spherical_bandwidth=bw, spherical_zero_padding=pad, spatial_n_voxels=4,
                    spherical_fusion=nat.PHGPU_FUSION_NONE, flags=nat.PHGPU_FLAG_KEEP_VOLUMES)
    c.sph_correlate(list(f), list(g))
    vol = c.sph_result(volume=True)[2]
    ref = O.spherical_correlation(f, g, bw, bw_out=bw + ref_pad)
    ref = ref[0] if isinstance(ref, tuple) else ref
    return np.asarray(vol).reshape((2 * (bw + pad),) * 3), np.asarray(ref).reshape((2 * (bw + ref_pad),) * 3)


# n = 64 | 66, 100 | 120, 150 | 200 | 256 | 300, 320 | 392, 512
@pytest.mark.parametrize("bw,pad", [(31, 1), (33, 0), (40, 10), (17, 43), (75, 0), (41, 59), (24, 104), (30, 120), (25, 135),
                                    (6, 190), (5, 251)])
def test_lengths_around_the_rule(bw, pad):
    vol, ref = _volumes(bw, pad, pad)
    assert np.linalg.norm(vol - ref) <= REL_L2 * np.linalg.norm(ref)


def test_several_rounds_of_betas():
    """2 (B + padding) = 1032: two rounds of 128 threads.  Every third bin from beta 1, alpha 0, gamma 0 on is a bin
    of the 344-point volume."""
    vol, ref = _volumes(4, 512, 168)
    vol = vol[1::3, ::3, ::3]
    assert np.linalg.norm(vol - ref) <= REL_L2 * np.linalg.norm(ref)
