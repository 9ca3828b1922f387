"""Device clouds read in place: ones that are not 16-byte aligned (copied instead), ones whose size changes from call to
call on one context (its buffers grow in between), one side on the device and the other in host memory.  Results equal
those of a fresh context on host copies, and the caller's tensors keep their values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nat():
    from phaser_b200 import native
    native.load()
    return native


def cloud(seed, n):
    rng = np.random.default_rng([seed, n])
    v = rng.standard_normal((n, 3))
    v *= rng.uniform(3, 9, (n, 1)) / np.linalg.norm(v, axis=1, keepdims=True)
    return np.concatenate([v, rng.uniform(0, 1, (n, 1))], 1).astype(np.float32), rng.uniform(0, 1, n).astype(np.float32)


def on_device(c, shift):
    """The cloud in CUDA tensors `shift` floats past an aligned address."""
    import torch
    out = []
    for x in c:
        base = torch.zeros(x.size + shift, device="cuda")
        base[shift:] = torch.as_tensor(x.reshape(-1)).cuda()
        out.append(base[shift:].view(x.shape))
    torch.cuda.synchronize()
    assert out[0].is_contiguous() and out[0].data_ptr() % 16 == 4 * shift % 16
    return tuple(out)


KW = dict(spherical_bandwidth=12, spatial_n_voxels=24, spatial_discretize_lower=-10, spatial_discretize_upper=10)


def results(c, t, s):
    p = c.register_pair(t, s)
    samples = [c.samples(k) for k in (0, 1)]
    c.sample_s2(*t, side=1)
    c.voxelize(*s, side=0)
    return (p.rot_bin, p.voxel), samples + [c.samples(1)], c.voxel_index(0, len(s[0]))


def same(a, b):
    assert a[0] == b[0]
    for x, y in zip(a[1], b[1]):
        assert np.array_equal(x[0], y[0]) and np.array_equal(x[1], y[1])
    assert np.array_equal(a[2], b[2])


@pytest.mark.parametrize("shift", [0, 1, 2, 3, 4])
def test_any_alignment(nat, shift):
    t, s = cloud(1, 3001), cloud(2, 2500)
    want = results(nat.Context(**KW), t, s)
    dt, ds = on_device(t, shift), on_device(s, shift)
    same(results(nat.Context(**KW), dt, ds), want)
    same(results(nat.Context(**KW), dt, s), want)  # one side in host memory
    for dev, host in zip(dt + ds, t + s):
        assert np.array_equal(dev.cpu().numpy(), host)


def test_sizes_change_on_one_context(nat):
    c = nat.Context(max_points=64, **KW)
    for i, (n, m) in enumerate([(50, 60), (5000, 40), (40, 9000), (9001, 12000), (1, 12000), (300, 2)]):
        t, s = cloud(i, n), cloud(10 + i, m)
        dt, ds = on_device(t, i % 2), on_device(s, 0)
        want = results(nat.Context(**KW), t, s)
        same(results(c, dt, ds), want)
        same(results(c, t, ds), want)
