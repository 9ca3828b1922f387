"""Performance cases: the work a user of this framework has it do, through its public entry points.

Kinds of work:
  pair    SphOptRegistration.registerPointCloud on one pair of scans (the plain path, one pair at a time)
  served  a batch of requests submitted to a running Server, drained and polled
  align   voxelise two clouds and correlate them (the translation stage by itself, as PhaseAligner runs it)
  sample  S^2 sampling of one scan without allocation (sample_s2_noalloc)
  grid    voxel-grid downsampling of one scan into buffers of the caller's (phgpu_voxel_grid_filter of the C interface)

Clouds are seeded synthetic scans: the room of phaser_b200.scene, ray-cast here on the GPU, the target seen from a pose
uniform on SO(3) and within 2 m of the source's.  exact() restates the reference's arithmetic in plain torch in 64 bits;
what the reference itself decides in 32 bits (projected directions, nearest points, voxel and leaf indices) is decided
in 32 bits there too.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from phaser_b200 import core, native, scene

PRECISIONS = {"fp32": native.PHGPU_PRECISION_FP32, "tf32x3": native.PHGPU_PRECISION_TF32X3}
FUSIONS = {"laplace": native.PHGPU_FUSION_LAPLACE, "mix": native.PHGPU_FUSION_MIX}


def _pair_case(name, bw, n, half, beams, cols, pad=0, refl=True, precision="fp32", fusion="laplace", host=False):
    return dict(name=name, kind="pair", bw=bw, pad=pad, n=n, half=half, beams=beams, cols=cols, refl=refl,
                precision=precision, fusion=fusion, host=host)


def listed():
    return [
        # the smallest workload: a sparse scan on coarse grids, where launches and latency count
        _pair_case("pair_b32_n64", 32, 64, 10, 64, 1024, refl=False),
        # the reference's default flags (bandwidth 75, 100 voxels over [-50, 50]^3 m), the scans in host memory
        # as a reader of PLY files has them
        _pair_case("pair_b75_n100_host", 75, 100, 50, 64, 1024, host=True),
        # the headline workload, one pair at a time
        _pair_case("pair_b100_n200", 100, 200, 10, 128, 1024),
        # the same on the tensor-core contractions
        _pair_case("pair_b100_n200_tf32x3", 100, 200, 10, 128, 1024, precision="tf32x3"),
        # the reference's run script for a very fine registration: bandwidth 150 padded by 10, 201 voxels (odd)
        _pair_case("pair_b150p10_n201", 150, 201, 50, 128, 1024, pad=10),
        # the largest: a dense scan (about a million points) on the finest grids
        _pair_case("pair_b256_n512", 256, 512, 20, 256, 4096),
        # a full wave of the request server at the headline shape
        dict(name="served_16x_b100_n200", kind="served", shapes="100/200", count=16, wave=16, half=10, beams=128,
             cols=1024, precision="tf32x3"),
        # the arrivals mix of the server (50 % B=64/N=128, 35 % B=100/N=200, 15 % B=128/N=256)
        dict(name="served_mixed", kind="served", shapes="64/128,64/128,64/128,100/200,100/200,128/256", count=6, wave=4,
             half=10, beams=64, cols=1024, precision="tf32x3"),
        # the translation stage alone: a scan already rotated, four channels kept
        dict(name="align_n256", kind="align", n=256, half=10, beams=128, cols=1024),
        # sampling inside a loop that cannot allocate
        dict(name="sample_b100", kind="sample", bw=100, beams=128, cols=1024),
        # ingest: one scan downsampled to 0.25 m leaves on the device
        dict(name="grid_128x1024", kind="grid", leaf=0.25, beams=128, cols=1024, host=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _largest_prime(n):
    p, big = 2, 1
    while n > 1:
        if n % p:
            p += 1
        else:
            n, big = n // p, p
    return big


def _size(rng, lo, hi):
    """A transform length the framework takes (prime factors below 128); half of the draws are round sizes."""
    n = _log(rng, lo, hi)
    if rng.random() < 0.5:
        n = max(lo, n // 8 * 8)
    while _largest_prime(n) > 127:
        n += 1
    return n


def draw(rng):
    u = rng.random()
    scan = dict(beams=_log(rng, 16, 160), cols=_log(rng, 400, 2048))
    if u < 0.6:
        c = _pair_case("", _size(rng, 16, 160), _size(rng, 32, 256), rng.choice((10, 20, 50)), scan["beams"], scan["cols"],
                       pad=rng.choice((0, 0, 0, 4, 10)), refl=rng.random() < 0.7,
                       precision="tf32x3" if rng.random() < 0.3 else "fp32",
                       fusion="mix" if rng.random() < 0.15 else "laplace", host=rng.random() < 0.3)
        c.pop("name")
        return c
    if u < 0.7:
        shapes = ",".join("%d/%d" % (rng.choice((32, 64, 100, 128)), rng.choice((64, 128, 200))) for _ in range(rng.choice((1, 2))))
        return dict(kind="served", shapes=shapes, count=rng.randint(2, 12), wave=rng.choice((4, 8)), half=10, precision="tf32x3", **scan)
    if u < 0.8:
        return dict(kind="align", n=_size(rng, 32, 256), half=rng.choice((10, 20)), **scan)
    if u < 0.9:
        return dict(kind="sample", bw=rng.randint(16, 128), **scan)
    return dict(kind="grid", leaf=rng.choice((0.1, 0.25, 0.5)), host=rng.random() < 0.5, **scan)


# ---------------------------------------------------------------- inputs


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _hits(sc, origin, d):
    """Distance and unit normal of the first surface of the room, its boxes and its cylinders along each ray."""
    dev = d.device
    far = torch.as_tensor

    def t64(x):
        return far(x, dtype=torch.float64, device=dev)

    inv = 1.0 / torch.where(d.abs() < 1e-12, torch.full_like(d, 1e-12), d)
    best, axis = torch.maximum((t64(scene.ROOM_LO) - origin) * inv, (t64(scene.ROOM_HI) - origin) * inv).min(1)
    normal = torch.zeros_like(d).scatter_(1, axis[:, None], 1.0) * -torch.sign(d)
    for lo, hi in zip(sc.box_lo, sc.box_hi):
        a, b = (t64(lo) - origin) * inv, (t64(hi) - origin) * inv
        enter, axis = torch.minimum(a, b).max(1)
        hit = (enter <= torch.maximum(a, b).amin(1)) & (enter > 1e-6) & (enter < best)
        best = torch.where(hit, enter, best)
        normal = torch.where(hit[:, None], torch.zeros_like(d).scatter_(1, axis[:, None], 1.0) * -torch.sign(d), normal)
    qa = d[:, 0] ** 2 + d[:, 1] ** 2
    for (cx, cy), r in zip(sc.cyl_xy, sc.cyl_r):
        ox, oy = origin[0] - cx, origin[1] - cy
        qb = 2 * (ox * d[:, 0] + oy * d[:, 1])
        disc = qb * qb - 4 * qa * (ox * ox + oy * oy - r * r)
        t = (-qb - disc.clamp(min=0).sqrt()) / (2 * qa.clamp(min=1e-12))
        hit = (disc > 0) & (qa > 1e-12) & (t > 1e-6) & (t < best)
        best = torch.where(hit, t, best)
        n = torch.stack([(ox + t * d[:, 0]) / r, (oy + t * d[:, 1]) / r, torch.zeros_like(t)], 1)
        normal = torch.where(hit[:, None], n, normal)
    return best, normal


def _scan(sc, gen, R, t, beams, cols):
    """(xyzi, reflectivity) of a spinning scan in the sensor's frame, float32 on the GPU."""
    dev = gen.device
    el = torch.deg2rad(torch.linspace(-22.5, 22.5, beams, dtype=torch.float64, device=dev))
    az = 2 * math.pi * torch.arange(cols, dtype=torch.float64, device=dev) / cols
    E, A = torch.meshgrid(el, az, indexing="ij")
    ds = torch.stack([E.cos() * A.cos(), E.cos() * A.sin(), E.sin()], -1).reshape(-1, 3)
    dw = ds @ torch.as_tensor(R, dtype=torch.float64, device=dev).T
    dist, normal = _hits(sc, torch.as_tensor(t, dtype=torch.float64, device=dev), dw)

    def noise(sigma):
        return sigma * torch.randn(len(ds), generator=gen, dtype=torch.float64, device=dev)

    r = dist + noise(0.01)
    inten = (0.5 + 0.3 * (normal * dw).sum(1).abs() + noise(0.05)).clamp(0.0, 1.0)
    refl = inten * r * r
    xyzi = torch.cat([ds * r[:, None], inten[:, None]], 1).to(torch.float32).contiguous()
    return xyzi, (refl / refl.max()).to(torch.float32)


def _clouds(case, seed, k=0):
    """Target and source scans of one pair: ((xyzi, reflectivity), (xyzi, reflectivity))."""
    rng = np.random.default_rng([seed, k])
    sc = scene.make_scene(rng)
    R, t = scene.uniform_rotation(rng), rng.uniform(-2.0, 2.0, size=3)
    gen = torch.Generator(_device())
    gen.manual_seed(1000003 * seed + k)
    source = _scan(sc, gen, np.eye(3), np.zeros(3), case["beams"], case["cols"])
    target = _scan(sc, gen, R, t, case["beams"], case["cols"])
    if not case.get("refl", True):
        target, source = (target[0], None), (source[0], None)
    if case.get("host") and torch.cuda.is_available():  # page-locked, as a reader that uploads next keeps them
        target, source = (tuple(None if x is None else x.cpu().pin_memory() for x in c) for c in (target, source))
    return target, source


class _Grid:
    """A voxel-grid filter's handle."""

    def __init__(self, max_points):
        self.lib, self.h = native.load(), ctypes.c_void_p()
        if self.lib.phgpu_voxel_grid_create(max_points, 0, ctypes.byref(self.h)) != native.PHGPU_OK:
            raise RuntimeError("phgpu_voxel_grid_create failed")

    def __del__(self):
        self.lib.phgpu_voxel_grid_destroy(self.h)


def _shapes(case):
    s = [tuple(int(x) for x in p.split("/")) for p in case["shapes"].split(",")]
    return [s[k % len(s)] for k in range(case["count"])]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "pair":
        reg = core.SphOptRegistration(case["bw"], case["n"], -case["half"], case["half"],
                                      spherical_zero_padding=case["pad"], precision=PRECISIONS[case["precision"]],
                                      spherical_fusion=FUSIONS[case["fusion"]], max_points=case["beams"] * case["cols"])
        target, source = _clouds(case, seed)
        return dict(kind=kind, reg=reg, target=target, source=source)
    if kind == "served":
        srv = native.Server(max_wave=case["wave"], max_points=case["beams"] * case["cols"])
        reqs = [(native.default_params(spherical_bandwidth=b, spatial_n_voxels=n, spatial_discretize_lower=-case["half"],
                                       spatial_discretize_upper=case["half"], precision=PRECISIONS[case["precision"]]),
                 *_clouds(case, seed, k)) for k, (b, n) in enumerate(_shapes(case))]
        state = dict(kind=kind, srv=srv, reqs=reqs)
        torch.cuda.synchronize()  # the clouds are ready before the server's threads read them
        run(state)  # a running server has its executors
        return state
    if kind == "align":
        ctx = native.Context(spherical_bandwidth=2, spatial_n_voxels=case["n"], spatial_discretize_lower=-case["half"],
                             spatial_discretize_upper=case["half"], max_points=case["beams"] * case["cols"])
        target, source = _clouds(case, seed)
        return dict(kind=kind, ctx=ctx, target=target, source=source)
    cloud = _clouds(case, seed)[0]
    if kind == "sample":
        prm = native.default_params(spherical_bandwidth=case["bw"])
        nq = 4 * case["bw"] ** 2
        return dict(kind=kind, prm=prm, cloud=cloud, values=torch.empty(4, nq, dtype=torch.float32, device=_device()),
                    index=torch.empty(nq, dtype=torch.int32, device=_device()), stream=torch.cuda.current_stream())
    pts = case["beams"] * case["cols"]
    where = dict(dtype=torch.float32, device="cpu" if case["host"] else _device(), pin_memory=bool(case["host"]))
    return dict(kind=kind, vg=_Grid(pts), cloud=cloud, leaf=(ctypes.c_float * 3)(*(case["leaf"],) * 3), count=ctypes.c_uint32(),
                xyzi=torch.zeros(pts, 4, **where), refl=torch.zeros(pts, **where), on_device=0 if case["host"] else 1)


def run(state):
    kind = state["kind"]
    if kind == "pair":
        return state["reg"].registerPointCloud(state["target"], state["source"])
    if kind == "served":
        srv = state["srv"]
        tickets = [srv.submit(prm, t, s) for prm, t, s in state["reqs"]]
        srv.drain()
        poses = [srv.poll(t)[0] for t in tickets]
        return dict(rot_bin=np.array([p.rot_bin for p in poses], np.int64), voxel=np.array([p.voxel for p in poses], np.int64),
                    rot_peak=np.array([p.rot_peak for p in poses], np.float32),
                    trans_peak=np.array([p.trans_peak for p in poses], np.float32),
                    quat=np.array([list(p.quat) for p in poses]), trans=np.array([list(p.trans) for p in poses]))
    if kind == "align":
        ctx = state["ctx"]
        ctx.voxelize(*state["target"], side=0)
        ctx.voxelize(*state["source"], side=1)
        ctx.spatial_correlate_voxelized()
        voxel, peak = ctx.spatial_result()
        return dict(voxel=voxel, peak=peak)
    if kind == "sample":
        xyzi, refl = state["cloud"]
        rc = native.sample_s2_noalloc(state["prm"], xyzi, refl, None, state["values"], state["index"], state["stream"])
        if rc != native.PHGPU_OK:
            raise RuntimeError("sample_s2_noalloc: %d" % rc)
        return dict(values=state["values"], index=state["index"])
    vg, o, r = state["vg"], state["xyzi"], state["refl"]
    cloud, _keep = native.make_cloud(*state["cloud"])
    rc = vg.lib.phgpu_voxel_grid_filter(vg.h, ctypes.byref(cloud), state["leaf"], 0, o.data_ptr(), r.data_ptr(), None,
                                        state["on_device"], ctypes.byref(state["count"]))
    if rc != native.PHGPU_OK:
        raise RuntimeError("phgpu_voxel_grid_filter: %d" % rc)
    return dict(leaves=state["count"].value, xyzi=o, reflectivity=r)  # entries past the leaves stay zero


# ---------------------------------------------------------------- work


def _pair_flops(bw, pad, n, channels, mix=False):
    no, c = 2 * (bw + pad), 1 if mix else channels
    sht = 2 * c * (2.5 * (2 * bw) ** 2 * math.log2(2 * bw) + 2 * 2 * bw * bw * bw)  # phi transforms, Legendre sums
    synth = 4 * no * (2 * bw ** 3 / 3)  # a complex coefficient times a real d-value, half of the orders
    angles = 2 * 2.5 * no ** 3 * math.log2(no)
    return sht + synth + angles + _spatial_flops(n, channels)


def _spatial_flops(n, channels):
    return (2 * channels + 1) * 2.5 * n ** 3 * math.log2(n ** 3) + n ** 3 * 4 * channels


def work(case):
    kind, pts = case["kind"], case["beams"] * case["cols"]
    if kind == "pair":
        ch = 3 if case["refl"] else 2
        return dict(bytes=2 * pts * 4 * (ch + 2), flops=_pair_flops(case["bw"], case["pad"], case["n"], ch, case["fusion"] == "mix"))
    if kind == "served":
        return dict(bytes=case["count"] * 2 * pts * 20, flops=sum(_pair_flops(b, 0, n, 3) for b, n in _shapes(case)))
    if kind == "align":
        return dict(bytes=2 * pts * 20, flops=_spatial_flops(case["n"], 3))
    if kind == "sample":
        return dict(bytes=pts * 20 + 4 * case["bw"] ** 2 * 20, flops=pts * 20)
    return dict(bytes=pts * 20 + pts, flops=pts * 5)


# ---------------------------------------------------------------- 64-bit values


def _sampled(cloud, bw):
    """Range, intensity and reflectivity of the nearest point (32-bit directions and distances, the lowest index
    among equals) of each grid direction, in 64 bits, and the points' indices."""
    xyzi, refl = cloud
    x, y, z, w = xyzi.unbind(1)
    dist = ((x * x + y * y).sqrt().double() ** 2 + (z * z).double()).sqrt()
    oz = (z.double() / dist).float()
    th, ph = torch.acos(oz.double()).float().double(), torch.atan2(y.double(), x.double()).float().double()
    ph = torch.fmod(ph + 2 * math.pi, 2 * math.pi)
    px, py, pz = (th.sin() * ph.cos()).float(), (th.sin() * ph.sin()).float(), oz
    n = 2 * bw
    tq = (math.pi * (2 * np.arange(n) + 1) / (4 * bw)).astype(np.float32)
    pq = (2 * math.pi * np.arange(n) / (2 * bw)).astype(np.float32)
    st, ct, sp, cp = (fn(v.astype(np.float64)).astype(np.float32) for v in (tq, pq) for fn in (np.sin, np.cos))
    grid = np.stack([np.outer(st, cp), np.outer(st, sp), np.outer(ct, np.ones_like(ct))], -1)
    q = torch.as_tensor(grid.reshape(-1, 3), device=xyzi.device)
    at = torch.arange(len(x), device=x.device, dtype=torch.int32)
    index = []
    step = max(1, (1 << 27) // max(len(x), 1))
    for c in q.split(step):
        d = (c[:, 0:1] - px) ** 2
        d += (c[:, 1:2] - py) ** 2
        d += (c[:, 2:3] - pz) ** 2
        low = d.amin(1, keepdim=True)
        index.append(torch.where(d == low, at, torch.full_like(at, 0x7fffffff)).amin(1))
    index = torch.cat(index).long()
    chans = [dist.float().double(), w.double()] + ([] if refl is None else [refl.double()])
    return [c[index].reshape(n, n) for c in chans], index


def _bands(n, levels=5):
    """(start, end, zero end) of each level of the channel pyramid over n shifted positions."""
    out, cur, f = [], n, np.float32
    for _ in range(levels):
        lower = f(cur) / f(4)
        lo, up = math.floor(float(lower) + 0.5), math.floor(float(f(f(cur) - lower)) + 0.5)
        out.append((lo, cur - lo, up))
        cur = up - lo
    return out


def _fuse(chans, p, n):
    """Channels at shifted positions p of n: the largest inside the pyramid's bands, their mean (over four) in the core."""
    x = torch.stack(chans)
    i = (x.real ** 2 + x.imag ** 2).argmax(0, keepdim=True)
    big, mean, zero = x.gather(0, i)[0], x.sum(0) / 4, torch.zeros_like(x[0])
    out, inside, p = big, torch.ones_like(p, dtype=torch.bool), p.clone()
    for lo, end, up in _bands(n):
        into = inside & (p >= lo) & (p < end)
        out = torch.where(inside & ~into & (p >= lo) & (p < up), zero, out)
        p = torch.where(into, p - lo, p)
        inside = into
    return torch.where(inside, mean, out)


def _harmonics(grid, bw):
    """Coefficients [l][m + bw - 1] of a real signal on the 2B x 2B grid (Driscoll-Healy quadrature)."""
    dev, n = grid.device, 2 * bw
    k = torch.arange(n, device=dev, dtype=torch.float64)
    th = math.pi * (2 * k + 1) / (4 * bw)
    i = torch.arange(bw, device=dev, dtype=torch.float64)[:, None]
    w = 2.0 / bw * th.sin() * (((2 * i + 1) * th).sin() / (2 * i + 1)).sum(0)
    F = torch.fft.fft(grid, dim=1)[:, :bw].T * (math.sqrt(2 * math.pi) / n)  # [m][theta]
    m = torch.arange(bw, device=dev, dtype=torch.float64)[:, None]
    lg = 0.5 * (((2 * m + 1) / 2).log() + torch.lgamma(2 * m + 1) - 2 * torch.lgamma(m + 1) - m * math.log(4.0)) + m * th.sin().log()
    seed = torch.where(m % 2 == 1, -1.0, 1.0) * lg.exp()
    cur, prev = torch.zeros(bw, n, device=dev, dtype=torch.float64), torch.zeros(bw, n, device=dev, dtype=torch.float64)
    out = torch.zeros(bw, 2 * bw - 1, device=dev, dtype=torch.complex128)
    sign = torch.where(m[:, 0] % 2 == 1, -1.0, 1.0)
    for l in range(bw):
        if l:
            den = ((l - m) * (l + m)).clamp(min=1.0)
            a = ((2 * l - 1.0) * (2 * l + 1.0) / den).sqrt()
            b = ((2 * l + 1.0) * ((l - 1 - m) * (l - 1 + m)).clamp(min=0.0) / ((2 * l - 3.0) * den)).sqrt() if l > 1 else 0 * m
            cur, prev = a * th.cos() * cur - b * prev, cur
        cur = torch.where(m == l, seed, torch.where(m > l, torch.zeros_like(cur), cur))
        prev = torch.where(m >= l, torch.zeros_like(prev), prev)
        c = ((w * cur) * F).sum(1)
        out[l, bw - 1:bw + l] = c[:l + 1]
        out[l, bw - 1 - l:bw] = (sign * c.conj())[:l + 1].flip(0)
    return out


def _rotation_volume(fused_f, fused_g, bw, bw_out):
    """Yields (first beta, the correlation's squared values [beta][alpha][gamma]) in slabs of betas."""
    dev, n = fused_f.device, 2 * bw_out
    m1 = torch.arange(-(bw - 1), bw, device=dev)[:, None]
    m2 = torch.arange(0, bw, device=dev)[None, :]
    a, b = m1.double(), m2.double()
    j = torch.maximum(m1.abs(), m2)
    mn = torch.minimum(m1.abs(), m2).double()
    outer = (m1.abs() >= m2)
    cp = torch.where(outer, torch.where(m1 >= 0, j + m2, j - m2), j + m1).double()
    sp = torch.where(outer, torch.where(m1 >= 0, j - m2, j + m2), j - m1).double()
    sgn = torch.where(outer & (m1 >= 0) & ((j - m2) % 2 == 1), -1.0, 1.0).double()
    jd = j.double()
    lnorm = 0.5 * ((jd + 0.5).log() + torch.lgamma(2 * jd + 1) - torch.lgamma(jd - mn + 1) - torch.lgamma(jd + mn + 1))
    par = torch.where((m1 + m2) % 2 == 0, 1.0, -1.0).double()
    direct = (m1 >= 0) | (m2 == -m1)
    rows, cols = (torch.arange(bw, device=dev), torch.arange(-(bw - 1), bw, device=dev))
    step = max(2, min(n, (1 << 24) // (2 * bw * bw)))
    for k0 in range(0, n, step):
        k = torch.arange(k0, min(n, k0 + step), device=dev, dtype=torch.float64)
        beta = math.pi * (2 * k + 1) / (4 * bw_out)
        cb, lc, ls = beta.cos(), (0.5 * beta).cos().log(), (0.5 * beta).sin().log()
        seed = sgn[..., None] * (lnorm[..., None] + cp[..., None] * lc + sp[..., None] * ls).exp()
        cur = torch.zeros_like(seed)
        prev = torch.zeros_like(seed)
        S = torch.zeros(seed.shape, dtype=torch.complex128, device=dev)
        for l in range(bw):
            if l:
                d = l - 1.0
                t1 = (((d + 1) ** 2 - a * a).clamp(min=0) * ((d + 1) ** 2 - b * b).clamp(min=0)).sqrt()
                inv = torch.where(t1 > 0, 1 / t1, torch.zeros_like(t1))
                fb = math.sqrt((2 * d + 3) / (2 * d + 1)) * (d + 1) * (2 * d + 1) * inv
                if l > 1:
                    t0 = ((d * d - a * a).clamp(min=0) * (d * d - b * b).clamp(min=0)).sqrt()
                    fa = -math.sqrt((2 * d + 3) / (2 * d - 1)) * (d + 1) / d * t0 * inv
                    sh = -a * b / (d * (d + 1))
                else:
                    fa, sh = torch.zeros_like(fb), torch.zeros_like(fb)
                cur, prev = fa[..., None] * prev + fb[..., None] * (cb + sh[..., None]) * cur, cur
            new = (j == l)[..., None]
            cur = torch.where(new, seed, torch.where((j > l)[..., None], torch.zeros_like(cur), cur))
            prev = torch.where(new, torch.zeros_like(prev), prev)
            f, g = fused_f[l], fused_g[l]  # [m + bw - 1]
            wn = 2 * math.pi * math.sqrt(2 / (2 * l + 1.0))
            one = f.flip(0)[:, None] * g.conj().flip(0)[None, bw - 1:]  # f(l, -m1) conj(g(l, -m2)), m2 >= 0
            two = (f[:, None] * g.conj()[None, bw - 1:]).conj() * par    # the conjugate of the pair (-m1, -m2)
            S += (wn * par * torch.where(direct, one, two))[..., None] * cur
        full = torch.zeros(n, n, len(k), dtype=torch.complex128, device=dev)
        full[(m1 % n).reshape(-1, 1), m2.reshape(1, -1)] = S
        T = torch.fft.fft(full, dim=0)
        T[:, 0] = 0.5 * T[:, 0].real
        z = 2 * torch.fft.fft(T, dim=1).real * (bw_out / (math.pi * n))
        yield k0, (z * z).permute(2, 0, 1)


def _rotation(target, source, case):
    """(bin, squared correlation) of the best rotation."""
    bw, bw_out = case["bw"], case["bw"] + case.get("pad", 0)
    spectra = []
    m = torch.arange(-(bw - 1), bw, device=target[0].device)[None, :]
    l = torch.arange(bw, device=m.device)[:, None]
    L, am = bw - 1, m.abs()
    pos = torch.where(m >= 0, m * (L + 1) - (m * (m - 1)) // 2 + (l - m),
                      (L * (L + 3)) // 2 + 1 + ((L + m) * (L + m + 1)) // 2 + (l - am))
    for cloud in (target, source):
        ch, _ = _sampled(cloud, bw)
        if case.get("fusion") == "mix":
            spectra.append(_harmonics(0.6 * ch[1] + 0.4 * ch[0], bw))
        else:
            f = _fuse([_harmonics(c, bw) for c in ch], torch.where(l >= am, (pos + bw * bw // 2) % (bw * bw), 0 * pos), bw * bw)
            spectra.append(torch.where(l >= am, f, torch.zeros_like(f)))
    best, where = -1.0, 0
    for k0, v in _rotation_volume(*spectra, bw, bw_out):
        top = v.reshape(-1).argmax()
        if v.reshape(-1)[top].item() > best:
            best, where = v.reshape(-1)[top].item(), k0 * v.shape[1] * v.shape[2] + top.item()
    return where, best


def _rotated(cloud, rot_bin, bw_out):
    """The cloud turned by the rotation of a bin: its Euler angles' matrices and the points in 32 bits, as the reference."""
    n, f = 2 * bw_out, np.float32
    i, jk = divmod(rot_bin, n * n)
    al, be, ga = math.pi * (jk // n) / bw_out, math.pi * (2 * i + 1) / (4.0 * bw_out), math.pi * (jk % n) / bw_out
    c, s = math.cos(be / 2), math.sin(be / 2)
    w, x, y, z = c * math.cos((al + ga) / 2), s * math.sin((ga - al) / 2), s * math.cos((ga - al) / 2), c * math.sin((al + ga) / 2)
    e = (math.atan2(-2 * (y * z - w * x), w * w - x * x - y * y + z * z), math.asin(2 * (x * z + w * y)),
         -math.atan2(-2 * (x * y - w * z), w * w + x * x - y * y - z * z))
    (ca, cb, cc), (sa, sb, sc) = ([f(fn(float(f(v)))) for v in e] for fn in (math.cos, math.sin))
    X = np.array([[1, 0, 0], [0, ca, -sa], [0, sa, ca]], f)
    Y = np.array([[cb, 0, sb], [0, 1, 0], [-sb, 0, cb]], f)
    Z = np.array([[cc, sc, 0], [-sc, cc, 0], [0, 0, 1]], f)

    def product(A, B):
        return np.array([[f(f(f(A[r, 0] * B[0, q]) + f(A[r, 1] * B[1, q])) + f(A[r, 2] * B[2, q])) for q in range(3)] for r in range(3)], f)

    T = product(product(X, Y), Z)
    p = cloud[0].unbind(1)
    o = []
    for r in range(3):
        v = float(T[r, 0]) * p[0]
        v = v + float(T[r, 1]) * p[1]
        o.append(v + float(T[r, 2]) * p[2])
    return torch.stack([*o, p[3]], 1), cloud[1]


def _voxels(cloud, n, half):
    """Mean intensity, range and reflectivity per voxel [z][x][y], in 64 bits."""
    xyzi, refl = cloud
    f = np.float32
    e = (f(-half) + np.arange(n).astype(f) * ((f(half) - f(-half)) / f(n - 1))).astype(f)
    e[-1] = half
    E = torch.as_tensor(e, device=xyzi.device)
    b = []
    for v in xyzi[:, :3].unbind(1):
        i = (torch.searchsorted(E, v.contiguous(), right=True) - 1).clamp(max=n - 1)
        b.append(torch.where((v < E[0]) | (v > E[-1]), torch.full_like(i, 0xffffffff), i))
    lin = (((b[0] * n) & 0xffffffff) + b[1] + ((n * n * b[2]) & 0xffffffff)) & 0xffffffff
    ok = lin < n ** 3
    lin = lin[ok]
    x, y, z, w = xyzi[ok].unbind(1)
    chans = [w.double(), ((x * x + y * y) + z * z).sqrt().double()] + ([] if refl is None else [refl[ok].double()])
    count = torch.zeros(n ** 3, dtype=torch.float64, device=x.device).index_add_(0, lin, torch.ones_like(chans[0]))
    return [(torch.zeros_like(count).index_add_(0, lin, c) / count.clamp(min=1)).reshape(n, n, n) for c in chans]


def _translation(target, source, n, half):
    """The largest value of the spatial correlation."""
    h = n // 2 + 1
    p = (torch.arange(n * n * h, device=target[0].device).reshape(n, n, h) + n ** 3 // 2) % n ** 3
    F, G = (_fuse([torch.fft.rfftn(c, dim=(0, 1, 2)) for c in _voxels(cloud, n, half)], p, n ** 3) for cloud in (target, source))
    C = torch.fft.ifft2(F * G.conj(), dim=(0, 1), norm="forward")
    C[..., 0].imag.zero_()
    if n % 2 == 0:
        C[..., h - 1].imag.zero_()
    return torch.fft.irfft(C, n=n, dim=2, norm="forward").max().item()


def _on_device(cloud):
    return tuple(None if x is None else x.to(_device()) for x in cloud)


def _peaks(target, source, case):
    target, source = _on_device(target), _on_device(source)
    b, rot = _rotation(target, source, case)
    return rot, _translation(target, _rotated(source, b, case["bw"] + case.get("pad", 0)), case["n"], case["half"])


def exact(case, seed):
    kind = case["kind"]
    none = None
    if kind == "pair":
        rot, trans = _peaks(*_clouds(case, seed), case)
        return dict(rot_peak=rot, trans_peak=trans)
    if kind == "served":
        got = [_peaks(*_clouds(case, seed, k), dict(case, bw=b, n=n)) for k, (b, n) in enumerate(_shapes(case))]
        return dict(rot_bin=none, voxel=none, rot_peak=np.array([g[0] for g in got]), trans_peak=np.array([g[1] for g in got]),
                    quat=none, trans=none)
    target, source = (_on_device(c) for c in _clouds(case, seed))
    if kind == "align":
        return dict(voxel=none, peak=_translation(target, source, case["n"], case["half"]))
    if kind == "sample":
        ch, _ = _sampled(target, case["bw"])
        return dict(values=torch.stack([*(c.reshape(-1) for c in ch), torch.zeros_like(ch[0].reshape(-1))]), index=none)
    xyzi, refl = target
    inv = 1 / np.float32(case["leaf"])
    ijk = (xyzi[:, :3] * float(inv)).floor().long()
    ijk = ijk - ijk.amin(0)
    d = ijk.amax(0) + 1
    _, leaf, count = torch.unique(ijk[:, 0] + d[0] * (ijk[:, 1] + d[1] * ijk[:, 2]), return_inverse=True, return_counts=True)
    rows = torch.cat([xyzi, refl[:, None]], 1).double()
    mean = torch.zeros(len(rows), 5, dtype=torch.float64, device=rows.device).index_add_(0, leaf, rows)
    mean[:len(count)] /= count[:, None]
    return dict(leaves=none, xyzi=mean[:, :4].contiguous(), reflectivity=mean[:, 4].contiguous())
