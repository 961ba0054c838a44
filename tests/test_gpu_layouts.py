"""Large trilinear calls, whose kernel may depend on the layout of their points:
which route a layout takes (named in the debug log), that every route gives
the same bits as calls below the thresholds, and that calls other than those
on dense float volumes return without waiting for their stream."""
import threading

import numpy as np
import pytest

from openvkl_b200.fields import orbit_camera_samples_torch, shell_leaves, sinusoid_field, uniform_points_torch
from tests.conftest import bits

pytestmark = pytest.mark.gpu

DIMS = (160, 150, 170)
TYPES = [np.uint8, np.int16, np.uint16, np.float16, np.float64]


def _voxels(dtype, dims=DIMS):
    f = sinusoid_field(dims, seed=3)
    return (f * 25 + 100).astype(dtype) if np.dtype(dtype).kind in "iu" else f.astype(dtype)


def _points(order, n, hi):
    """n points by rays of `order` samples (an image 125 rays wide, the last
    ray cut), in no order, or close together in no order by rays: each 2048
    consecutive ones anywhere in one box of a few hundred sort bins."""
    import torch
    if order == "none":
        return uniform_points_torch(n, (-1, -1, -1), hi, seed=6)
    if order == "boxes":
        g = torch.Generator(device="cuda")
        g.manual_seed(7)
        size = torch.tensor([64.0, 64.0, 32.0], device="cuda")
        boxes = n // 2048 + 1
        at = torch.rand((boxes, 1, 3), generator=g, device="cuda") * (torch.tensor(hi, device="cuda") - size)
        return (at + torch.rand((boxes, 2048, 3), generator=g, device="cuda") * size).reshape(-1, 3)[:n].contiguous()
    return orbit_camera_samples_torch(125, n // (125 * order) + 1, order, (0, 0, 0), hi, seed=5)[:n].contiguous()


def _logged(vkl, **params):
    dev = vkl.Device("cuda")
    log = []
    dev.capture_log(log)
    dev.set_int("logLevel", 1)  # debug
    for k, v in params.items():
        dev.set_int(k, v)
    return dev, log


def _check(vkl, vol, log, route, pts, step, times=None):
    """Whole calls against calls of `step` points, which no detector looks at.
    route: what the log names, None where the layout does not matter."""
    import torch
    n = pts.shape[0]
    s = vkl.Sampler(vol, filter=100, gradient_filter=100)
    cut = [slice(i, min(i + step, n)) for i in range(0, n, step)]
    t = (lambda c: None) if times is None else (lambda c: times[c].contiguous())
    for call, shape in ((s.sample, (n,)), (s.gradient, (n, 3))):
        out = torch.full(shape, -77.0, device="cuda")
        log.clear()
        call(pts, out=out, times=times)
        named = [m for m in log if "sampling" in m]
        assert (not named) if route is None else any(route in m for m in named), (route, log)
        log.clear()
        parts = torch.cat([call(pts[c].contiguous(), times=t(c)) for c in cut])
        assert not any("sampling" in m for m in log), log
        np.testing.assert_array_equal(bits(out.cpu().numpy()), bits(parts.cpu().numpy()))


@pytest.mark.parametrize("texture", [1, 0])
@pytest.mark.parametrize("order,route", [(37, "as runs of 37 samples"), (19, "by rays of 19 samples"),
                                         (24, "by rays of 24 samples"), ("none", "point by point"),
                                         ("boxes", "in sorted tiles")])
def test_float(vkl, order, route, texture):
    """Rays whose warps touch up to 12 blocks of 16x16x2 voxels, up to 20, and
    points of either other kind."""
    dev, log = _logged(vkl, textureSampling=texture)
    vol = vkl.structured_regular(dev, _voxels(np.float32), background=[0.5])
    pts = _points(order, (1 << 20) + 5, tuple(float(d - 1) for d in DIMS))
    _check(vkl, vol, log, route, pts, 500009)


@pytest.mark.parametrize("dtype,texture", [(t, 1) for t in TYPES] + [(np.uint8, 0), (np.int16, 0)])
@pytest.mark.parametrize("order", [37, "none"])
def test_types_other_than_float(vkl, dtype, texture, order):
    """Sorted tiles from 2^22 points, whatever the layout."""
    dev, log = _logged(vkl, textureSampling=texture)
    vol = vkl.structured_regular(dev, _voxels(dtype), background=[0.5])
    pts = _points(order, (1 << 22) + 5, tuple(float(d - 1) for d in DIMS))
    _check(vkl, vol, log, None, pts, 3000007)


@pytest.mark.parametrize("order,route", [(50, "by rays of 50 samples"), (300, "by rays of 300 samples"),
                                         (40, "point by point"), ("none", "point by point")])
@pytest.mark.parametrize("dtype,steps", [("float32", 3), ("uint8", 11)])
def test_temporal(vkl, dtype, steps, order, route):
    import torch
    dev, log = _logged(vkl)
    dims = (256, 256, 200)
    g = torch.Generator(device="cuda")
    g.manual_seed(2)
    vox = torch.rand((dims[0] * dims[1] * dims[2] * steps,), generator=g, device="cuda")
    vox = (vox * 255).to(torch.uint8) if dtype == "uint8" else vox
    vol = vkl.structured_regular(dev, vox, dims=dims, num_timesteps=steps, background=[0.5], shared=True)
    n = (3 << 22) + 77
    pts = _points(order, n, tuple(float(d - 1) for d in dims))
    _check(vkl, vol, log, route, pts, 7000003, torch.rand(n, generator=g, device="cuda"))


def test_small_temporal_volume(vkl):
    """A volume that the caches hold takes its points as they come."""
    import torch
    dev, log = _logged(vkl)
    vox = np.random.default_rng(2).normal(size=(DIMS[0] * DIMS[1] * DIMS[2] * 2,)).astype(np.float32)
    vol = vkl.structured_regular(dev, vox, dims=DIMS, num_timesteps=2, background=[0.5])
    n = (3 << 22) + 77
    _check(vkl, vol, log, None, _points(300, n, tuple(float(d - 1) for d in DIMS)), 7000003, torch.rand(n, device="cuda"))


@pytest.mark.parametrize("order", [37, "none"])
@pytest.mark.parametrize("compression", ["fp16_blocks", "fp8_blocks"])
def test_block_leaves(vkl, compression, order):
    dev, log = _logged(vkl)
    origins, values = shell_leaves(domain=96, shells=2, thickness=0.1, seed=9)
    L = len(origins)
    vol = vkl.vdb_volume(dev, np.full(L, 3), origins, np.ones(L), packed_dense=values, compression=compression,
                         background=[0.25])
    _check(vkl, vol, log, None, _points(order, (1 << 20) + 77, (95.0, 95.0, 95.0)), 1000003)


def _volume(vkl, dev, kind):
    """A volume of the kind, and points per call as large calls have them."""
    import torch
    if kind == "temporal":
        dims = (256, 256, 200)
        g = torch.Generator(device="cuda")
        g.manual_seed(2)
        vox = torch.rand((dims[0] * dims[1] * dims[2] * 3,), generator=g, device="cuda")
        return vkl.structured_regular(dev, vox, dims=dims, num_timesteps=3, background=[0.5], shared=True), 3 << 22
    if kind == "blocks":
        origins, values = shell_leaves(domain=96, shells=2, thickness=0.1, seed=9)
        L = len(origins)
        return vkl.vdb_volume(dev, np.full(L, 3), origins, np.ones(L), packed_dense=values, compression="fp16_blocks",
                              background=[0.25]), 1 << 20
    return vkl.structured_regular(dev, _voxels(kind), background=[0.5]), 1 << 22


@pytest.mark.parametrize("kind", TYPES + ["temporal", "blocks"])
def test_call_returns_before_its_stream(vkl, kind):
    """Behind half a second of other work on the stream, the call has to
    return while that work still runs."""
    import torch
    dev = vkl.Device("cuda")
    stream = torch.cuda.Stream()
    dev.set_stream(stream.cuda_stream)
    vol, n = _volume(vkl, dev, kind)
    pts = _points(37, n, tuple(float(d - 1) for d in DIMS))
    out = torch.empty(n, device="cuda")
    s = vkl.Sampler(vol, filter=100)
    s.sample(pts, out=out)
    torch.cuda.synchronize()
    done = torch.cuda.Event()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(1_000_000_000)
        done.record()
    s.sample(pts, out=out)
    returned_first = not done.query()
    torch.cuda.synchronize()
    assert returned_first


def test_many_streams_and_threads(vkl):
    """More streams than the detector keeps answers for, with different
    layouts, queued without waiting; then threads on one device."""
    import torch
    dev = vkl.Device("cuda")
    vol, n = _volume(vkl, dev, "temporal")
    n += 3
    s = vkl.Sampler(vol, filter=100)
    orders = [50, "none", 300, 37]
    pts = [_points(o, n, (255.0, 255.0, 199.0)) for o in orders]
    tm = torch.rand(n, device="cuda")
    step = 7000003
    want = [torch.cat([s.sample(p[i:i + step].contiguous(), times=tm[i:i + step].contiguous())
                       for i in range(0, n, step)]) for p in pts]
    streams = [torch.cuda.Stream() for _ in range(20)]
    outs = [torch.full((n,), -77.0, device="cuda") for _ in range(40)]  # 2 GB
    torch.cuda.synchronize()
    for k, out in enumerate(outs):
        dev.set_stream(streams[k % 20].cuda_stream)
        s.sample(pts[k * 7 % 4], out=out, times=tm)
    torch.cuda.synchronize()
    for k, out in enumerate(outs):
        assert torch.equal(out, want[k * 7 % 4]), k
        out.fill_(-77.0)
    torch.cuda.synchronize()

    def work(w):
        for k in range(w, 40, 4):
            s.sample(pts[w], out=outs[k], times=tm)

    threads = [threading.Thread(target=work, args=(w,)) for w in range(4)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    torch.cuda.synchronize()
    for k, out in enumerate(outs):
        assert torch.equal(out, want[k % 4]), k
