"""Several attributes of one call: below some hundred thousand points a thread
per point, above it sorted tiles.  Every column has the bits of the
single-attribute call on both sides of the lines (2^18 points, 2^19 where the
tiles would gather with plain loads), and a call of few points takes about as
long as its attributes one by one."""
import numpy as np
import pytest

from openvkl_b200.fields import orbit_camera_samples_torch, shell_leaves, sinusoid_field
from tests.conftest import bits

pytestmark = pytest.mark.gpu

DIMS = (60, 70, 50)


def _dense(vkl, dtype, count, **params):
    dev = vkl.Device("cuda")
    for k, v in params.items():
        dev.set_int(k, v)
    scale, offset = (25, 100) if np.dtype(dtype).kind in "iu" else (1, 0)
    vox = [(sinusoid_field(DIMS, seed=50 + i) * scale + offset).astype(dtype) for i in range(count)]
    return vkl.structured_regular(dev, vox, background=[0.5] * count)


def _sparse(vkl, count, leaf_map=True, compression=None):
    origins, values = shell_leaves(domain=64, shells=2, thickness=0.1, seed=9)
    L = len(origins)
    return vkl.vdb_volume(vkl.Device("cuda"), np.full(L, 3), origins, np.ones(L),
                          packed_dense=[values * (1 + 0.25 * i) for i in range(count)], leaf_map=leaf_map,
                          compression=compression, background=[0.25] * count)


VOLUMES = {
    "float": lambda v: _dense(v, np.float32, 5), "uchar": lambda v: _dense(v, np.uint8, 2),
    "short": lambda v: _dense(v, np.int16, 3), "ushort": lambda v: _dense(v, np.uint16, 2),
    "half": lambda v: _dense(v, np.float16, 4), "double": lambda v: _dense(v, np.float64, 3),
    "float bricked": lambda v: _dense(v, np.float32, 2, textureSampling=0),
    "vdb": lambda v: _sparse(v, 4), "vdb fp16": lambda v: _sparse(v, 2, compression="fp16"),
    "vdb fp8_blocks": lambda v: _sparse(v, 3, compression="fp8_blocks"), "vdb no map": lambda v: _sparse(v, 2, leaf_map=False),
}


@pytest.mark.parametrize("kind", sorted(VOLUMES))
def test_around_the_lines(vkl, kind):
    import torch
    vol = VOLUMES[kind](vkl)
    ids = list(range(vol.num_attributes()))[::-1] + [0]
    for n in ((1 << 18) - 1, (1 << 18) + 5, (1 << 19) - 3, (1 << 19) + 1):
        pts = orbit_camera_samples_torch(125, n // (125 * 37) + 1, 37, (-2, -2, -2), (62, 72, 52), seed=5)[:n].contiguous()
        for filt in (0, 100, 200):
            s = vkl.Sampler(vol, filter=filt)
            out = torch.full((n, len(ids)), -77.0, device="cuda")
            s.sample_m(pts, ids, out=out)
            for c, a in enumerate(ids):
                one = s.sample(pts, attr=a)
                np.testing.assert_array_equal(bits(out[:, c].cpu().numpy()), bits(one.cpu().numpy()))


def _time(f, reps=50):
    import torch
    best = 1e9
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        f()
        a.record()
        for _ in range(reps):
            f()
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b) / reps * 1e3)
    return best


@pytest.mark.parametrize("kind", ["double", "vdb"])
def test_few_points_cost_as_much_as_one_by_one(vkl, kind):
    """Tricubic, where a tile's CTA once worked through a few thousand points
    alone: 3.3 to 3.7 times the calls one by one, 0.9 with a thread per point."""
    import torch
    vol = VOLUMES[kind](vkl)
    vol.device.set_stream(torch.cuda.current_stream().cuda_stream)
    ids = list(range(vol.num_attributes()))
    n = 4099
    pts = orbit_camera_samples_torch(125, 1, 37, (0, 0, 0), (59, 69, 49), seed=5)[:n].contiguous()
    s = vkl.Sampler(vol, filter=200)
    out, one = torch.empty((n, len(ids)), device="cuda"), torch.empty(n, device="cuda")
    together = _time(lambda: s.sample_m(pts, ids, out=out))
    apart = _time(lambda: [s.sample(pts, attr=a, out=one) for a in ids])
    assert together < 2 * apart, (together, apart)
