"""Tricubic floats without a texture atlas take the sorted tiles from 3 * 2^17
points: the bits of smaller calls around that line, and calls below the other
kinds' line (2^20) no slower than one above it."""
import numpy as np
import pytest

from openvkl_b200.fields import orbit_camera_samples_torch, sinusoid_field, sinusoid_field_torch
from tests.conftest import bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(3 << 17) - 1, 3 << 17, (3 << 17) + 1029])
def test_around_the_line(vkl, n):
    import torch
    dev = vkl.Device("cuda")
    dev.set_int("textureSampling", 0)
    vol = vkl.structured_regular(dev, sinusoid_field((70, 61, 83), seed=3), background=[0.5])
    pts = orbit_camera_samples_torch(125, n // (125 * 37) + 1, 37, (0, 0, 0), (69, 60, 82), seed=5)[:n].contiguous()
    s = vkl.Sampler(vol, filter=200, gradient_filter=200)
    for call in (s.sample, s.gradient):
        parts = [call(pts[i:i + 100003].contiguous()) for i in range(0, n, 100003)]
        np.testing.assert_array_equal(bits(call(pts).cpu().numpy()), bits(torch.cat(parts).cpu().numpy()))


def test_time_below_the_general_line(vkl):
    import torch
    dev = vkl.Device("cuda")
    dev.set_int("textureSampling", 0)
    dev.set_stream(torch.cuda.current_stream().cuda_stream)
    vol = vkl.structured_regular(dev, sinusoid_field_torch((300, 280, 310), seed=1), background=[0.0], shared=True)
    s = vkl.Sampler(vol, filter=200)
    times = []
    for n in (1000000, (1 << 20) + 1):
        pts = orbit_camera_samples_torch(256, n // (256 * 200) + 1, 200, (0, 0, 0), (299, 279, 309), seed=5)[:n].contiguous()
        out = torch.empty(n, device="cuda")
        best = 1e9
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(10):
                s.sample(pts, out=out)
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        times.append(best)
    assert times[0] < 1.06 * times[1], times
