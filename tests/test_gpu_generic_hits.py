"""The batched hit kernel of any voxel type and filter, in its two forms (few
rays; many rays and few isovalues): the bits of the float kernel where both
compute the same values, and for few rays its time in proportion (1.0 of the
float kernel's where the march's registers spill, 0.8 where they do not)."""
import numpy as np
import pytest

from openvkl_b200.fields import random_rays, sinusoid_field
from tests.conftest import bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,count", [(4000, 40), (50001, 2), (50001, 5)])
def test_bytes_against_float(vkl, n, count):
    import torch
    dims = (128, 120, 110)
    vox = (sinusoid_field(dims, seed=1) * 25 + 128).round().clip(0, 255)
    dev = vkl.Device("cuda")
    dev.set_stream(torch.cuda.current_stream().cuda_stream)
    rays = [torch.from_numpy(np.ascontiguousarray(r)).cuda() for r in random_rays(n, (0, 0, 0), dims, seed=7)]
    values = [20.5 + 200 / count * i for i in range(count)]
    found, times = [], []
    for dtype in (np.float32, np.uint8):
        vol = vkl.structured_regular(dev, vox.astype(dtype), background=[0.0])
        ctx = vkl.HitIteratorContext(vkl.Sampler(vol, filter=100), values)
        best = 1e9
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            hits, counts = ctx.iterate_n(*rays, max_per_ray=64)
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        counts = counts.cpu().numpy()
        hits = hits.cpu().numpy()
        hits[np.arange(64)[None, :] >= counts[:, None]] = 0
        found.append((hits, counts))
        times.append(best)
    np.testing.assert_array_equal(found[0][1], found[1][1])
    np.testing.assert_array_equal(bits(found[0][0]), bits(found[1][0]))
    assert found[0][1].sum() > n
    if n == 4000:
        assert times[1] < 0.9 * times[0], times
