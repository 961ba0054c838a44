"""Batched intervals of dense volumes whose rays cross few cells or whose
contexts have many value ranges: against the oracle, with cells of every level,
and in a time that does not grow with the ranges where a ray has one cell."""
import ctypes

import numpy as np
import pytest

from openvkl_b200.fields import random_rays, sinusoid_field
from tests.conftest import bits

pytestmark = pytest.mark.gpu


def _ranges(lo, hi, count):
    e = np.linspace(lo, hi, 2 * count + 1, dtype=np.float32)
    return np.stack([e[0:-1:2], e[1::2]], 1)


@pytest.mark.parametrize("dims,hint,count", [((600, 20, 140), 0.3, 40), ((600, 20, 140), 0.0, 3), ((4200, 9, 6), 0.0, 33),
                                             ((130, 40, 30), 0.3, 1), ((70, 60, 50), 0.5, 5), ((40, 40, 40), 1.0, 3)])
def test_few_cells_many_ranges(vkl, device, oracle, dims, hint, count):
    vox = sinusoid_field(dims, seed=5)
    ref = oracle.OracleVolume.dense_volume(vox)
    b = ref.info()["bounds"]
    o, d, t = random_rays(777, b[:3], b[3:], seed=3)
    vr = _ranges(float(vox.min()), float(vox.max()), count)
    ctx = vkl.IntervalIteratorContext(vkl.Sampler(vkl.structured_regular(device, vox)), value_ranges=vr, hint=hint)
    want, wcnt = ref.intervals(o, d, t, value_ranges=vr, hint=hint, max_intervals=128)
    got, cnt = ctx.iterate_n(o, d, t, max_per_ray=128)
    np.testing.assert_array_equal(cnt, wcnt)
    for r in range(len(cnt)):
        k = min(int(cnt[r]), 128)
        np.testing.assert_array_equal(bits(got[r, :k]), bits(want[r, :k]), err_msg=f"ray {r}")


def test_time_with_many_ranges(vkl):
    """One cell per ray: 40 ranges took 3.1 times as long as one where the
    steps past the rays' ends went through all of them, 1.0 where not."""
    import torch
    dims = (128, 120, 110)
    vox = sinusoid_field(dims, seed=5)
    dev = vkl.Device("cuda")
    dev.set_stream(torch.cuda.current_stream().cuda_stream)
    s = vkl.Sampler(vkl.structured_regular(dev, vox))
    n = 400000
    rays = [torch.from_numpy(np.ascontiguousarray(r)).cuda() for r in random_rays(n, (0, 0, 0), dims, seed=7)]
    out, cnt = torch.zeros((n, 8, 5), device="cuda"), torch.zeros(n, dtype=torch.int32, device="cuda")
    times = []
    for count in (1, 40):
        ctx = vkl.IntervalIteratorContext(s, value_ranges=_ranges(float(vox.min()), float(vox.max()), count), hint=0.0)
        best = 1e9
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(10):
                ctx._call(ctx.lib.vklIterateIntervalsN, ctypes.byref(ctx.h), n, rays[0].data_ptr(), rays[1].data_ptr(),
                          rays[2].data_ptr(), 8, out.data_ptr(), cnt.data_ptr())
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        times.append(best)
    assert times[1] < 1.8 * times[0], times


@pytest.mark.parametrize("count", [1, 2, 3, 33])
def test_ranges_that_nothing_overlaps(vkl, device, oracle, count):
    """NaN ranges overlap nothing, not even cells that hold both infinities."""
    vox = sinusoid_field((40, 33, 26), seed=5)
    vox[::3, ::5, ::4] = np.inf
    vox[1::3, ::5, ::4] = -np.inf
    ref = oracle.OracleVolume.dense_volume(vox)
    b = ref.info()["bounds"]
    o, d, t = random_rays(300, b[:3], b[3:], seed=3)
    smp = vkl.Sampler(vkl.structured_regular(device, vox))
    for vr in (np.full((count, 2), np.nan, np.float32), np.array([[np.nan, np.nan]] * (count - 1) + [[0, 0.5]], np.float32)):
        ctx = vkl.IntervalIteratorContext(smp, value_ranges=vr)
        want, wcnt = ref.intervals(o, d, t, value_ranges=vr, max_intervals=64)
        got, cnt = ctx.iterate_n(o, d, t, max_per_ray=64)
        np.testing.assert_array_equal(cnt, wcnt)
        for r in range(len(cnt)):
            np.testing.assert_array_equal(bits(got[r, :cnt[r]]), bits(want[r, :cnt[r]]), err_msg=f"ray {r}")
