"""A commit that finds memory for its voxels but not for their texture atlases
goes without atlases, whatever the type and the number of attributes, and
memory that released volumes' atlases still hold makes room for it."""
import numpy as np
import pytest

from openvkl_b200.fields import sinusoid_field_torch, uniform_points_torch
from tests.conftest import bits

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _volume(vkl, dev, vox):
    return vkl.structured_regular(dev, vox, background=[0.5] * len(vox), shared=True)


def _free():
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("pooled", [False, True])
@pytest.mark.parametrize("dtype", ["uint8", "int16", "float16", "float32"])
def test_commit_without_room_for_atlases(vkl, dtype, pooled):
    import torch
    dims = (256, 256, 256)
    f = sinusoid_field_torch(dims, seed=1)
    one = (f * 25 + 100).round().to(getattr(torch, dtype)) if dtype in ("uint8", "int16") else f.to(getattr(torch, dtype))
    del f
    vox = [one, one.flip(0).contiguous(), one.flip(1).contiguous()]
    pts = uniform_points_torch(5000, (0, 0, 0), (255, 255, 255), seed=2)
    out = torch.empty((5000, 3), device="cuda")
    # what the commit needs without atlases, and every kernel loaded
    dev = vkl.Device("cuda")
    want = None
    for texture in (1, 0):
        dev.set_int("textureSampling", texture)
        before = _free()
        vol = _volume(vkl, dev, vox)
        need = before - _free()
        vkl.Sampler(vol, filter=100).sample_m(pts, [0, 1, 2], out=out)
        want = out.cpu().numpy()
        vol.release()
    dev.release()
    dev = vkl.Device("cuda")
    if pooled:  # the new device keeps two atlases of a volume released before
        _volume(vkl, dev, [v[:255].contiguous() for v in vox]).release()
        need -= 2 * one.numel() * one.element_size() - 8 * MB
    fill = torch.empty(_free() - need - 6 * MB, dtype=torch.uint8, device="cuda")
    try:
        vol = _volume(vkl, dev, vox)
        out.zero_()
        vkl.Sampler(vol, filter=100).sample_m(pts, [0, 1, 2], out=out)
        got = out.cpu().numpy()
    finally:
        del fill
        torch.cuda.empty_cache()
    np.testing.assert_array_equal(bits(got), bits(want))
