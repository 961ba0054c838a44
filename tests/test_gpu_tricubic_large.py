"""Tricubic sampling of values whose weighted sums overflow: the fused sums
would stay finite, or become infinite, where the sums as written end in an
infinity or NaN.  Values on both sides of the magnitude from which the kernels
take the sums as written (2^100), a large background alone, on every path
(direct through the atlas, bricked, sorted tiles, sparse), against the oracle."""
import numpy as np
import pytest

from openvkl_b200.fields import shell_leaves, uniform_points
from tests.conftest import bits

pytestmark = pytest.mark.gpu


def _values(shape, kind, seed):
    rng = np.random.default_rng(seed)
    v = rng.normal(size=shape)
    if kind == "huge":
        pick = rng.random(shape)
        big = rng.choice([5e37, -5e37, 2e37, -7e37, 1.2e37, 3.3e38, -3e38], size=shape)
        v = np.where(pick < 0.15, big, v * 1e36)
    elif kind == "line":
        v = v * 2.0 ** 100
    elif kind == "spots":
        v[rng.random(shape) < 0.004] = 6e37
        v[rng.random(shape) < 0.002] = np.inf
    return v.astype(np.float32)


@pytest.mark.parametrize("kind", ["huge", "line", "spots", "background"])
@pytest.mark.parametrize("texture", [1, 0])
def test_dense(vkl, oracle, kind, texture):
    import torch
    vox = _values((26, 30, 34), kind, 1)
    background = 6e37 if kind == "background" else 0.25
    dev = vkl.Device("cuda")
    dev.set_int("textureSampling", texture)
    vol = vkl.structured_regular(dev, vox, background=[background])
    ref = oracle.OracleVolume.dense_volume(vox, background=background)
    s = vkl.Sampler(vol, filter=200, gradient_filter=200)
    for n in (5000, (1 << 20) + 5):
        pts = uniform_points(n, (-2, -2, -2), (35, 31, 27), seed=4)
        tp = torch.from_numpy(pts).cuda()
        np.testing.assert_array_equal(bits(s.sample(tp).cpu().numpy()), bits(ref.sample_parallel(pts, filter=200)))
        np.testing.assert_array_equal(bits(s.gradient(tp).cpu().numpy()), bits(ref.gradient_parallel(pts, filter=200)))


@pytest.mark.parametrize("kind", ["huge", "line"])
def test_double_and_sparse(vkl, oracle, kind):
    pts = uniform_points(20000, (-2, -2, -2), (35, 31, 27), seed=4)
    vox = _values((26, 30, 34), kind, 2).astype(np.float64)
    vox[::5, ::7, ::3] = 4e38  # beyond float
    vol = vkl.structured_regular(vkl.Device("cuda"), vox, background=[0.5])
    ref = oracle.OracleVolume.dense_volume(vox, background=0.5)
    s = vkl.Sampler(vol, filter=200, gradient_filter=200)
    np.testing.assert_array_equal(bits(s.sample(pts)), bits(ref.sample(pts, filter=200)))
    np.testing.assert_array_equal(bits(s.gradient(pts)), bits(ref.gradient(pts, filter=200)))
    origins, values = shell_leaves(domain=64, shells=2, thickness=0.1, seed=9)
    values = _values(values.shape, kind, 3)
    L = len(origins)
    vol = vkl.vdb_volume(vkl.Device("cuda"), np.full(L, 3), origins, np.ones(L), packed_dense=values, background=[0.5])
    ref = oracle.OracleVolume.vdb_volume(np.full(L, 3), origins, np.ones(L), values, background=0.5)
    pts = uniform_points(20000, (0, 0, 0), (64, 64, 64), seed=5)
    s = vkl.Sampler(vol, filter=200, gradient_filter=200)
    np.testing.assert_array_equal(bits(s.sample(pts)), bits(ref.sample(pts, filter=200)))
    np.testing.assert_array_equal(bits(s.gradient(pts)), bits(ref.gradient(pts, filter=200)))
