"""Device construction of points in raster order (voxel grids, images): the host
builder's bytes, in about the time that the same points take in random order."""
import time

import numpy as np
import pytest

import kiddo_b200 as kb
from test_gpu_build import _device_vs_host

pytestmark = pytest.mark.gpu


def _raster(shape, dtype, jitter=0.0):
    """Grid points, the first axis fastest."""
    axes = [np.arange(n, dtype=np.float64) for n in shape]
    m = np.meshgrid(*axes[::-1], indexing="ij")
    P = np.stack([a.ravel() for a in m[::-1]], 1)
    if jitter:
        P += jitter * np.random.default_rng(2).normal(size=P.shape)
    return np.ascontiguousarray(P.astype(dtype))


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape,jitter", [((64, 64, 64), 0.0), ((128, 128, 32), 0.3),
                                          ((512, 512), 0.0), ((1024, 256), 0.3),
                                          ((300, 77, 9), 0.0)])
def test_raster_matches_host(dtype, shape, jitter):
    _device_vs_host(_raster(shape, dtype, jitter))


def _milliseconds(p):
    import torch
    best = 1e9
    for _ in range(6):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        t = kb.GpuTree.build(p)
        torch.cuda.synchronize()
        best = min(best, 1e3 * (time.perf_counter() - t0))
        del t
    return best


@pytest.mark.parametrize("shape,jitter", [((256, 256, 256), 0.0), ((2048, 2048), 0.3)])
def test_raster_order_costs_no_more_than_random_order(shape, jitter):
    """Both sides build the same set of points; the raster took 19 and 12 times
    as long when samples were evenly spaced.  Twice leaves room for noise."""
    import torch
    p = torch.from_numpy(_raster(shape, np.float32, jitter)).cuda()
    g = torch.Generator(device="cuda").manual_seed(3)
    r = p[torch.randperm(len(p), device="cuda", generator=g)].contiguous()
    assert _milliseconds(p) < 2.0 * _milliseconds(r)
