"""Device construction where nodes do not fit a block's share when the last
levels begin: shares that are full (n at a power of two) and run over by a point
or two, and many equal values.  The host builder's bytes, and only the nodes
that do not fit go through more level passes."""
import numpy as np
import pytest

import kiddo_b200 as kb
from test_gpu_build import _device_vs_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("dims", [1, 2, 3, 4])
@pytest.mark.parametrize("n", [65_536, 262_144, 262_143])
def test_full_shares_match_host(dtype, dims, n):
    # coordinates of 1/4096: every top pivot moves by some points
    P = np.round(np.random.default_rng(n + dims).random((n, dims)) * 4096) / 4096
    if dims == 1:
        P = P + np.random.default_rng(1).random((n, 1))  # 64 equal values a leaf at most
    _device_vs_host(np.ascontiguousarray(P.astype(dtype)))


@pytest.mark.parametrize("dims", [1, 2, 3])
def test_random_power_of_two(dims):
    _device_vs_host(np.random.default_rng(dims).random((1 << 20, dims)).astype(np.float32))


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_axis_of_one_value(dtype):
    """Every second level splits nothing, so nodes pass the share by far."""
    rng = np.random.default_rng(9)
    P = rng.random((150_000, 3))
    P[:, 1] = 0.0
    _device_vs_host(np.ascontiguousarray(P.astype(dtype)))
    P[:, 1] = np.where(rng.random(len(P)) < 0.6, 0.0, P[:, 0])
    _device_vs_host(np.ascontiguousarray(P.astype(dtype)))


def test_few_launches_more():
    """One more level for the nodes that run over: a list, five passes, the last
    levels and the leaf tables again (12 launches or so), not all of the
    remaining levels for every node."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(3)

    def launches(n):
        p = torch.rand((n, 2), generator=g, device="cuda")
        kb.GpuTree.build(p)
        n0 = kb.launch_count()
        kb.GpuTree.build(p)
        return kb.launch_count() - n0

    assert launches(1 << 22) <= launches(4_000_000) + 20
