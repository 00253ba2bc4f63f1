"""Device construction of values that leave long gaps beside the pivot: spread over
many exponents (no bin resolves them), or equal in large parts.  The host
builder's bytes, in a small multiple of what uniform points take."""
import time

import numpy as np
import pytest

import kiddo_b200 as kb
from test_gpu_build import _device_vs_host

pytestmark = pytest.mark.gpu

N = 1_200_000  # the gaps of the first levels pass the 131,072 points one block splits


def _case(name, n, rng):
    u = rng.random((n, 3))
    if name == "octaves":
        return np.exp(u * 80.0 - 40.0)
    if name == "signed_octaves":
        return np.exp(u * 80.0 - 40.0) * np.where(rng.random((n, 3)) < 0.5, -1.0, 1.0)
    if name == "infinities":  # a bracket from -inf to +inf has no bins
        return np.where(u < 0.45, -np.inf, np.where(u < 0.9, np.inf, u * 1e4)) + 0.0
    if name == "half_zero":
        u[:, 2] = np.where(rng.random(n) < 0.5, 0.0, u[:, 2])
        return u
    if name == "tenth_at_one_value":  # beside the middle of every axis
        return np.where(rng.random((n, 3)) < 0.1, 0.5, u)
    raise KeyError(name)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("name", ["octaves", "signed_octaves", "infinities", "half_zero",
                                  "tenth_at_one_value"])
def test_long_gaps_match_host(name, dtype):
    P = np.ascontiguousarray(_case(name, N, np.random.default_rng(6)).astype(dtype))
    try:
        kb.ImmutableKdTree.new_from_slice(P)
    except kb.KiddoGpuError:  # a leaf above the limit: refused on both sides
        with pytest.raises(kb.KiddoGpuError):
            _device_vs_host(P)
        return
    _device_vs_host(P)


def _milliseconds(p):
    import torch
    best = 1e9
    for _ in range(5):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        t = kb.GpuTree.build(p)
        torch.cuda.synchronize()
        best = min(best, 1e3 * (time.perf_counter() - t0))
        del t
    return best


def test_octaves_cost_a_small_multiple():
    """The levels run twice and wait for the host; one block per gap took 9 times
    the uniform cloud's time."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(3)
    u = torch.rand((8_000_000, 3), generator=g, device="cuda")
    assert _milliseconds(torch.exp(u * 80.0 - 40.0)) < 5.0 * _milliseconds(u)
