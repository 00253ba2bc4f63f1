"""Device construction at the sizes and value patterns where its two stages
change hands or their slow paths run: the host builder's bytes throughout."""
import numpy as np
import pytest

from test_gpu_build import _device_vs_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2047, 2048, 2049, 4096, 4097, 8191, 65_537, 300_001])
@pytest.mark.parametrize("dtype,dims", [(np.float32, 3), (np.float64, 3), (np.float32, 2),
                                        (np.float64, 4)])
def test_sizes_beside_a_blocks_share(dtype, dims, n):
    rng = np.random.default_rng(n + dims)
    _device_vs_host((rng.random((n, dims)) - 0.5).astype(dtype))


def _patterns(rng, n):
    u = rng.random((n, 3))
    yield "outliers", np.where(rng.random((n, 3)) < 1e-4, u * 1e30 - 5e29, u)
    yield "octaves", np.exp(u * 80.0 - 40.0) * np.where(rng.random((n, 3)) < 0.5, -1.0, 1.0)
    yield "one_axis_two_values", np.stack([u[:, 0], np.round(u[:, 1]) + 1.0, u[:, 2]], 1)
    # whole nodes of one value on an axis: gaps that stay long
    yield "coarse", np.round(u * 6) + 1.0 + np.where(rng.random((n, 3)) < 0.02, u * 1e-3, 0.0)
    yield "most_equal", np.where(rng.random((n, 3)) < 0.7, 0.25, u)
    yield "ends", np.where(rng.random((n, 3)) < 1e-3, np.inf, u)
    yield "negative", -np.exp(u * 10.0)
    yield "mostly_smallest", np.where(rng.random((n, 1)) < 0.6, 0.125, u + 1.0)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_value_patterns(dtype):
    """Wide and narrow key ranges, long runs of equal values at the pivot and
    below it, infinities; leaves above the limit are refused on both sides."""
    import kiddo_b200 as kb
    rng = np.random.default_rng(5)
    compared = 0
    for name, P in _patterns(rng, 200_000):
        P = np.ascontiguousarray(P.astype(dtype))
        try:
            kb.ImmutableKdTree.new_from_slice(P)
        except kb.KiddoGpuError:
            with pytest.raises(kb.KiddoGpuError):
                _device_vs_host(P)
            continue
        _device_vs_host(P)
        compared += 1
    assert compared >= 5
