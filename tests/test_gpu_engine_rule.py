"""The default engine of a batch (by family, list length and batch size)
against the thread engine asked for by name: the same bytes on either side of
the rule's lines, for every family and option it reads."""
import numpy as np
import pytest

import kiddo_b200 as kb

pytestmark = pytest.mark.gpu

SE, MAN, CHEB = kb.SquaredEuclidean, kb.Manhattan, kb.Chebyshev


def _same(a, b, label):
    for f in ("offsets", "distances", "items", "counts"):
        x, y = getattr(a, f, None), getattr(b, f, None)
        if x is None:
            assert y is None
            continue
        x, y = x.cpu().numpy(), y.cpu().numpy()
        assert x.shape == y.shape, f"{label}: {f}"
        assert x.tobytes() == y.tobytes(), f"{label}: {f} differs"


def _families(dtype, dims, r):
    box = np.ones(dims)
    f64 = dtype == np.float64
    return {
        "one": (28672, lambda b: b.nearest_one(SE)),
        "one_manhattan": (28672, lambda b: b.nearest_one(MAN)),
        "n5": (36608, lambda b: b.nearest_n(SE, 5)),
        "n16_unsorted": (57344 if f64 else 45056, lambda b: b.nearest_n(CHEB, 16).unsorted()),
        "n32_within_excl": (57344 if f64 else 49152,
                            lambda b: b.nearest_n(SE, 32).within(r).exclusive_boundaries()),
        "n40": (36864, lambda b: b.nearest_n(SE, 40)),
        "best7": (40960, lambda b: b.best_n_within(SE, r, 7)),
        "within": (16384 if dims == 3 else 40960, lambda b: b.within(SE, r)),
        "within_unsorted_excl": (16384 if dims == 3 else 40960,
                                 lambda b: b.within(MAN, r).unsorted().exclusive_boundaries()),
        "periodic_n9": ((22528 if f64 else 28672) + 3456,
                        lambda b: b.periodic_boundary_condition(box).nearest_n(SE, 9)),
        "periodic_within": (18432 if f64 else 24576,
                            lambda b: b.periodic_boundary_condition(box).within(SE, r)),
    }


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("dims", [2, 3])
def test_default_engine_gives_the_thread_engines_bytes(dtype, dims):
    """Batches of 1, 37, the last below and the first above each line, NaN
    query rows among them."""
    import torch
    rng = np.random.default_rng(3)
    P = rng.random((5_001, dims)).astype(dtype)
    P[100:140] = P[100]                       # equal distances
    tree = kb.ImmutableKdTree.new_from_slice(P)
    for name, (line, make) in _families(dtype, dims, 2e-3 if dims == 3 else 4e-4).items():
        Q = rng.random((line + 1, dims)).astype(dtype)
        Q[5::1009] = P[(np.arange(len(Q[5::1009])) * 7) % len(P)]
        Q[11::4001] = np.nan
        dq = torch.from_numpy(Q).cuda()
        for nq in (1, 37, line - 1, line + 1):
            q = dq[:nq]
            _same(make(tree.query(q)).execute_gpu(),
                  make(tree.query(q).with_engine("thread")).execute_gpu(),
                  f"{name} nq={nq}")


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_nearest_one_beside_nan_points(dtype):
    """A NaN coordinate among a leaf's points hides no other point from the
    warp engine, which small batches take."""
    import torch
    rng = np.random.default_rng(4)
    P = rng.random((25, 3)).astype(dtype)
    P[[3, 16, 17], [0, 1, 2]] = np.nan
    tree = kb.ImmutableKdTree.new_from_slice(P)
    dq = torch.from_numpy(rng.random((64, 3)).astype(dtype)).cuda()
    for make in (lambda b: b.nearest_one(SE), lambda b: b.nearest_n(SE, 4)):
        _same(make(tree.query(dq)).execute_gpu(),
              make(tree.query(dq).with_engine("thread")).execute_gpu(), "nan points")
