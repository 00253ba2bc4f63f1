"""Periodic nearest_n batches whose listed rows (those the box's faces can change)
number few or many: the warp engine answers few of them, threads many, and the
device decides by their number.  Against the oracle's periodic walk and against
the thread engine asked for by name, bit for bit."""
import numpy as np
import pytest

import kiddo_b200 as kb
import oracle
from helpers import assert_same_fixed

pytestmark = pytest.mark.gpu

SE = kb.SquaredEuclidean
NQ = 140_000  # above the batch size from which the device is asked


def _queries(rng, dims, near_faces):
    """`near_faces` of the queries within a list radius of a face."""
    q = 0.4 + 0.2 * rng.random((NQ, dims))
    rows = rng.permutation(NQ)[:near_faces]
    q[rows, rng.integers(0, dims, near_faces)] = rng.random(near_faces) * 0.002
    return q


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("k", [1, 8, 32])
def test_few_and_many_listed_rows(dtype, dims, k):
    import torch
    rng = np.random.default_rng(dims * 10 + k)
    P = rng.random((60_000, dims)).astype(dtype)
    P[P >= 1.0] = 0.0
    P[500:540] = P[500]                         # equal distances
    box = np.ones(dims, dtype=dtype)
    tree = kb.ImmutableKdTree.new_from_slice(P)
    ref = oracle.OracleTree.build(P)
    line = 28672 + 576 * k
    for near in (0, 1, line - 1, line, line + 1, 90_000):
        Q = _queries(rng, dims, near).astype(dtype)
        dq = torch.from_numpy(Q).cuda()
        a, b = [[x.cpu().numpy() for x in (r.distances, r.items.view(torch.int32), r.counts)]
                for r in (tree.query(dq).with_engine(e).periodic_boundary_condition(box)
                          .nearest_n(SE, k).execute_gpu() for e in (None, "thread"))]
        for x, y in zip(a, b):
            assert x.tobytes() == y.tobytes(), f"near={near}"
        rows = np.sort(rng.choice(NQ, 4_000, replace=False))
        assert_same_fixed(a[0][rows], a[1][rows].view(np.uint32), a[2][rows],
                          *ref.periodic_nearest_n(Q[rows], box, k), f"near={near}")


def test_batches_that_are_not_asked():
    """Below 131,072 queries the rows go to warps, whatever their number."""
    import torch
    rng = np.random.default_rng(4)
    P = rng.random((900, 3))                    # so few points that most rows are listed
    Q = rng.random((131_071, 3))
    box = np.ones(3)
    tree = kb.ImmutableKdTree.new_from_slice(P)
    ref = oracle.OracleTree.build(P)
    rows = np.arange(0, len(Q), 37)
    for nq in (70_000, 131_071):
        g = tree.query(torch.from_numpy(Q[:nq]).cuda()).periodic_boundary_condition(
            box).nearest_n(SE, 12).execute_gpu()
        r = rows[rows < nq]
        assert_same_fixed(g.distances.cpu().numpy()[r], g.items.cpu().numpy().view(np.uint32)[r],
                          g.counts.cpu().numpy()[r], *ref.periodic_nearest_n(Q[r], box, 12), "warps")


def test_one_launch_more_where_the_device_decides():
    import torch
    rng = np.random.default_rng(5)
    tree = kb.ImmutableKdTree.new_from_slice(rng.random((50_000, 3)))
    q = torch.from_numpy(rng.random((131_072, 3))).cuda()

    def launches(nq):
        n0 = kb.launch_count()
        tree.query(q[:nq]).with_spatial_order(False).periodic_boundary_condition(
            np.ones(3)).nearest_n(SE, 8).execute_gpu()
        torch.cuda.synchronize()
        return kb.launch_count() - n0

    launches(131_072)                           # the tree's bounds are measured once
    assert launches(131_071) == 3
    assert launches(131_072) == 4
