"""Filling from kept hits (kgpu_query_radius_fill_kept and its forest form) when
the caller's arguments do not belong together: refused, or held to the rows
and the outputs it was given.  And the right call, twice, against the oracle,
on the engine that keeps records."""
import ctypes

import numpy as np
import pytest

import kiddo_b200 as kb
import oracle

pytestmark = pytest.mark.gpu

VP = ctypes.c_void_p
NQ, GUARD = 800, 4096


class _Batch:
    """One radius batch over a tree, or over a forest of that tree and another."""

    def __init__(self, forest, trees, q, radius, srt):
        import torch
        from kiddo_b200 import _capi as C
        self.L, self.q, self.forest = C.lib(), q, forest
        target = trees[0] if forest is None else forest
        if forest is None:
            b = target.query(q).with_engine("thread").within(kb.SquaredEuclidean, radius)
            self.extra = ()
        else:
            self.of = torch.zeros(NQ, dtype=torch.int32, device="cuda")
            self.radii = torch.full((NQ,), radius, dtype=q.dtype, device="cuda")
            b = target.query(q, self.of, self.radii).with_engine("thread").within(
                kb.SquaredEuclidean, 0.0)
            self.extra = (VP(self.of.data_ptr()), VP(self.radii.data_ptr()))
        self.d = (b if srt else b.unsorted())._desc(False)
        self.h = target._h
        name = "kgpu_query_radius" if forest is None else "kgpu_forest_query_radius"
        self.fill_call = getattr(self.L, name + "_fill_kept")
        self.offsets = torch.empty(NQ + 1, dtype=torch.int64, device="cuda")
        total, self.hits = ctypes.c_uint64(), VP()
        C.check(getattr(self.L, name + "_count_keep")(
            self.h, ctypes.byref(self.d), VP(q.data_ptr()), *self.extra, NQ,
            VP(self.offsets.data_ptr()), ctypes.byref(total), ctypes.byref(self.hits), None))
        self.total = total.value

    def fill(self, offsets, handle=None):
        """Outputs of `total` entries with a guard of marks behind them."""
        import torch
        dist = torch.full((self.total + GUARD,), -7.0, dtype=self.q.dtype, device="cuda")
        items = torch.full((self.total + GUARD,), -7, dtype=torch.int32, device="cuda")
        st = self.fill_call(handle or self.h, ctypes.byref(self.d), VP(self.q.data_ptr()),
                            *self.extra, NQ, VP(offsets.data_ptr()), self.hits,
                            VP(dist.data_ptr()), VP(items.data_ptr()), None)
        torch.cuda.synchronize()
        return st, dist, items

    def free(self):
        self.L.kgpu_hits_free(self.hits)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("in_forest", [False, True])
@pytest.mark.parametrize("srt", [False, True])
def test_offsets_of_another_batch_stay_inside(dtype, in_forest, srt):
    import torch
    from kiddo_b200 import _capi as C
    rng = np.random.default_rng(8)
    P = rng.random((6_000, 3)).astype(dtype)
    Q = rng.random((NQ, 3)).astype(dtype)
    trees = [kb.GpuTree.build(torch.from_numpy(p).cuda()) for p in (P, P[:2_000])]
    forest = kb.Forest(trees) if in_forest else None
    q = torch.from_numpy(Q).cuda()
    small = _Batch(forest, trees, q, 0.01, srt)
    large = _Batch(forest, trees, q, 0.04, srt)
    try:
        assert 0 < small.total < large.total
        # rows of the larger batch run past the smaller one's outputs
        st, dist, items = small.fill(large.offsets)
        assert st == C.KGPU_OK
        assert (dist[small.total:] == -7.0).all() and (items[small.total:] == -7).all()
        # rows of the smaller batch are too short for the larger one's hits
        st, dist, items = large.fill(small.offsets)
        assert st == C.KGPU_OK
        assert (dist[small.total:] == -7.0).all() and (items[small.total:] == -7).all()
        # the handle of another tree or forest
        other = kb.Forest(trees) if in_forest else trees[1]
        assert small.fill(small.offsets, other._h)[0] == C.KGPU_EINVAL
        # the right call, as often as asked
        ref = oracle.OracleTree.build(P).within(Q, 0.01, sorted=srt)
        for _ in range(2):
            st, dist, items = small.fill(small.offsets)
            assert st == C.KGPU_OK
            assert np.array_equal(small.offsets.cpu().numpy(), ref[0].astype(np.int64))
            assert np.array_equal(dist[:small.total].cpu().numpy(), ref[1])
            assert np.array_equal(items[:small.total].cpu().numpy().view(np.uint32), ref[2])
            assert (dist[small.total:] == -7.0).all()
    finally:
        small.free()
        large.free()
