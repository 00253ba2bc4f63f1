"""What a radius batch holds between counting and filling: nothing after the
handle is freed, and nothing that the caller's outputs need."""
import ctypes

import numpy as np
import pytest

import kiddo_b200 as kb
import oracle
from helpers import assert_same_csr
from kiddo_b200 import _capi as C

pytestmark = pytest.mark.gpu

VP = ctypes.c_void_p


def _count_keep(tree, q, radius):
    import torch
    d = tree.query(q).with_engine("thread").within(kb.SquaredEuclidean, radius).unsorted()._desc(False)
    off = torch.empty(len(q) + 1, dtype=torch.int64, device="cuda")
    total, hits = ctypes.c_uint64(), VP()
    C.check(C.lib().kgpu_query_radius_count_keep(
        tree._h, ctypes.byref(d), VP(q.data_ptr()), len(q), VP(off.data_ptr()),
        ctypes.byref(total), ctypes.byref(hits), None))
    torch.cuda.synchronize()
    return hits, total.value


def test_a_handle_gives_everything_back():
    import torch
    rng = np.random.default_rng(12)
    n, nq = 45_000, 800                        # 1,407+ chunks a query against 16 and 2^20 in all
    tree = kb.GpuTree.build(torch.from_numpy(rng.random((n, 3)).astype(np.float32)).cuda())
    q = torch.from_numpy(rng.random((nq, 3)).astype(np.float32)).cuda()
    torch.cuda.synchronize()
    before = C.scratch_stats()[0]
    for radius in (0.001, 4.0):                # records that fit, and that do not
        hits, total = _count_keep(tree, q, radius)
        assert total == n * nq if radius == 4.0 else total > 0
        held = C.scratch_stats()[0] - before
        assert 20 << 20 < held < 24 << 20      # 2^20 and 16 a query, 20 bytes each
        C.lib().kgpu_hits_free(hits)
        torch.cuda.synchronize()
        assert C.scratch_stats()[0] == before


@pytest.mark.parametrize("in_forest", [False, True])
@pytest.mark.parametrize("srt", [False, True])
def test_outputs_come_before_records(monkeypatch, in_forest, srt):
    """Where the outputs cannot be allocated beside the records, these go and the
    batch is walked again, with the same rows."""
    import torch
    rng = np.random.default_rng(13)
    P = rng.random((8_000, 3)).astype(np.float32)
    Q = rng.random((600, 3)).astype(np.float32)
    ref = oracle.OracleTree.build(P).within(Q, 0.01, sorted=srt)
    tree = kb.GpuTree.build(torch.from_numpy(P).cuda())
    q = torch.from_numpy(Q).cuda()
    if in_forest:
        of = torch.zeros(600, dtype=torch.int32, device="cuda")
        b = kb.Forest([tree]).query(q, of, torch.full((600,), 0.01, device="cuda"))
    else:
        b = tree.query(q)
    b = b.with_engine("thread").within(kb.SquaredEuclidean, 0.01)
    b = b if srt else b.unsorted()
    real, used = torch.empty, []

    def empty(*a, **k):
        if a == (len(ref[1]),):
            used.append(C.scratch_stats()[0])
            if len(used) == 1:
                raise torch.OutOfMemoryError("no room")
        return real(*a, **k)

    monkeypatch.setattr(torch, "empty", empty)
    g = b.execute_gpu()
    monkeypatch.undo()
    assert len(used) == 3 and used[1] + (20 << 20) < used[0]  # the records had gone
    assert_same_csr((g.offsets.cpu().numpy(), g.distances.cpu().numpy(),
                     g.items.cpu().numpy().view(np.uint32)), ref, "after the retry")
