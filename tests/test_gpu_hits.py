"""Radius batches answered in one walk (hits recorded by the counting pass)
against the oracle, and the calls' refusals."""
import ctypes

import numpy as np
import pytest

import kiddo_b200 as kb
import oracle
from helpers import assert_same_csr

pytestmark = pytest.mark.gpu

NAMES = {"sqeuclidean": kb.SquaredEuclidean, "manhattan": kb.Manhattan,
         "chebyshev": kb.Chebyshev}


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("metric", ["sqeuclidean", "manhattan", "chebyshev"])
@pytest.mark.parametrize("exclusive", [False, True])
def test_recorded_hits_match_the_oracle(dtype, metric, exclusive):
    """Rows of zero to all hits, leaves longer than one chunk (equal points),
    NaN rows; sorted and in traversal order."""
    import torch
    rng = np.random.default_rng(11)
    P = (np.round(rng.random((6_000, 3)) * 256) / 256).astype(dtype)
    P[1000:1100] = P[1000]
    Q = np.concatenate([rng.random((500, 3)), P[:200], P[1000:1001], P[:1] + 0.5 ** 7]).astype(dtype)
    Q[[7, 300]] = np.nan
    tree = kb.ImmutableKdTree.new_from_slice(P)
    ref = oracle.OracleTree.build(P)
    dq = torch.from_numpy(Q).cuda()
    for r in (0.0, 0.5 ** 9, 0.02, 0.2, 4.0):
        for srt in (True, False):
            b = tree.query(dq).with_engine("thread").within(NAMES[metric], r)
            b = b if srt else b.unsorted()
            b = b.exclusive_boundaries() if exclusive else b
            g = b.execute_gpu()
            assert_same_csr((g.offsets.cpu().numpy(), g.distances.cpu().numpy(),
                             g.items.cpu().numpy().view(np.uint32)),
                            ref.within(Q, r, metric=metric, exclusive=exclusive, sorted=srt),
                            f"r={r} sorted={srt}")


def test_more_hits_than_records_hold():
    """Every query hits every chunk of every leaf: more records than the handle
    keeps, so the filling call walks again."""
    import torch
    n, nq = 45_000, 800                    # 1,407+ chunks a query against 16 and 2^20 in all
    rng = np.random.default_rng(12)
    P = rng.random((n, 3)).astype(np.float32)
    Q = rng.random((nq, 3)).astype(np.float32)
    tree = kb.ImmutableKdTree.new_from_slice(P)
    g = tree.query(torch.from_numpy(Q).cuda()).with_engine("thread").within(
        kb.SquaredEuclidean, 4.0).unsorted().execute_gpu()
    off = g.offsets.cpu().numpy()
    assert (np.diff(off) == n).all()
    rows = [0, 399, nq - 1]
    o = oracle.OracleTree.build(P).within(Q[rows], 4.0, sorted=False)
    for j, i in enumerate(rows):
        a, b = int(off[i]), int(off[i + 1])
        assert np.array_equal(g.distances[a:b].cpu().numpy(), o[1][j * n:(j + 1) * n])
        assert np.array_equal(g.items[a:b].cpu().numpy().view(np.uint32), o[2][j * n:(j + 1) * n])


def test_handles_are_checked():
    import torch
    from kiddo_b200 import _capi as C
    L = C.lib()
    P = np.random.default_rng(1).random((500, 3)).astype(np.float32)
    tree = kb.ImmutableKdTree.new_from_slice(P).to_gpu()
    q = torch.from_numpy(P[:64]).cuda()
    d = tree.query(q).within(kb.SquaredEuclidean, 0.01)._desc(False)
    off = torch.empty(65, dtype=torch.int64, device="cuda")
    total, h = ctypes.c_uint64(), ctypes.c_void_p()
    vp = ctypes.c_void_p
    args = (tree._h, ctypes.byref(d), vp(q.data_ptr()))
    C.check(L.kgpu_query_radius_count_keep(*args, 64, vp(off.data_ptr()), ctypes.byref(total),
                                           ctypes.byref(h), None))
    assert total.value == int(off[-1].item()) > 0
    dist = torch.empty(total.value, device="cuda")
    items = torch.empty(total.value, dtype=torch.int32, device="cuda")
    out = (vp(dist.data_ptr()), vp(items.data_ptr()))
    fill = L.kgpu_query_radius_fill_kept
    assert fill(*args, 63, vp(off.data_ptr()), h, *out, None) == C.KGPU_EINVAL
    other = torch.cuda.Stream()
    assert fill(*args, 64, vp(off.data_ptr()), h, *out, vp(other.cuda_stream)) == C.KGPU_EINVAL
    assert fill(*args, 64, vp(off.data_ptr()), None, *out, None) == C.KGPU_EINVAL
    for _ in range(2):                      # a handle fills as often as asked
        dist.zero_()
        C.check(fill(*args, 64, vp(off.data_ptr()), h, *out, None))
        torch.cuda.synchronize()
        o = oracle.OracleTree.build(P).within(P[:64], 0.01)
        assert np.array_equal(dist.cpu().numpy(), o[1])
    C.check(L.kgpu_hits_free(h))
    hd = tree.query(P[:4]).within(kb.SquaredEuclidean, 0.01)._desc(True)
    assert L.kgpu_query_radius_count_keep(tree._h, ctypes.byref(hd), vp(q.data_ptr()), 4,
                                          vp(off.data_ptr()), ctypes.byref(total),
                                          ctypes.byref(h), None) == C.KGPU_EINVAL
