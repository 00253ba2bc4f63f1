"""best_n_within where leaves are left out by their least item: items rising
and falling in iteration order, equal items, lists that never fill; every
engine and list kind, bit for bit with the oracle and its traversal counters."""
import numpy as np
import pytest

import kiddo_b200 as kb
import oracle
from helpers import assert_same_fixed

pytestmark = pytest.mark.gpu


def _items(kind, n, rng):
    if kind == "rising":
        return np.arange(n, dtype=np.uint32)
    if kind == "falling":
        return np.arange(n, dtype=np.uint32)[::-1].copy()
    if kind == "equal":
        return np.full(n, 7, dtype=np.uint32)
    if kind == "few":
        return rng.integers(0, 5, n).astype(np.uint32)
    return (rng.permutation(n).astype(np.uint32) + np.uint32(2 ** 32 - 1 - n))  # up to 2^32 - 2


@pytest.mark.parametrize("dtype,dims", [(np.float32, 3), (np.float64, 3), (np.float32, 2),
                                        (np.float64, 1)])
@pytest.mark.parametrize("kind", ["rising", "falling", "equal", "few", "high"])
def test_best_n(dtype, dims, kind):
    import torch
    rng = np.random.default_rng(21)
    n = 4_000
    P = (np.round(rng.random((n, dims)) * 64) / 64 if dims == 3 else
         rng.random((n, dims))).astype(dtype)
    it = _items(kind, n, rng)
    Q = np.concatenate([rng.random((150, dims)), P[:50]]).astype(dtype)
    tree = kb.ImmutableKdTree.new_from_entries(it, P)
    ref = oracle.OracleTree.build(P, it)
    dev = kb.GpuTree.build(torch.from_numpy(P).cuda(), torch.from_numpy(it.view(np.int32)).cuda())
    dq = torch.from_numpy(Q).cuda()
    for k in (1, 5, 32, 33, 300):
        if dims == 1 and k > 256:
            continue
        for r in (0.003, 0.09, 9.0):
            want = ref.best_n_within(Q, r, k)
            for engine in (None, "thread", "warp"):
                for t in (tree, dev):
                    b = t.query(dq).with_engine(engine).best_n_within(kb.SquaredEuclidean, r, k)
                    g = b.execute_gpu()
                    assert_same_fixed(g.distances.cpu().numpy(),
                                      g.items.cpu().numpy().view(np.uint32),
                                      g.counts.cpu().numpy(), *want,
                                      f"{kind} k={k} r={r} {engine}")
