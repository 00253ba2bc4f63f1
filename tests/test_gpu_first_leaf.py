"""The thread engine's first leaf (lists of up to 16 filled from one sorted
leaf) where its words cannot tell distances apart, against the oracle."""
import numpy as np
import pytest

import kiddo_b200 as kb
import oracle
from helpers import assert_same_fixed

pytestmark = pytest.mark.gpu


def _clouds(rng):
    x = 1.0 + np.arange(31) * 2.0 ** -23     # distances from 0 differ in their last bits
    yield "last bits", np.stack([rng.permutation(x), np.zeros(31), np.zeros(31)], 1)
    yield "equal", np.repeat(rng.random((4, 3)), 8, axis=0)[:30]
    yield "some equal", np.round(rng.random((32, 3)) * 4) / 4
    yield "spread", rng.random((32, 3))
    yield "short", rng.random((9, 3))
    yield "two leaves", np.round(rng.random((45, 3)) * 64) / 64
    yield "long leaf", np.repeat(rng.random((2, 3)), 40, axis=0)
    yield "many", np.round(rng.random((3000, 3)) * 32) / 32


@pytest.mark.parametrize("k", [1, 2, 7, 8, 15, 16, 17])
def test_first_leaf_lists(k):
    import torch
    rng = np.random.default_rng(k)
    for name, P in _clouds(rng):
        P = np.ascontiguousarray(P.astype(np.float32))
        Q = np.concatenate([np.zeros((40, 3)), rng.random((60, 3)), P[:20]]).astype(np.float32)
        tree = kb.ImmutableKdTree.new_from_slice(P)
        ref = oracle.OracleTree.build(P)
        dq = torch.from_numpy(Q).cuda()
        for radius in (np.inf, 0.3):
            for srt in (True, False):
                b = tree.query(dq).with_engine("thread").nearest_n(kb.SquaredEuclidean, k)
                if radius != np.inf:
                    b = b.within(radius)
                b = b if srt else b.unsorted()
                g = b.execute_gpu()
                assert_same_fixed(g.distances.cpu().numpy(), g.items.cpu().numpy().view(np.uint32),
                                  g.counts.cpu().numpy(),
                                  *ref.nearest_n(Q, k, radius=radius, sorted=srt),
                                  f"{name} k={k} r={radius} sorted={srt}")
