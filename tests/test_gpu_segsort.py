"""Sorted radius rows at the edges of the segment sort's classes (one lane, one
warp, blocks of 128 and 512 threads, merged runs), against the oracle."""
import numpy as np
import pytest

import kiddo_b200 as kb
import oracle
from helpers import assert_same_csr

pytestmark = pytest.mark.gpu

EDGES = [1, 8, 32, 64, 128, 256, 512, 1024, 2048, 4096, 8192, 16384, 32768]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_rows_at_class_edges(dtype):
    """Rows of edge - 1, edge, edge + 1 hits (and an empty and a full one) of
    one point set with many equal distances, one radius per query."""
    import torch
    rng = np.random.default_rng(17)
    n = 40_000
    # coarse coordinates: equal distances throughout, none shared by many points
    P = (np.round(rng.random((n, 3)) * 512) / 512).astype(dtype)
    tree = kb.ImmutableKdTree.new_from_slice(P)
    ref = oracle.OracleTree.build(P)
    q = np.array([0.25, 0.5, 0.125], dtype=dtype)
    d = np.sort(oracle.scan_dists(P, q, "sqeuclidean"))
    assert (np.diff(d) == 0).any()
    radii = [0.0, d[-1]]
    for e in EDGES:
        radii += [d[m - 1] for m in (e - 1, e, e + 1) if m >= 1]
    radii = np.asarray(radii, dtype=dtype)
    Q = np.broadcast_to(q, (len(radii), 3)).copy()
    dev = torch.from_numpy(Q).cuda()
    of = torch.zeros(len(Q), dtype=torch.int32, device="cuda")
    g = kb.Forest([tree]).query(dev, of, torch.from_numpy(radii).cuda()).within(
        kb.SquaredEuclidean, 0.0).execute_gpu()
    o = ref.within(Q, radii)
    assert_same_csr((g.offsets.cpu().numpy(), g.distances.cpu().numpy(),
                     g.items.cpu().numpy().view(np.uint32)), o)
