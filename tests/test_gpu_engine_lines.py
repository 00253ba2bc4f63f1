"""f64 lists of 33 to 64 entries on either side of the batch sizes where they
change engines: the thread engine's bytes, and the oracle's rows."""
import numpy as np
import pytest

import kiddo_b200 as kb
import oracle
from helpers import assert_same_fixed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("k,line", [(33, 65_536), (36, 131_072), (44, None), (45, None)])
def test_long_f64_lists(dims, k, line):
    import torch
    rng = np.random.default_rng(k)
    P = rng.random((4_000, dims))
    P[100:160] = P[100]                        # equal distances
    tree = kb.ImmutableKdTree.new_from_slice(P)
    ref = oracle.OracleTree.build(P)
    sizes = (line - 1, line, line + 1) if line else (70_000,)
    Q = rng.random((sizes[-1], dims))
    Q[7::5000] = np.nan
    dq = torch.from_numpy(Q).cuda()
    for nq in sizes:
        a, b = [[x.cpu().numpy() for x in (r.distances, r.items.view(torch.int32), r.counts)]
                for r in (tree.query(dq[:nq]).with_engine(e).nearest_n(kb.SquaredEuclidean, k)
                          .execute_gpu() for e in (None, "thread"))]
        for x, y in zip(a, b):
            assert x.tobytes() == y.tobytes(), f"nq={nq}"
        rows = np.sort(rng.choice(nq, 1_000, replace=False))
        assert_same_fixed(a[0][rows], a[1][rows].view(np.uint32), a[2][rows],
                          *ref.nearest_n(Q[rows], k), f"nq={nq}")
