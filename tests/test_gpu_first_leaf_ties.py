"""The thread engine's first leaf where distances of equal leading bits straddle
the list's end, and where fewer points than the list is long pass the radius."""
import numpy as np
import pytest

import kiddo_b200 as kb
import oracle
from helpers import assert_same_fixed

pytestmark = pytest.mark.gpu


def _leaf(rng, groups, per):
    """`groups` shells of `per` points each around the origin, whose distances in a
    shell differ in the last bits only (some not at all); in random order."""
    r = np.repeat(1.0 + rng.random(groups), per) + rng.integers(0, 4, groups * per) * 2.0 ** -23
    P = np.zeros((groups * per, 3))
    P[np.arange(len(P)), rng.integers(0, 3, len(P))] = r
    return rng.permutation(P.astype(np.float32), axis=0)


@pytest.mark.parametrize("k", [3, 4, 5, 8, 11, 15, 16])
@pytest.mark.parametrize("metric", ["sqeuclidean", "manhattan"])
def test_ties_at_the_end_of_the_list(k, metric):
    import torch
    rng = np.random.default_rng(k)
    m = {"sqeuclidean": kb.SquaredEuclidean, "manhattan": kb.Manhattan}[metric]
    for groups, per in ((1, 32), (2, 15), (4, 8), (7, 4), (10, 3), (16, 2), (6, 5)):
        for trial in range(3):
            P = _leaf(rng, groups, per)
            Q = np.concatenate([np.zeros((33, 3)), P[:5],
                                rng.normal(0, 1e-4, (20, 3))]).astype(np.float32)
            tree = kb.ImmutableKdTree.new_from_slice(P)
            ref = oracle.OracleTree.build(P)
            dq = torch.from_numpy(Q).cuda()
            cuts = np.sort(ref.nearest_n(Q[:1], len(P), metric=metric)[0][0])
            # all points; a radius that leaves k - 1, k, or one shell more
            for radius in (np.inf, cuts[min(k, len(P)) - 1], cuts[max(0, k - 2)],
                           cuts[min(len(P) - 1, k + per)]):
                for excl in (False, True):
                    b = tree.query(dq).with_engine("thread").nearest_n(m, k)
                    b = b.within(float(radius)) if radius != np.inf else b
                    b = b.exclusive_boundaries() if excl and radius != np.inf else b
                    g = b.execute_gpu()
                    assert_same_fixed(
                        g.distances.cpu().numpy(), g.items.cpu().numpy().view(np.uint32),
                        g.counts.cpu().numpy(),
                        *ref.nearest_n(Q, k, metric=metric, radius=float(radius),
                                       exclusive=bool(excl and radius != np.inf)),
                        f"{groups}x{per} k={k} r={radius} excl={excl}")
