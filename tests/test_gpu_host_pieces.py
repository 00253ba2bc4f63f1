"""Host-buffer batches on either side of the sizes where they go through in one
piece, in two slots and in three: the rows of the same batch in device buffers
(and of the oracle), counts of rows that find nothing among them; several
threads at once."""
import threading

import numpy as np
import pytest

import kiddo_b200 as kb
import oracle
from helpers import assert_same_fixed

pytestmark = pytest.mark.gpu

SE = kb.SquaredEuclidean
CHUNK = 1 << 19   # of trees of up to 2^18 leaves
PIECE = 1 << 21   # no piece is larger


def _same(h, d, label):
    for f in ("distances", "items", "counts"):
        x, y = getattr(h, f), getattr(d, f).cpu().numpy()
        assert np.asarray(x).tobytes() == y.tobytes(), f"{label}: {f}"


@pytest.mark.parametrize("nq", [2 * CHUNK - 1, 2 * CHUNK, 2 * CHUNK + 1])
def test_around_the_first_pipelined_size(nq):
    import torch
    rng = np.random.default_rng(nq)
    P = rng.random((100_000, 3)).astype(np.float32)
    Q = rng.random((nq, 3)).astype(np.float32)
    Q[rng.choice(nq, 50, replace=False), 1] = np.nan
    Q[[0, nq - 1]] = np.nan
    tree = kb.ImmutableKdTree.new_from_slice(P)
    h = tree.query(Q).nearest_n(SE, 4).execute_gpu()
    _same(h, tree.query(torch.from_numpy(Q).cuda()).nearest_n(SE, 4).execute_gpu(), f"nq={nq}")
    rows = np.unique(np.concatenate([np.flatnonzero(np.isnan(Q[:, 1])),
                                     rng.choice(nq, 20_000, replace=False)]))
    assert_same_fixed(h.distances[rows], h.items[rows], h.counts[rows],
                      *oracle.OracleTree.build(P).nearest_n(Q[rows], 4), "oracle")


@pytest.mark.parametrize("nq", [PIECE, PIECE + 1, 2 * PIECE - 1])
def test_pieces_of_a_tree_of_many_leaves(nq):
    """More than 2^19 leaves: chunks of 2^21, and no piece above that."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(5)
    tree = kb.GpuTree.build(torch.rand((17_000_000, 3), generator=g, device="cuda"))
    q = torch.rand((nq, 3), generator=g, device="cuda")
    h = tree.query(q.cpu().numpy()).nearest_n(SE, 2).execute_gpu()
    _same(h, tree.query(q).nearest_n(SE, 2).execute_gpu(), f"nq={nq}")


def test_threads_at_once():
    import torch
    rng = np.random.default_rng(9)
    tree = kb.GpuTree.build(torch.from_numpy(rng.random((200_000, 3)).astype(np.float32)).cuda())
    torch.cuda.synchronize()
    Qs = [rng.random((n, 3)).astype(np.float32) for n in (700, 60_000, 300_000, 2 * CHUNK + 5)]
    out = [None] * len(Qs)

    def work(i):
        for _ in range(4):
            out[i] = tree.query(Qs[i]).nearest_n(SE, 4).execute_gpu()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(Qs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for Q, h in zip(Qs, out):
        _same(h, tree.query(torch.from_numpy(Q).cuda()).nearest_n(SE, 4).execute_gpu(), len(Q))
