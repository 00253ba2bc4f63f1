"""The oracle tests whose small batches the default rule gives to the warp
engine, on each engine asked for by name: periodic families, periodic
lists of listed rows, forest radius batches with a radius per query, and
captured forest queries."""
import numpy as np
import pytest

import kiddo_b200 as kb
import test_gpu_forest
import test_gpu_periodic
import test_gpu_periodic_fast

pytestmark = pytest.mark.gpu


@pytest.fixture(params=["thread", "warp"])
def engine(request, monkeypatch):
    """Every query built inside the test asks for this engine."""
    real = kb.QueryBuilder.__init__

    def init(self, *a, **k):
        real(self, *a, **k)
        self.engine = request.param

    monkeypatch.setattr(kb.QueryBuilder, "__init__", init)
    b = kb.ImmutableKdTree.new_from_slice(np.zeros((4, 3))).query(np.zeros((1, 3)))
    assert b.engine == request.param
    return request.param


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("metric", ["sqeuclidean", "manhattan", "chebyshev", "minkowski3"])
def test_periodic_families(engine, dtype, dims, metric):
    test_gpu_periodic.test_periodic_families(dtype, dims, metric)


def test_periodic_small_trees(engine):
    test_gpu_periodic.test_periodic_non_unit_box_and_small_trees()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("dims", [2, 3])
def test_periodic_large_batches(engine, dtype, dims):
    test_gpu_periodic_fast.test_fast_path_matches_the_periodic_walk(dtype, dims, "sqeuclidean")


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_periodic_tie_heavy_grid(engine, dtype):
    test_gpu_periodic_fast.test_fast_path_on_a_tie_heavy_grid(dtype)


@pytest.mark.parametrize("srt", [True, False])
def test_forest_radii(engine, srt):
    test_gpu_forest.test_forest_radius_with_per_query_radii(srt)


def test_captured_forest(engine):
    test_gpu_forest.test_captured_graph_replays_forest_queries()
