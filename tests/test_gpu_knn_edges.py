"""Ranking and graph kernels at the sizes where their code changes: candidates a query around
a warp and past the shared list (equal distances make every tied row a candidate), neighbour
counts around 32, and components around the eight partial sums. The oracle's graph is exact,
so indices and distances are compared as bits."""

import numpy as np
import pytest

import kyto_b200 as K
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _equal(a, b):
    assert np.array_equal(a.indices, b.indices)
    assert np.array_equal(a.distances.view(np.uint32), b.distances.view(np.uint32))


@pytest.fixture(scope="module")
def ctx():
    return K.Context(0)


@pytest.mark.parametrize("k", [2, 16, 32, 33, 34, 64, 65, 129])
@pytest.mark.parametrize("values", [2, 4, 1000])
def test_ties_and_neighbour_counts(ctx, k, values):
    rng = np.random.default_rng(k * 1000 + values)
    x = rng.integers(0, values, size=(701, 5)).astype(np.float32)
    _equal(K.neighbors(x, k, ctx=ctx), O.neighbors(x, k))


@pytest.mark.parametrize("d", [1, 7, 8, 9, 31, 33, 50, 63, 64])
@pytest.mark.parametrize("n", [33, 1025, 4099])
def test_components_and_rows(ctx, d, n):
    x = np.random.default_rng(d + n).standard_normal((n, d)).astype(np.float32)
    k = min(30, n - 1)
    _equal(K.neighbors(x, k, ctx=ctx), O.neighbors(x, k))


@pytest.mark.parametrize("k", [15, 40])
def test_batch_of_ragged_samples(ctx, k):
    rng = np.random.default_rng(k)
    parts = [rng.standard_normal((m, 20)).astype(np.float32) for m in (k + 1, 127, 128, 129, 500)]
    for g, x in zip(K.neighbors_batch(parts, k, ctx=ctx), parts):
        _equal(g, O.neighbors(x, k))
