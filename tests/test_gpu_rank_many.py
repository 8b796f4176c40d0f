"""The re-rank of queries with more candidates than one batch holds (256): rows far from the mean, whose
slack covers most of the others, through each filter; ties by the hundred; neighbour counts around 32
and up to the most. The oracle's graph is exact: indices and distances are compared as bits."""

import numpy as np
import pytest

import kyto_b200 as K
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _far(n, d, seed):
    """Two tight groups far apart: every row of a group is within the other's slack."""
    rng = np.random.default_rng(seed)
    x = rng.normal(0.0, 1e-3, (n, d))
    x[:, 0] += np.where(np.arange(n) % 2, 60.0, -60.0)
    return x.astype(np.float32)


@pytest.mark.parametrize("filter_kind", ["simt", "fp16", "split", "bf16"])
@pytest.mark.parametrize("k", [2, 15, 33, 34, 65, 129])
@pytest.mark.parametrize("n", [520, 900, 1900])
def test_far_groups(monkeypatch, filter_kind, k, n):
    monkeypatch.setenv("KYTO_GPU_KNN_FILTER", filter_kind)
    x = _far(n, 12, n + k)
    got, want = K.neighbors(x, k), O.neighbors(x, k)
    assert np.array_equal(got.indices, want.indices)
    assert np.array_equal(got.distances.view(np.uint32), want.distances.view(np.uint32))
    if filter_kind in ("fp16", "bf16") and n >= 900:
        assert got.stats.candidates > 400 * n  # several batches a row


@pytest.mark.parametrize("filter_kind", ["simt", "fp16", "bf16"])
@pytest.mark.parametrize("k", [15, 40, 129])
def test_ties(monkeypatch, filter_kind, k):
    monkeypatch.setenv("KYTO_GPU_KNN_FILTER", filter_kind)
    x = np.random.default_rng(k).integers(0, 2, (1500, 3)).astype(np.float32)
    got, want = K.neighbors(x, k), O.neighbors(x, k)
    assert np.array_equal(got.indices, want.indices)
    assert np.array_equal(got.distances.view(np.uint32), want.distances.view(np.uint32))


@pytest.mark.parametrize("k", [15, 31, 33, 100])
def test_wide_slack_on_scores(monkeypatch, k):
    """bf16's slack on rows like a PCA's scores: hundreds of candidates a row, of any distance."""
    monkeypatch.setenv("KYTO_GPU_KNN_FILTER", "bf16")
    n, d = 20_000, 50
    rng = np.random.default_rng(1)
    centre = rng.normal(size=(40, d)) * 24.0 / (1.0 + np.arange(d)) ** 0.55
    x = centre[rng.integers(40, size=n)]
    x += (1.0 + 1.5 / np.sqrt(1.0 + np.arange(d))) * rng.normal(size=(n, d))
    x = x.astype(np.float32)
    got, want = K.neighbors(x, k), O.neighbors(x, k)
    assert got.stats.candidates > 400 * n
    assert np.array_equal(got.indices, want.indices)
    assert np.array_equal(got.distances.view(np.uint32), want.distances.view(np.uint32))
