"""Connectivities where the row kernels' tiles end: neighbours a row around a warp (31, 32,
33) and up to the most, rows named by none, by one and by hundreds of others, distances with
ties, zeros and wide ranges, distances that decide a bisection step late; against the oracle.

Edges are equal; a weight is one f32 exponential (evaluated in f64 by both sides and rounded
once, so equal but where the two f64 exponentials fall on two sides of a rounding) and two f32
operations: 1e-6, and all but one in a thousand bit for bit."""

import numpy as np
import pytest

import kyto_b200 as K
from oracle import connectivities as OC

pytestmark = pytest.mark.gpu


def _graph(n, k, seed, hub, kind):
    rng = np.random.default_rng(seed)
    cols = np.empty((n, k), dtype=np.uint32)
    for r in range(n):
        pick = rng.choice(n, k, replace=False)
        if hub and 0 not in pick:
            pick[0] = 0
        cols[r] = np.sort(pick)
    if kind == "ties":
        dist = rng.integers(0, 4, (n, k)).astype(np.float32)
    elif kind == "wide":
        dist = np.exp(rng.uniform(np.log(1e-6), np.log(1e6), (n, k))).astype(np.float32)
    else:
        dist = (rng.uniform(2, 3, (n, 1)) * rng.uniform(1.0, 1.2, (n, k))).astype(np.float32)
    return K.Graph(np.arange(n + 1, dtype=np.uint64) * np.uint64(k), cols.reshape(-1),
                   dist.reshape(-1))


@pytest.mark.parametrize("n,k,hub,kind", [
    (2, 1, False, "near"), (130, 2, False, "ties"), (500, 14, True, "near"),
    (500, 14, False, "wide"), (129, 31, True, "near"), (257, 32, True, "ties"),
    (300, 33, True, "wide"), (400, 192, False, "near"), (300, 255, True, "near")])
def test_matches_the_oracle(n, k, hub, kind):
    g = _graph(n, k, n + k, hub, kind)
    got = K.connectivities(g)
    want = OC.connectivities(g.indptr, g.indices, g.distances, k + 1)
    assert np.array_equal(got.indptr, want[0])
    assert np.array_equal(got.indices, want[1])
    assert np.abs(got.weights.astype(np.float64) - want[2]).max(initial=0) <= 1e-6
    assert (got.weights.view(np.uint32) == want[2].view(np.uint32)).mean() > 0.999
