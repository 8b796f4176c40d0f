"""Krylov blocks whose Cholesky step fails (numerically rank-deficient data) on memory that holds
NaNs: the block SVD must take nothing from factors that no step has written, and the Householder
form gives the answer.

Against the oracle with f64 products: variances within 1e-9 of the largest (f64 rounding), the
loadings of the data's own directions orthonormal to their f32 rounding (64 columns: 64 x 2^-24)."""

import numpy as np
import pytest

import kyto_b200 as K
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _leave_nans():
    """Fills blocks of the library's pool, of the sizes a block's factors have, with NaNs."""
    for count in (256, 900, 1800, 3600, 7200, 10800, 12288, 24576, 65536, 400000):
        nan = np.full(count, np.nan, dtype=np.float32)
        K.normalize_log1p(np.array([0, count], dtype=np.uint64), nan, target_sum=None)


@pytest.mark.parametrize("rank,g,k", [(1, 40, 5), (3, 64, 20), (12, 64, 20), (12, 300, 50),
                                      (30, 200, 44), (59, 500, 50)])
def test_rank_deficient_blocks(monkeypatch, rank, g, k):
    monkeypatch.setenv("KYTO_GPU_PCA_PRODUCTS", "simt")
    rng = np.random.default_rng(rank * g + k)
    cells = 700
    pattern = rng.integers(1, 9, (rank, g)).astype(np.float64)
    dense = pattern[np.arange(cells) % rank]
    indptr = np.arange(cells + 1, dtype=np.uint64) * np.uint64(g)
    x = O.Csr(indptr, np.tile(np.arange(g, dtype=np.uint32), cells),
              dense.astype(np.float32).reshape(-1), g)
    ref = O.pca(x, k)
    for _ in range(3):
        _leave_nans()
        res = K.pca(x.indptr, x.indices, x.values, g, k)
        assert np.max(np.abs(res.variance - ref.variance)) <= 1e-9 * max(ref.variance[0], 1.0)
        own = min(rank - 1, k)  # the rank of the centred rows
        load = res.loadings.astype(np.float64)[:, :own]
        assert np.max(np.abs(load.T @ load - np.eye(own)), initial=0.0) <= 64 * 2.0**-24
