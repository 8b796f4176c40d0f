"""The PCA's dense FP64 steps at the widths where their tiles end (Krylov blocks of 11 to
64 columns, bases that fill the genes, ranks below the block), against the oracle's LAPACK.

The products run in f64 (KYTO_GPU_PCA_PRODUCTS=simt), so what differs from the oracle is
f64 rounding of the dense steps: variances within 1e-9 of the largest (a basis of at most
540 columns orthonormal to 1e-13, eigenvalues backward stable to n 2^-52), loadings
orthonormal to their f32 rounding (64 columns: 64 x 2^-24)."""

import numpy as np
import pytest

import kyto_b200 as K
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _matrix(n, g, rank, seed):
    rng = np.random.default_rng(seed)
    if rank is None:
        dense = rng.gamma(1.0, 1.0, (n, g)) * (rng.random((n, g)) < 0.4)
    else:  # exactly rank `rank` in f32: small integers
        dense = rng.integers(0, 3, (n, rank)) @ rng.integers(0, 3, (rank, g))
    dense = dense.astype(np.float32)
    indptr = np.zeros(n + 1, dtype=np.uint64)
    indptr[1:] = np.cumsum((dense != 0).sum(1))
    rows, idx = np.nonzero(dense)
    return O.Csr(indptr, idx.astype(np.uint32), dense[rows, idx], g)


@pytest.mark.parametrize("k,g,rank", [(1, 40, None), (5, 15, None), (22, 200, None),
                                      (38, 500, None), (54, 700, None), (54, 64, None),
                                      (20, 90, 12), (50, 300, 57)])
def test_block_widths_match_the_oracle(monkeypatch, k, g, rank):
    monkeypatch.setenv("KYTO_GPU_PCA_PRODUCTS", "simt")
    x = _matrix(900, g, rank, k + g)
    res = K.pca(x.indptr, x.indices, x.values, g, k)
    ref = O.pca(x, k)
    assert res.passes_run == ref.passes_run
    assert np.max(np.abs(res.variance - ref.variance)) <= 1e-9 * ref.variance[0]
    gram = res.loadings.astype(np.float64).T @ res.loadings.astype(np.float64)
    assert np.max(np.abs(gram - np.eye(k))) <= 64 * 2.0**-24
