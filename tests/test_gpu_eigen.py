"""The PCA's last eigenproblem at the sizes where its kernels change (bases of 9 to 576 columns,
50 and 51 pairs, row counts around a lane's block) and on spectra that are hard for inverse
iteration: equal eigenvalues, a few distinct ones, many zeros.

Products in f64, so what differs from the oracle's LAPACK is f64 rounding: variances within 1e-9
of the largest, loadings orthonormal to their f32 rounding (64 columns: 64 x 2^-24), and each
loading an eigenvector to that rounding times the spread (residual within 1e-5 of the largest)."""

import numpy as np
import pytest

import kyto_b200 as K
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _csr(dense):
    dense = dense.astype(np.float32)
    indptr = np.zeros(dense.shape[0] + 1, dtype=np.uint64)
    indptr[1:] = np.cumsum((dense != 0).sum(1))
    rows, idx = np.nonzero(dense)
    return O.Csr(indptr, idx.astype(np.uint32), dense[rows, idx], dense.shape[1])


def _check(monkeypatch, dense, k):
    monkeypatch.setenv("KYTO_GPU_PCA_PRODUCTS", "simt")
    n, g = dense.shape
    x = _csr(dense)
    res = K.pca(x.indptr, x.indices, x.values, g, k)
    ref = O.pca(x, k)
    assert np.max(np.abs(res.variance - ref.variance)) <= 1e-9 * ref.variance[0]
    load = res.loadings.astype(np.float64)
    assert np.max(np.abs(load.T @ load - np.eye(k))) <= 64 * 2.0**-24
    c = dense - dense.mean(0)
    residual = c.T @ (c @ load) / (n - 1) - load * res.variance
    assert np.max(np.linalg.norm(residual, axis=0)) <= 1e-5 * ref.variance[0]


@pytest.mark.parametrize("k,g", [(1, 2), (1, 33), (2, 100), (6, 150), (14, 216), (15, 300),
                                 (18, 256), (47, 513), (50, 700), (51, 700), (54, 700)])
def test_sizes(monkeypatch, k, g):
    rng = np.random.default_rng(k + g)
    dense = rng.gamma(1.0, 1.0, (500, g)) * (rng.random((500, g)) < 0.5)
    dense = dense.astype(np.float32).astype(np.float64)
    dense *= np.float32(1.5) ** -np.minimum(np.arange(g) // 2, 60)  # a decaying spectrum
    _check(monkeypatch, dense.astype(np.float32).astype(np.float64), k)


@pytest.mark.parametrize("kind", ["equal", "steps", "rank"])
@pytest.mark.parametrize("k", [5, 20])
def test_close_eigenvalues(monkeypatch, kind, k):
    g = 64
    cells = np.arange(640)
    dense = np.zeros((640, g))
    if kind == "equal":  # one gene a cell: all variances alike
        dense[cells, cells % g] = 3.0
    elif kind == "steps":  # three variances, many times each
        dense[cells, cells % g] = 1.0 + cells % g % 3
    else:  # 12 patterns of disjoint genes: rank 12
        dense[cells[:, None], (cells % 12 * 5)[:, None] + np.arange(5)] = 2.0
    _check(monkeypatch, dense, k)
