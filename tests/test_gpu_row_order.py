"""Rows whose genes do not increase, at the places where the blocked layouts' builder changes
chunks (32 entries) and windows (256 and 512 columns): a PCA takes them (the products then run in
f64), the product diagnostic refuses them.

The PCA of rows in any order is that of the sorted rows: variances within 1e-9 of the oracle's
largest (f64 products; only the order of a row's sum differs), loadings within f32 rounding of the
sorted input's (64 x 2^-24, entries at most 1 in size)."""

import numpy as np
import pytest

import kyto_b200 as K
from oracle import oracle as O

pytestmark = pytest.mark.gpu

N = 200


def _matrix(g):
    rng = np.random.default_rng(g)
    dense = rng.gamma(1.0, 2.0, (N, g)) * (rng.random((N, g)) < 0.7)
    dense *= 1.3 ** -np.minimum(np.arange(g), 40.0)
    dense[7] = np.linspace(0.5, 1.5, g)  # a full row
    dense[::17] = 0.0  # empty rows
    dense = dense.astype(np.float32)
    rows, idx = np.nonzero(dense)
    indptr = np.zeros(N + 1, dtype=np.uint64)
    indptr[1:] = np.cumsum(np.bincount(rows, minlength=N))
    return indptr, idx.astype(np.uint32), dense[rows, idx]


def _swap(indptr, idx, val, a, b):
    """Row 7's entries a and b change places."""
    idx, val, s = idx.copy(), val.copy(), int(indptr[7])
    for arr in (idx, val):
        arr[s + a], arr[s + b] = arr[s + b], arr[s + a]
    return idx, val


@pytest.mark.parametrize("g,a,b", [(40, 0, 1), (300, 31, 32), (300, 0, 299), (600, 255, 256),
                                   (600, 511, 512), (1030, 3, 1029), (1030, 512, 1024),
                                   (1030, None, None)])
def test_pca_takes_any_order(monkeypatch, g, a, b):
    indptr, idx, val = _matrix(g)
    ref = O.pca(O.Csr(indptr, idx, val, g), 6)
    if a is None:  # every row backwards
        order = np.concatenate([np.arange(int(e) - 1, int(s) - 1, -1)
                                for s, e in zip(indptr, indptr[1:])] or [[]]).astype(np.int64)
        u_idx, u_val = idx[order], val[order]
    else:
        u_idx, u_val = _swap(indptr, idx, val, a, b)
    got = K.pca(indptr, u_idx, u_val, g, 6)
    assert np.max(np.abs(got.variance - ref.variance)) <= 1e-9 * ref.variance[0]
    monkeypatch.setenv("KYTO_GPU_PCA_PRODUCTS", "simt")
    want = K.pca(indptr, idx, val, g, 6)
    assert np.max(np.abs(got.loadings - want.loadings)) <= 64 * 2.0**-24


@pytest.mark.parametrize("transposed", [False, True])
@pytest.mark.parametrize("g,a,b", [(40, 0, 1), (300, 31, 32), (600, 255, 256), (600, 511, 512),
                                   (1030, 3, 1029)])
def test_product_refuses_them(transposed, g, a, b):
    indptr, idx, val = _matrix(g)
    d = np.ones((N if transposed else g, 3))
    K.product(indptr, idx, val, g, d, transposed=transposed)
    for wrong, _ in (_swap(indptr, idx, val, a, b), (np.where(
            np.arange(idx.size) == int(indptr[7]) + b, idx[int(indptr[7]) + b - 1], idx), None)):
        with pytest.raises(K.KytoError) as err:
            K.product(indptr, wrong.astype(np.uint32), val, g, d, transposed=transposed)
        assert err.value.status == K.KG_ERR_INVALID
