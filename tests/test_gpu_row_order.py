"""Rows whose genes do not increase, at the places where the blocked layouts' builder changes
chunks (32 entries) and windows (256 and 512 columns). Where the order does not reach the layout, the
answer is the sorted rows', bit for bit; elsewhere a PCA's products run in f64, and the product
diagnostic refuses the rows.

A PCA with f64 products differs from the oracle by the order of a row's sums: variances within 1e-9
of the largest; loadings within f32 rounding of the sorted input's with f64 products (64 x 2^-24,
entries at most 1 in size)."""

import numpy as np
import pytest

import kyto_b200 as K
from oracle import oracle as O

pytestmark = pytest.mark.gpu

N = 200


def _matrix(g):
    rng = np.random.default_rng(g)
    dense = rng.uniform(0.5, 2.0, (N, g)) * (rng.random((N, g)) < 0.7)
    dense *= 1.05 ** -np.minimum(np.arange(g), 60.0)  # within the tensor cores' range of values
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


def _pca(indptr, idx, val, g):
    """The result and whether the products ran on the tensor cores."""
    sess = K.PcaSession(6, g)
    sess.push(indptr, idx, val)
    sess.run()
    return sess.results(), sess.stats().product_launches > 0


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
    got, tensor = _pca(indptr, u_idx, u_val, g)
    same, sorted_tensor = _pca(indptr, idx, val, g)
    assert sorted_tensor
    assert tensor == (a is not None and a // 256 == b // 256)  # swapped inside a window
    if tensor:
        assert np.array_equal(got.variance, same.variance)
        assert np.array_equal(got.loadings, same.loadings)
        assert np.array_equal(got.embedding, same.embedding)
        return
    assert np.max(np.abs(got.variance - ref.variance)) <= 1e-9 * ref.variance[0]
    monkeypatch.setenv("KYTO_GPU_PCA_PRODUCTS", "simt")
    want = K.pca(indptr, idx, val, g, 6)
    assert np.max(np.abs(got.loadings - want.loadings)) <= 64 * 2.0**-24


@pytest.mark.parametrize("transposed", [False, True])
@pytest.mark.parametrize("g,a,b", [(40, 0, 1), (300, 31, 32), (300, 0, 299), (600, 255, 256),
                                   (600, 511, 512), (1030, 3, 1029)])
def test_product_is_refused_or_right(transposed, g, a, b):
    indptr, idx, val = _matrix(g)
    d = np.ones((N if transposed else g, 3))
    want = K.product(indptr, idx, val, g, d, transposed=transposed)
    u_idx, u_val = _swap(indptr, idx, val, a, b)
    try:
        got = K.product(indptr, u_idx, u_val, g, d, transposed=transposed)
    except K.KytoError as err:
        assert err.status == K.KG_ERR_INVALID
    else:
        assert np.array_equal(got, want)
    twice = idx.copy()
    twice[int(indptr[7]) + b] = twice[int(indptr[7]) + b - 1]
    with pytest.raises(K.KytoError) as err:
        K.product(indptr, twice, val, g, d, transposed=transposed)
    assert err.value.status == K.KG_ERR_INVALID


def test_a_gene_twice_in_a_row(monkeypatch):
    indptr, idx, val = _matrix(300)
    at = int(indptr[7]) + 20
    idx[at] = idx[at - 1]
    got, tensor = _pca(indptr, idx, val, 300)
    assert not tensor
    monkeypatch.setenv("KYTO_GPU_PCA_PRODUCTS", "simt")
    want = K.pca(indptr, idx, val, 300, 6)
    assert np.array_equal(got.loadings, want.loadings)  # the f64 products both times
