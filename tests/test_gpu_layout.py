"""The blocked layouts at the sizes where their builders' windows end: rows around a quarter and a
tile, columns around the windows of 256 and 512, rows empty, sparse and full.

A product through the layout stays within the product's own bar, 2^-15 sum |s| |d|; an entry lost,
doubled or misplaced is off by the entry."""

import numpy as np
import pytest

import kyto_b200 as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 32, 33, 129])
@pytest.mark.parametrize("g", [1, 33, 255, 256, 257, 513, 1030])
@pytest.mark.parametrize("density", [0.02, 1.0])
def test_window_edges(n, g, density):
    rng = np.random.default_rng(n * 2000 + g)
    s = rng.uniform(0.5, 2.0, (n, g)) * (rng.random((n, g)) < density)
    s[n // 2] = 0.0  # an empty row
    s[:, g - 1] = 1.0  # and a full last column
    s = s.astype(np.float32).astype(np.float64)
    rows, idx = np.nonzero(s)
    indptr = np.zeros(n + 1, dtype=np.uint64)
    indptr[1:] = np.cumsum(np.bincount(rows, minlength=n))
    args = indptr, idx.astype(np.uint32), s[rows, idx].astype(np.float32), g
    for transposed in (False, True):
        m = s.T if transposed else s
        d = rng.uniform(-1.0, 1.0, (m.shape[1], 5))
        got = K.product(*args, d, transposed)
        assert np.all(np.abs(got - m @ d) <= (np.abs(m) @ np.abs(d)) * 2.0**-15 + 1e-300)


@pytest.mark.parametrize("n", [40, 600, 16_400, 33_000])
def test_split_work_items_keep_the_bits(n):
    # 16,000 columns are work items enough for the chip, 300 are not and are split: a column's
    # f64 sums come out in the same order either way.
    g, few = 16_000, 300
    rng = np.random.default_rng(n)
    rows = np.repeat(np.arange(n), 6)
    idx = (rng.integers(0, few // 6, (n, 6)) * 6 + np.arange(6)) % few
    idx[:, 5] = rng.integers(few, g, n)  # one entry a row past the few
    idx.sort(axis=1)
    assert np.all(np.diff(idx, axis=1) > 0)
    val = rng.uniform(0.5, 2.0, (n, 6)).astype(np.float32)
    val[0, 0] = 2.0  # the same largest value in both
    d = rng.uniform(-1.0, 1.0, (n, 7))
    d[0] = 1.0
    whole = K.product(np.arange(n + 1, dtype=np.uint64) * 6, idx.ravel().astype(np.uint32),
                      val.ravel(), g, d, True)
    keep = idx < few
    indptr = np.zeros(n + 1, dtype=np.uint64)
    indptr[1:] = np.cumsum(keep.sum(1))
    part = K.product(indptr, idx[keep].astype(np.uint32), val[keep], few, d, True)
    assert np.array_equal(whole[:few].view(np.uint64), part.view(np.uint64))
    m = np.zeros((n, few))
    m[rows[keep.ravel()], idx[keep]] = val[keep]
    assert np.all(np.abs(part - m.T @ d) <= (m.T @ np.abs(d)) * 2.0**-15 + 1e-300)


@pytest.mark.parametrize("n", [60, 127, 128, 129, 2500])
@pytest.mark.parametrize("g", [512, 513, 1030])
def test_rows_from_split_work_items(n, g):
    # Few tiles of cells: their rows come from work items of 512 columns. Each is (x - mean) V to
    # the product's bar, 2^-15 of |x| |V| (and of the means' part), and its f32 rounding.
    rng = np.random.default_rng(n * 7 + g)
    x = (rng.gamma(1.0, 1.0, (n, g)) * (rng.random((n, g)) < 0.3)).astype(np.float32)
    x[:, g - 1] = 1.0
    rows, idx = np.nonzero(x)
    indptr = np.zeros(n + 1, dtype=np.uint64)
    indptr[1:] = np.cumsum(np.bincount(rows, minlength=n))
    res = K.pca(indptr, idx.astype(np.uint32), x[rows, idx], g, 5)
    m, v = x.astype(np.float64), res.loadings.astype(np.float64)
    ref = (m - m.mean(0)) @ v
    bar = ((np.abs(m) + np.abs(m).mean(0)) @ np.abs(v)) * (2.0**-15 + 2.0**-22)
    assert np.all(np.abs(res.embedding - ref) <= bar)
