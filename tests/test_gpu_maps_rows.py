"""The maps where their row forms change: rows around a table's 64 values, blocks around 16,384 rows of
64 values on average (eight lanes a row from there on) and around 32,768 rows of f32 values that are
no counts, rows far longer than the rest, f32 rows that start like counts and are none, counts above
2^24. Bit for bit the oracle's."""

import numpy as np
import pytest

import kyto_b200 as K
from oracle import oracle as O

pytestmark = pytest.mark.gpu

EDGES = np.array([63, 64, 65, 2**24, 2**24 + 1, 2**31 + 1, 2**32 - 1], dtype=np.uint32)


def _values(rng, count, dtype):
    counts = rng.integers(1, 90, count).astype(np.uint32)
    if dtype == "u32":
        at = rng.random(count) < 0.02
        counts[at] = rng.choice(EDGES, int(at.sum()))
        return counts
    values = counts.astype(np.float32)
    if dtype == "f32":
        values += rng.choice(np.array([0.0, 0.25, 0.7], dtype=np.float32), count)
    elif dtype == "late":  # whole numbers but for one value near the end of the block
        values[-3] = 2.5
    elif dtype == "early":  # no counts at the start only
        values[:3] = 0.5
    return values


@pytest.mark.parametrize("dtype", ["u32", "whole", "f32", "late", "early"])
@pytest.mark.parametrize("target,log1p", [(1e4, True), (None, True), (1e4, False)])
@pytest.mark.parametrize("rows,mean", [(300, 64), (16383, 20), (16384, 20), (16385, 64), (16387, 66),
                                       (32767, 70), (32768, 70), (33001, 5)])
def test_row_forms(rows, mean, target, log1p, dtype):
    rng = np.random.default_rng(rows + mean)
    lengths = rng.integers(mean - min(mean, 5), mean + 6, rows)
    lengths[rows // 3] = 0
    lengths[rows // 2] = 700
    indptr = np.concatenate([[0], np.cumsum(lengths)]).astype(np.uint64)
    values = _values(rng, int(indptr[-1]), dtype)
    got = K.normalize_log1p(indptr, values, target, log1p)
    idx = np.zeros(values.size, dtype=np.uint32)
    want = O.normalize_log1p(O.Csr(indptr, idx, values, 1), target, log1p).values
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("dtype", ["u32", "whole", "f32", "late", "early"])
@pytest.mark.parametrize("length", [30, 63, 64, 65, 200])
@pytest.mark.parametrize("keep", [None, 40, 70])
def test_pca_input_maps(monkeypatch, length, dtype, keep):
    """The same maps as a pushed block's, through a whole PCA with f64 products: a wrong value is
    off by far more than their rounding (variances within 1e-9 of the largest)."""
    monkeypatch.setenv("KYTO_GPU_PCA_PRODUCTS", "simt")
    rows, genes = 120, 260
    rng = np.random.default_rng(length)
    idx = np.sort(np.argsort(rng.random((rows, genes)), 1)[:, :length], 1).astype(np.uint32)
    indptr = np.arange(rows + 1, dtype=np.uint64) * np.uint64(length)
    values = _values(rng, idx.size, dtype if dtype != "u32" else "whole").astype(
        np.uint32 if dtype == "u32" else np.float32)
    flags = None
    if keep:
        flags = np.zeros(genes, dtype=bool)
        flags[rng.permutation(genes)[:keep]] = True
    got = K.pca(indptr, idx.reshape(-1), values, genes, 5, gene_set=flags, target_sum=1e4,
                log1p=True)
    mapped = O.normalize_log1p(O.Csr(indptr, idx.reshape(-1), values, genes), 1e4, True)
    dense = np.zeros((rows, genes), dtype=np.float32)
    np.put_along_axis(dense, idx.astype(np.int64), mapped.values.reshape(rows, length), 1)
    if keep:
        dense = dense[:, flags]
    r, c = np.nonzero(dense)
    ptr = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=rows))]).astype(np.uint64)
    ref = O.pca(O.Csr(ptr, c.astype(np.uint32), dense[r, c], dense.shape[1]), 5)
    assert np.max(np.abs(got.variance - ref.variance)) <= 1e-9 * ref.variance[0]
