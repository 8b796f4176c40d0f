"""Gene moments of blocks whose offsets step back: such a row is empty, and the block goes to the sort,
which takes each stored value once. Bit for bit the sorting form's (kg_hvg_moments_noalloc). No
normalization, which would depend on the row a value is in. And blocks of many rows with one out of
gene order, wherever it stands, with and without a gene out of range after it."""

import ctypes
import math

import numpy as np
import pytest

import kyto_b200 as K

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _moments(name, indptr, idx, values, n_genes):
    d = [torch.from_numpy(a.view(t)).cuda() for a, t in
         ((indptr, np.int64), (idx, np.int32), (values, np.int32))]
    out = [torch.empty(n_genes, dtype=t, device="cuda")
           for t in (torch.float64, torch.float64, torch.int64)]
    torch.cuda.synchronize()  # the library's stream does not wait for torch's
    K._check(getattr(K.library(), name)(
        K.default_context().handle, *(t.data_ptr() for t in d), K.KG_U32, len(indptr) - 1,
        n_genes, ctypes.c_double(math.nan), 1, *(o.data_ptr() for o in out)))
    return [o.cpu().numpy() for o in out]


@pytest.mark.parametrize("n_genes", [32, 300, 9000])
@pytest.mark.parametrize("rows,at,back", [(4, 1, 2), (64, 31, 1), (300, 200, 17), (300, 297, 3)])
def test_offsets_that_step_back(n_genes, rows, at, back):
    rng = np.random.default_rng(rows + n_genes)
    per_row = 20
    idx = np.sort(np.stack([rng.permutation(n_genes)[:per_row] for _ in range(rows)]), 1)
    idx = idx.astype(np.uint32).reshape(-1)
    values = rng.integers(1, 90, idx.size).astype(np.uint32)
    indptr = np.arange(rows + 1, dtype=np.uint64) * np.uint64(per_row)
    # Row `at` takes in the next row and `back` values of the one after it, whose offset stays.
    indptr[at + 1] += np.uint64(per_row + back)
    assert indptr.max() <= idx.size and (np.diff(indptr.astype(np.int64)) < 0).sum() == 1
    got = _moments("kg_hvg_moments", indptr, idx, values, n_genes)
    want = _moments("kg_hvg_moments_noalloc", indptr, idx, values, n_genes)
    for a, b in zip(got, want):
        assert np.array_equal(a.view(np.uint64), b.view(np.uint64))


@pytest.mark.parametrize("where", [0, 1500, 2999])
@pytest.mark.parametrize("n_genes", [300, 9000])
def test_one_row_out_of_order(where, n_genes):
    rows, per_row = 3000, 300
    rng = np.random.default_rng(where + n_genes)
    idx = np.sort(np.argsort(rng.random((rows, n_genes)), 1)[:, :per_row], 1).astype(np.uint32)
    values = rng.integers(1, 90, idx.size).astype(np.uint32)
    idx[where, 3:5] = idx[where, 4:2:-1]
    indptr = np.arange(rows + 1, dtype=np.uint64) * np.uint64(per_row)
    idx = idx.reshape(-1)
    got = _moments("kg_hvg_moments", indptr, idx, values, n_genes)
    want = _moments("kg_hvg_moments_noalloc", indptr, idx, values, n_genes)
    for a, b in zip(got, want):
        assert np.array_equal(a.view(np.uint64), b.view(np.uint64))
    idx[-1], idx[5] = n_genes + 7, n_genes + 2  # the largest is named, wherever it stands
    with pytest.raises(K.KytoError, match=f"gene index {n_genes + 7} but has {n_genes} genes"):
        _moments("kg_hvg_moments", indptr, idx, values, n_genes)
