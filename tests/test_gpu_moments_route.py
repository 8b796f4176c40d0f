"""Gene moments of blocks on both sides of the rule that sends few values a row to the sort: the same
bits as the sorting form, and a block of few values a row takes no pass over every row a group of
genes (its scratch would grow by 4 bytes a row and group)."""

import ctypes

import numpy as np
import pytest

import kyto_b200 as K

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _block(n_rows, n_genes, per_row, seed):
    """Every row `per_row` genes at an even stride from a drawn start."""
    rng = np.random.default_rng(seed)
    start = rng.integers(0, max(n_genes // per_row, 1), (n_rows, 1))
    idx = start + np.arange(per_row) * (n_genes // per_row)
    indptr = np.arange(n_rows + 1, dtype=np.uint64) * np.uint64(per_row)
    return indptr, idx.astype(np.uint32).reshape(-1), rng.integers(1, 90, idx.size).astype(np.uint32)


def _moments(name, indptr, idx, values, n_genes):
    d = [torch.from_numpy(a.view(t)).cuda() for a, t in
         ((indptr, np.int64), (idx, np.int32), (values, np.int32))]
    out = [torch.empty(n_genes, dtype=t, device="cuda")
           for t in (torch.float64, torch.float64, torch.int64)]
    torch.cuda.synchronize()  # the library's stream does not wait for torch's
    K._check(getattr(K.library(), name)(
        K.default_context().handle, *(t.data_ptr() for t in d[:3]), K.KG_U32, len(indptr) - 1,
        n_genes, ctypes.c_double(1e4), 1, *(o.data_ptr() for o in out)))
    return [o.cpu().numpy() for o in out]


@pytest.mark.parametrize("n_rows,n_genes,per_row", [
    (4096, 300, 30), (4097, 300, 30),      # on the line of few rows
    (4200, 400, 259), (4200, 400, 261),    # on the line of values a row, groups of 32 genes
    (5003, 300, 280), (2049, 37000, 500)])  # many tiles of rows; two rounds of groups
def test_both_routes_give_the_sorting_forms_bits(n_rows, n_genes, per_row):
    indptr, idx, values = _block(n_rows, n_genes, per_row, n_rows + per_row)
    got = _moments("kg_hvg_moments", indptr, idx, values, n_genes)
    want = [np.zeros(n_genes), np.zeros(n_genes), np.zeros(n_genes, dtype=np.int64)]
    if idx.size <= 1048576 and n_genes <= 65536:
        want = _moments("kg_hvg_moments_noalloc", indptr, idx, values, n_genes)
    else:  # the same rows, one swapped pair: the sort, whose order within a gene is the rows'
        u_idx, u_values = idx.copy(), values.copy()
        u_idx[:2], u_values[:2] = idx[1::-1], values[1::-1]
        want = _moments("kg_hvg_moments", indptr, u_idx, u_values, n_genes)
    for a, b in zip(got, want):
        assert np.array_equal(a.view(np.uint64), b.view(np.uint64))


def test_few_values_a_row_take_little_memory():
    n_rows, n_genes = 200_000, 20_000  # 125 groups of genes: 99 MB of bounds
    indptr, idx, values = _block(n_rows, n_genes, 4, 1)
    _moments("kg_hvg_moments", indptr, idx, values, n_genes)
    before = K.pool_usage(reset_high=True)
    _moments("kg_hvg_moments", indptr, idx, values, n_genes)
    high = K.pool_usage()["used_high"] - before["used"]
    assert high <= 24 * idx.size + (8 << 20)  # a few words a value
