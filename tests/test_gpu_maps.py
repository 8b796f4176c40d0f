"""The maps' per-row tables and the moments' row tiles where they can go wrong:
counts at the table's end, above 2^24 and up to 2^32 - 1, f32 values that are whole, halves
and negative zeros, rows of 0 to a few hundred values; rows that end on a tile of 32 or a ring
of four, one to many groups of genes, more genes a row than a warp, rows out of gene order. All bit for bit: the maps against the oracle, the
moments against the library's sorting form (kg_hvg_moments_noalloc), which adds the same
values in the same order."""

import ctypes

import numpy as np
import pytest

import kyto_b200 as K
from oracle import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

EDGES = np.array([0, 1, 2, 62, 63, 64, 65, 1000, 2**24 - 1, 2**24, 2**24 + 1, 2**25 + 3,
                  2**31 + 1, 2**32 - 1], dtype=np.uint32)


def _block(n_rows, n_genes, longest, dtype, seed, shuffle=False):
    rng = np.random.default_rng(seed)
    lengths = rng.integers(0, min(longest, n_genes) + 1, n_rows)
    indptr = np.concatenate([[0], np.cumsum(lengths)]).astype(np.uint64)
    idx = [np.sort(rng.choice(n_genes, m, replace=False)) for m in lengths]
    if shuffle:
        idx[n_rows // 2] = idx[n_rows // 2][::-1]
    idx = np.concatenate(idx + [np.empty(0)]).astype(np.uint32)
    if dtype == "u32":
        values = rng.integers(1, 70, idx.size).astype(np.uint32)
        at = rng.random(idx.size) < 0.05
        values[at] = rng.choice(EDGES, int(at.sum()))
    else:
        values = rng.choice(np.array([0.0, -0.0, 1, 2, 63, 64, 0.5, 7.25, 63.5, 1e-30, 3e7],
                                     dtype=np.float32), idx.size)
        if dtype == "whole":
            values = np.trunc(values)
    return indptr, idx, values


@pytest.mark.parametrize("dtype", ["u32", "whole", "f32"])
@pytest.mark.parametrize("target,log1p", [(1e4, True), (1e4, False), (None, True), (None, False)])
def test_maps_match_the_oracle(dtype, target, log1p):
    indptr, idx, values = _block(97, 3000, 300, dtype, 5)
    got = K.normalize_log1p(indptr, values, target, log1p)
    want = O.normalize_log1p(O.Csr(indptr, idx, values, 3000), target, log1p).values
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


def _moments(name, indptr, idx, values, n_genes):
    lib, ctx = K.library(), K.default_context()
    d = [torch.from_numpy(a.view(t)).cuda() for a, t in
         ((indptr, np.int64), (idx, np.int32), (values, values.dtype if values.dtype == np.float32
                                               else np.int32))]
    out = [torch.empty(n_genes, dtype=torch.float64, device="cuda"),
           torch.empty(n_genes, dtype=torch.float64, device="cuda"),
           torch.empty(n_genes, dtype=torch.int64, device="cuda")]
    K._check(getattr(lib, name)(
        ctx.handle, d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), K._dtype_code(values),
        len(indptr) - 1, n_genes, ctypes.c_double(1e4), 1, *[o.data_ptr() for o in out]))
    return [o.cpu().numpy() for o in out]


@pytest.mark.parametrize("n_rows,n_genes,longest,dtype,shuffle", [
    (1, 1, 1, "u32", False), (31, 64, 64, "u32", False), (127, 32, 32, "u32", False), (129, 4768, 4768, "u32", False), (32, 65, 65, "f32", False),
    (33, 500, 300, "u32", False), (5000, 37, 37, "u32", False), (4737, 90, 60, "f32", False),
    (300, 27000, 400, "u32", False), (64, 37889, 900, "u32", False),
    (200, 65536, 700, "whole", False), (1200, 7, 7, "whole", False),
    (200, 800, 200, "u32", True)])
def test_moments_match_the_sorting_form(n_rows, n_genes, longest, dtype, shuffle):
    block = _block(n_rows, n_genes, longest, dtype, n_rows + n_genes, shuffle)
    got = _moments("kg_hvg_moments", *block, n_genes)
    want = _moments("kg_hvg_moments_noalloc", *block, n_genes)
    for a, b in zip(got, want):
        assert np.array_equal(a.view(np.uint64), b.view(np.uint64))


def test_moments_refuse_a_gene_out_of_range():
    indptr, idx, values = _block(50, 200, 80, "u32", 3)
    idx[-1] = 200
    with pytest.raises(K.KytoError, match="gene index 200 but has 200 genes"):
        _moments("kg_hvg_moments", indptr, idx, values, 200)
