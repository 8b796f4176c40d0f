"""The tile join around its inline tile starts (64 gene blocks travel as a kernel argument,
more in device memory) and its row chunks (128 entries a step): bit for bit the oracle's rows,
and the oracle's first problem for a damaged tile past that line."""

import numpy as np
import pytest

import kyto_b200 as K
from oracle import tiles as T

pytestmark = pytest.mark.gpu


def _layer(n_cells, n_genes, per_row, seed):
    rng = np.random.default_rng(seed)
    rows = [np.sort(rng.choice(n_genes, m, replace=False))
            for m in rng.integers(0, per_row + 1, n_cells)]
    indptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.uint64)
    idx = np.concatenate(rows).astype(np.uint32)
    return indptr, idx, rng.integers(1, 99, len(idx)).astype(np.uint32)


@pytest.mark.parametrize("n_genes,gene_block,per_row", [
    (64 * 5, 5, 300), (64 * 5 + 1, 5, 300), (700, 3, 90), (129, 129, 129), (260, 129, 257)])
def test_join_matches_the_oracle(n_genes, gene_block, per_row):
    grid = T.TileGrid(50, n_genes, 37, gene_block)
    shards, offsets, idx, vals = T.encode_fast(*_layer(50, n_genes, per_row, n_genes), grid)
    for b in range(grid.n_cell_blocks):
        want = T.decode_cell_block(grid, b, shards[b], offsets, idx, vals)
        got = K.tiles_to_csr(b, 37, gene_block, 50, n_genes, shards[b], offsets, idx, vals)
        for x, y in zip(got, want):
            assert np.array_equal(np.asarray(x), np.asarray(y))


def test_a_damaged_tile_past_the_inline_starts():
    grid = T.TileGrid(40, 700, 40, 7)
    shards, offsets, idx, vals = T.encode_fast(*_layer(40, 700, 200, 9), grid)
    tile = 90
    idx = idx.copy()
    idx[int(offsets[tile])] = 7  # a local index at the block width
    with pytest.raises(Exception) as want:
        T.decode_cell_block(grid, 0, shards[0], offsets, idx, vals)
    with pytest.raises(K.KytoError) as got:
        K.tiles_to_csr(0, 40, 7, 40, 700, shards[0], offsets, idx, vals)
    assert got.value.code == "KY-E107" and str(want.value) in str(got.value)
