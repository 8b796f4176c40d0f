"""The tile join past 32 gene blocks, where a warp takes 32 tiles of a row as one run of entries: tile
counts around a run's end, rows empty, short and full, tiles empty; bit for bit the oracle's rows, and
the oracle's first problem for damage anywhere in a run."""

import numpy as np
import pytest

import kyto_b200 as K
from oracle import tiles as T

pytestmark = pytest.mark.gpu

CELLS = 45


def _layer(n_genes, per_row, seed):
    rng = np.random.default_rng(seed)
    lengths = rng.integers(0, per_row + 1, CELLS)
    lengths[3], lengths[7] = 0, n_genes  # an empty row and a full one
    rows = [np.sort(rng.choice(n_genes, m, replace=False)) for m in lengths]
    indptr = np.concatenate([[0], np.cumsum(lengths)]).astype(np.uint64)
    idx = np.concatenate(rows).astype(np.uint32)
    return indptr, idx, rng.integers(1, 99, len(idx)).astype(np.uint32)


@pytest.mark.parametrize("blocks", [31, 32, 33, 63, 64, 65, 96, 97, 200])
@pytest.mark.parametrize("gene_block,per_row", [(1, 20), (3, 2), (40, 300)])
def test_join_matches_the_oracle(blocks, gene_block, per_row):
    n_genes = blocks * gene_block - (1 if gene_block > 1 else 0)  # a ragged last tile
    grid = T.TileGrid(CELLS, n_genes, 37, gene_block)
    layer = _layer(n_genes, min(per_row, n_genes), blocks)
    shards, offsets, idx, vals = T.encode_fast(*layer, grid)
    for b in range(grid.n_cell_blocks):
        want = T.decode_cell_block(grid, b, shards[b], offsets, idx, vals)
        got = K.tiles_to_csr(b, 37, gene_block, CELLS, n_genes, shards[b], offsets, idx, vals)
        for x, y in zip(got, want):
            assert np.array_equal(np.asarray(x), np.asarray(y))


def _problems(grid, shards, offsets, idx, vals):
    with pytest.raises(Exception) as want:
        T.decode_cell_block(grid, 0, shards[0], offsets, idx, vals)
    with pytest.raises(K.KytoError) as got:
        K.tiles_to_csr(0, grid.cell_block_size, grid.gene_block_size, grid.n_cells, grid.n_genes,
                       shards[0], offsets, idx, vals)
    assert got.value.code == "KY-E107" and str(want.value) in str(got.value)


@pytest.mark.parametrize("tile", [0, 31, 32, 50, 64, 69])
@pytest.mark.parametrize("damage", ["wide", "order", "equal", "both", "start", "end", "decrease"])
def test_first_problem(tile, damage):
    grid = T.TileGrid(CELLS, 70 * 6, CELLS, 6)
    shards, offsets, idx, vals = T.encode_fast(*_layer(70 * 6, 200, 5), grid)
    idx, shards = idx.copy(), [np.array(s) for s in shards]
    shard = shards[0].reshape(70, CELLS + 1)
    at = int(offsets[tile]) + int(shard[tile, 7])  # the full row's segment
    if damage in ("wide", "both"):
        idx[at + 5] = 6
    if damage == "order":
        idx[at + 2:at + 4] = idx[at + 2:at + 4][::-1]
    if damage in ("equal", "both"):
        idx[at + 1] = idx[at]
    if damage == "start":
        shard[tile, 0] = 1
    if damage == "end":
        shard[tile, -1] += 1
    if damage == "decrease":
        shard[tile, 20] = shard[tile, 19] - 1 if shard[tile, 19] else 0xFFFFFF
    shards[0] = shard.reshape(shards[0].shape)
    _problems(grid, shards, offsets, idx, vals)
