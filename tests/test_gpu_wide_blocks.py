"""Krylov blocks at the sizes where their sum of squares comes in more parts (16,384 values a part, 128
parts at most), up to the widest the tensor cores' layouts take. The norm decides which directions are
kept, so an error there shows in the passes and the variances: the oracle's, with f64 products within
1e-9 of the largest (f64 rounding)."""

import numpy as np
import pytest

import kyto_b200 as K
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("g", [546, 547, 1093, 20_000, 65_535, 71_000])
def test_block_sizes(monkeypatch, g):
    monkeypatch.setenv("KYTO_GPU_PCA_PRODUCTS", "simt")
    rng = np.random.default_rng(g)
    cells, per_row, k = 150, 200, 20  # blocks of 30 columns
    idx = np.sort(np.argsort(rng.random((cells, g)), 1)[:, :per_row], 1).astype(np.uint32)
    values = rng.gamma(2.0, 1.0, idx.shape) * (1.0 + 3.0 * (idx % 7 == (np.arange(cells) % 7)[:, None]))
    x = O.Csr(np.arange(cells + 1, dtype=np.uint64) * np.uint64(per_row), idx.reshape(-1),
              values.astype(np.float32).reshape(-1), g)
    got, want = K.pca(x.indptr, x.indices, x.values, g, k), O.pca(x, k)
    assert got.passes_run == want.passes_run
    assert np.max(np.abs(got.variance - want.variance)) <= 1e-9 * want.variance[0]
