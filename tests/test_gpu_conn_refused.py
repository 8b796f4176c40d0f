"""Graphs that kg_connectivities refuses, as device arrays: another number of neighbours than the
graph holds, a row of another length, columns out of order or out of range (the largest u32 among
them). Every array is long enough for n_rows x (n_neighbors - 1) entries. A refused call leaves
the outputs and the count as they were, and the next call works."""

import ctypes

import numpy as np
import pytest

import kyto_b200 as K
from oracle import connectivities as OC

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _call(indptr, cols, dist, n, neighbors, entries):
    out = (torch.full((n + 1,), 7, dtype=torch.int64, device="cuda"),
           torch.full((2 * entries,), 7, dtype=torch.int32, device="cuda"),
           torch.full((2 * entries,), 7.0, dtype=torch.float32, device="cuda"))
    dev = [torch.from_numpy(a).cuda() for a in (indptr.view(np.int64), cols.view(np.int32), dist)]
    torch.cuda.synchronize()  # the library's stream does not wait for torch's
    nnz = ctypes.c_uint64(7)
    status = K.library().kg_connectivities(
        K.default_context().handle, *(t.data_ptr() for t in dev), n, neighbors,
        *(t.data_ptr() for t in out), ctypes.byref(nnz))
    return status, out, nnz.value


def _graph(n, k):
    rng = np.random.default_rng(n + k)
    cols = np.sort(np.stack([rng.permutation(n)[:k] for _ in range(n)]), 1).astype(np.uint32)
    dist = rng.uniform(1.0, 2.0, (n, k)).astype(np.float32)
    return np.arange(n + 1, dtype=np.uint64) * np.uint64(k), cols.reshape(-1), dist.reshape(-1)


@pytest.mark.parametrize("k,neighbors", [(9, 15), (14, 10), (40, 50), (14, 34)])
def test_another_number_of_neighbors(k, neighbors):
    n, most = 500, max(k, neighbors - 1)
    indptr, cols, dist = _graph(n, k)
    long_cols, long_dist = np.zeros(n * most, dtype=np.uint32), np.zeros(n * most, dtype=np.float32)
    long_cols[:n * k], long_dist[:n * k] = cols, dist
    status, out, nnz = _call(indptr, long_cols, long_dist, n, neighbors, n * most)
    assert status == K.KG_ERR_INVALID and nnz == 7
    assert all(bool((t == 7).all()) for t in out)


@pytest.mark.parametrize("k", [14, 32, 33, 200])
@pytest.mark.parametrize("fault", ["row", "last", "order", "equal", "range", "largest"])
def test_a_row_out_of_shape(k, fault):
    n = 400
    indptr, cols, dist = _graph(n, k)
    row = 257
    if fault == "row":
        indptr[row] += np.uint64(1)
    elif fault == "last":
        indptr[n] -= np.uint64(1)
    elif fault == "order":
        cols[row * k:row * k + 2] = cols[row * k:row * k + 2][::-1]
    elif fault == "equal":
        cols[row * k + 1] = cols[row * k]
    elif fault == "range":
        cols[row * k + k - 1] = n
    else:  # in every row, the last one too
        cols[k - 1::k] = 0xFFFFFFFF
    status, out, nnz = _call(indptr, cols, dist, n, k + 1, n * k)
    assert status == K.KG_ERR_INVALID and nnz == 7
    assert all(bool((t == 7).all()) for t in out)
    indptr, cols, dist = _graph(n, k)
    status, out, nnz = _call(indptr, cols, dist, n, k + 1, n * k)
    want = OC.connectivities(indptr, cols, dist, k + 1)
    assert status == K.KG_OK and nnz == want[1].size
    assert np.array_equal(out[0].cpu().numpy().view(np.uint64), want[0])
    assert np.array_equal(out[1][:nnz].cpu().numpy().view(np.uint32), want[1])


@pytest.mark.parametrize("k,neighbors", [(9, 15), (14, 10)])
def test_host_arrays_of_another_number_of_neighbors(k, neighbors):
    """Host arrays as long as the graph they hold."""
    n = 500
    graph = _graph(n, k)
    most = 2 * n * max(k, neighbors)
    out = np.zeros(n + 1, dtype=np.uint64), np.zeros(most, dtype=np.uint32), np.zeros(most, np.float32)
    nnz = ctypes.c_uint64(7)
    status = K.library().kg_connectivities(
        K.default_context().handle, *(a.ctypes.data for a in graph), n, neighbors,
        *(a.ctypes.data for a in out), ctypes.byref(nnz))
    assert status == K.KG_ERR_INVALID and nnz.value == 7
    assert not any(a.any() for a in out)
