"""kg_connectivities into output arrays of every kind: device, host, some of each, and device addresses
that a copy takes but a kernel cannot write to (not a multiple of the element's size)."""

import ctypes

import numpy as np
import pytest

import kyto_b200 as K
from oracle import connectivities as OC

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

N, KN = 300, 9


@pytest.fixture(scope="module")
def graph():
    rng = np.random.default_rng(2)
    cols = np.sort(np.stack([rng.permutation(N)[:KN] for _ in range(N)]), 1).astype(np.uint32)
    dist = rng.uniform(1.0, 2.0, (N, KN)).astype(np.float32)
    indptr = np.arange(N + 1, dtype=np.uint64) * np.uint64(KN)
    return indptr, cols.reshape(-1), dist.reshape(-1)


@pytest.mark.parametrize("where", ["ddd", "hhh", "dhh", "hdd", "ddh"])
@pytest.mark.parametrize("skew", [(0, 0, 0), (4, 0, 0), (0, 2, 0), (0, 0, 1), (1, 3, 2)])
def test_every_kind_of_output(graph, where, skew):
    sizes = (8 * (N + 1), 8 * N * KN, 8 * N * KN)
    bufs = [torch.zeros(size + 8, dtype=torch.uint8, device="cuda" if w == "d" else "cpu")
            for size, w in zip(sizes, where)]
    torch.cuda.synchronize()  # the library's stream does not wait for torch's
    nnz = ctypes.c_uint64()
    K._check(K.library().kg_connectivities(
        K.default_context().handle, *(a.ctypes.data for a in graph), N, KN + 1,
        *(b.data_ptr() + o for b, o in zip(bufs, skew)), ctypes.byref(nnz)))
    want = OC.connectivities(*graph, KN + 1)
    assert nnz.value == want[1].size
    got = [b.cpu().numpy()[o:o + size].tobytes() for b, o, size in zip(bufs, skew, sizes)]
    assert got[0] == want[0].astype(np.uint64).tobytes()
    assert got[1][:4 * nnz.value] == want[1].astype(np.uint32).tobytes()
    weights = np.frombuffer(got[2][:4 * nnz.value], dtype=np.float32)
    assert np.abs(weights.astype(np.float64) - want[2]).max() <= 1e-6
