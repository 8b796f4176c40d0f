"""One allocation attempt that fails, where there is another way: a size that was rounded up is asked
for as it is. (Failures that stay are in test_gpu_errors.)"""

import numpy as np
import pytest

import kyto_b200 as K

pytestmark = pytest.mark.gpu

ONE = 1 << 63


@pytest.fixture(autouse=True)
def _off():
    yield
    K.fail_allocations(None)


@pytest.mark.parametrize("count", [262_144, 262_145, 300_001, 5_000_003])
def test_a_rounded_size_is_asked_for_as_it_is(count):
    """Host arrays: the offsets (small, never rounded), the values and the output (from 1 MB on)."""
    values = np.arange(count, dtype=np.uint32) % 50
    indptr = np.array([0, count // 3, count], dtype=np.uint64)
    want = K.normalize_log1p(indptr, values)
    unit = 1 << 17
    while unit < 64 << 20 and unit * 16 <= 4 * count:
        unit <<= 1
    rounded = 4 * count % unit != 0
    for attempt in (1, 2):
        K.fail_allocations(ONE | attempt)
        if rounded:
            assert np.array_equal(K.normalize_log1p(indptr, values), want)
        else:
            with pytest.raises(K.KytoError) as err:
                K.normalize_log1p(indptr, values)
            assert err.value.status == K.KG_ERR_OOM
    K.fail_allocations(ONE)  # the offsets
    with pytest.raises(K.KytoError) as err:
        K.normalize_log1p(indptr, values)
    assert err.value.status == K.KG_ERR_OOM
    assert np.array_equal(K.normalize_log1p(indptr, values), want)


def test_a_search_out_of_memory_for_its_lists_goes_without():
    """Each attempt of a search fails once: the answer is the graph or KG_ERR_OOM, and the graph
    wherever the scan's lists had been begun (all but the few attempts before them and the output's
    after)."""
    x = np.random.default_rng(0).normal(size=(6000, 20)).astype(np.float32)
    want = K.neighbors(x, 10)
    out_of_memory = []
    for attempt in range(200):  # more than a search makes
        K.fail_allocations(ONE | attempt)
        try:
            got = K.neighbors(x, 10)
        except K.KytoError as err:
            assert err.status == K.KG_ERR_OOM
            out_of_memory.append(attempt)
        else:
            assert np.array_equal(got.indices, want.indices)
            assert np.array_equal(got.distances, want.distances)
    assert max(out_of_memory) < 199
    listed = [a for a in range(max(out_of_memory)) if a not in out_of_memory]
    # The lists' own attempts come one after another, from the clustering to the filter's end.
    assert len(listed) >= 40 and listed == list(range(listed[0], listed[-1] + 1))


def test_a_product_out_of_memory_for_its_groups_goes_without():
    """A product's groups (300 rows x 4 groups x 256 bytes: never rounded) are worth having, not
    needed: the whole segments give the same bits. Eleven passes, a product of X in ten of them."""
    rng = np.random.default_rng(1)
    rows, genes, per_row = 300, 2000, 200
    idx = np.sort(np.argsort(rng.random((rows, genes)), 1)[:, :per_row], 1).astype(np.uint32)
    indptr = np.arange(rows + 1, dtype=np.uint64) * np.uint64(per_row)
    values = rng.uniform(0.5, 2.0, idx.size).astype(np.float32)

    def run():
        sess = K.PcaSession(5, genes)
        sess.push(indptr, idx.reshape(-1), values)
        sess.run()
        assert sess.stats().product_launches > 0
        return sess.results()

    want = run()
    out_of_memory = []
    for attempt in range(600):  # more than a run makes
        K.fail_allocations(ONE | attempt)
        try:
            got = run()
        except K.KytoError as err:
            assert err.status == K.KG_ERR_OOM
            out_of_memory.append(attempt)
        else:
            assert np.array_equal(got.variance, want.variance)
            assert np.array_equal(got.embedding, want.embedding)
    assert max(out_of_memory) < 599
    assert max(out_of_memory) + 1 - len(out_of_memory) >= 10
