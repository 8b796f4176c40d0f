"""Gene moments of tiny f32 values behind many rows that hold nothing of their gene: zeros add nothing
to a sum of squares, however many there are (2^19 rows; the sums are exact here, so bits)."""

import ctypes
import math

import numpy as np
import pytest

import kyto_b200 as K

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

ROWS, GENES, PER_ROW = 1 << 19, 300, 290


@pytest.mark.parametrize("value", [2.0**-28, 1.5 * 2.0**-28, 2.0**-27, 1.25 * 2.0**-27, 2.0**-26,
                                   2.0**-20])
def test_zeros_before_a_small_value_add_nothing(value):
    value = float(np.float32(value) * np.float32(1 + 2.0**-20))
    # Every row holds genes 1 .. PER_ROW; the last one gene 0 too, behind all the others.
    indptr = torch.arange(ROWS + 1, dtype=torch.int64, device="cuda") * PER_ROW
    indptr[-1] += 1
    idx = torch.arange(1, PER_ROW + 1, dtype=torch.int32, device="cuda").repeat(ROWS)
    last = (ROWS - 1) * PER_ROW
    idx = torch.cat([idx[:last], torch.zeros(1, dtype=torch.int32, device="cuda"), idx[last:]])
    values = torch.full((idx.numel(),), 0.5, dtype=torch.float32, device="cuda")
    values[last] = value
    out = [torch.empty(GENES, dtype=t, device="cuda")
           for t in (torch.float64, torch.float64, torch.int64)]
    torch.cuda.synchronize()  # the library's stream does not wait for torch's
    K._check(K.library().kg_hvg_moments(
        K.default_context().handle, indptr.data_ptr(), idx.data_ptr(), values.data_ptr(), K.KG_F32,
        ROWS, GENES, ctypes.c_double(math.nan), 0, *(o.data_ptr() for o in out)))
    sums, squares, positives = (o.cpu().numpy() for o in out)
    t = np.float32(math.expm1(value))
    assert positives[0] == 1 and sums[0] == np.float64(t)
    assert squares[0] == np.float64(t * t)
    half = np.float32(math.expm1(0.5))
    assert positives[1] == ROWS and sums[1] == ROWS * np.float64(half)
    assert squares[1] == ROWS * np.float64(half * half)
    assert positives[-1] == 0 and sums[-1] == 0.0 and squares[-1] == 0.0
