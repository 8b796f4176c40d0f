"""The order of a Krylov block's columns by their norms (csrc/kg_order.cuh, compiled here as host
code): whatever the norms hold, counting the columns before each one has to give every place once,
since a kernel indexes its arrays with what stands at each place."""

import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "kyto_b200" / "csrc"
SOURCE = """
#include "kg_order.cuh"
extern "C" int before(double na, uint32_t a, double nb, uint32_t b) {
  return kg::column_before(na, a, nb, b) ? 1 : 0;
}
"""


@pytest.fixture(scope="module")
def before(tmp_path_factory):
    d = tmp_path_factory.mktemp("order")
    (d / "order.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", f"-I{CSRC}",
                    str(d / "order.cpp"), "-o", str(d / "order.so")], check=True)
    fn = ctypes.CDLL(str(d / "order.so")).before
    fn.argtypes = [ctypes.c_double, ctypes.c_uint32, ctypes.c_double, ctypes.c_uint32]
    return fn


NAN, INF = float("nan"), float("inf")


@pytest.mark.parametrize("norms", [
    [1.0, NAN, 2.0], [NAN, NAN, NAN], [NAN, 0.0], [0.0, 0.0, NAN, 0.0], [INF, NAN, INF, 1.0],
    [3.0, 3.0, 1.0, 3.0], [2.0, 5.0, 1.0, 5.0], list(np.where(np.arange(60) % 7 == 3, np.nan,
                                                              np.arange(60) % 5.0))])
def test_every_place_once_and_descending(before, norms):
    w = len(norms)
    place = [sum(before(norms[o], o, norms[c], c) for o in range(w)) for c in range(w)]
    assert sorted(place) == list(range(w))
    order = np.argsort(place)
    held = [norms[c] for c in order if norms[c] == norms[c]]
    assert held == sorted(held, reverse=True)
    assert all(np.isnan(norms[c]) for c in order[len(held):])
    for a, b in zip(order, order[1:]):  # ties to the lower column
        if norms[a] == norms[b] or (np.isnan(norms[a]) and np.isnan(norms[b])):
            assert a < b
