"""Kernel attributes are set once on each device (csrc/kg_once.cuh, compiled here as host code), and
every kernel's limit of shared memory goes that way: a process that opens a second device has to set
it there too."""

import ctypes
import re
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "kyto_b200" / "csrc"
SOURCE = """
#include <stdexcept>
#include "kg_once.cuh"
static kg::OncePerDevice once;
static int calls = 0;
extern "C" int set_on(long key, int device, int fails) {
  try {
    once(reinterpret_cast<const void*>(key), device, [&] {
      ++calls;
      if (fails) throw std::runtime_error("not set");
    });
  } catch (const std::runtime_error&) {
    return -1;
  }
  return calls;
}
"""


def test_each_device_once(tmp_path):
    (tmp_path / "once.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}",
                    str(tmp_path / "once.cpp"), "-o", str(tmp_path / "once.so")], check=True)
    set_on = ctypes.CDLL(str(tmp_path / "once.so")).set_on
    assert [set_on(1, 0, 0), set_on(1, 0, 0)] == [1, 1]
    assert [set_on(1, 1, 0), set_on(1, 1, 0)] == [2, 2]  # the same kernel, another device
    assert [set_on(2, 0, 1), set_on(2, 0, 0), set_on(2, 0, 0)] == [-1, 4, 4]  # tried again
    assert set_on(1, 0, 0) == 4


def test_no_kernel_sets_its_own_limit():
    own = {f.name for f in CSRC.iterdir()
           if re.search(r"cudaFuncAttributeMaxDynamicSharedMemorySize", f.read_text())}
    assert own == {"kg_context.cu"}
