"""Which grid arrays the coefficient kernel reads where they stand
(grid_in_place of csrc/vert_grid.cuh, compiled as plain C++): a null pointer,
another device's memory and an unaligned address are left to the copy."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

SOURCE = """
#include "vert_grid.cuh"
extern "C" int in_place(unsigned long long p, int err, int type, int at, int device) {
  cudaPointerAttributes a{};
  a.type = cudaMemoryType(type);
  a.device = at;
  return gv::grid_in_place(reinterpret_cast<const void*>(p), cudaError_t(err), a, device);
}
"""
UNREGISTERED, HOST, DEVICE, MANAGED = range(4)  # cudaMemoryType


@pytest.fixture(scope="module")
def in_place(tmp_path_factory):
    import ctypes
    d = tmp_path_factory.mktemp("grid")
    src, so = d / "g.cpp", d / "g.so"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", f"-I{CUDA}/include",
                    "-I" + os.path.join(ROOT, "gitm_b200", "csrc"), str(src), "-o", str(so)], check=True)
    f = ctypes.CDLL(str(so)).in_place
    f.argtypes = [ctypes.c_ulonglong] + [ctypes.c_int] * 4
    return f


@pytest.mark.parametrize("p,err,kind,at,device,want", [
    (0x7f0000000200, 0, DEVICE, 0, 0, 1), (0x7f0000000208, 0, DEVICE, 3, 3, 1), (0x7f0000000200, 0, MANAGED, 1, 0, 1),
    (0, 0, DEVICE, 0, 0, 0), (0, 0, UNREGISTERED, -2, 0, 0),  # a null pointer
    (0x7f0000000200, 0, DEVICE, 1, 0, 0),  # another device's memory
    (0x7f0000000204, 0, DEVICE, 0, 0, 0), (0x7f0000000201, 0, MANAGED, 0, 0, 0),  # no address of a double
    (0x7f0000000200, 0, HOST, 0, 0, 0), (0x7f0000000200, 0, UNREGISTERED, -2, 0, 0),
    (0x7f0000000200, 1, DEVICE, 0, 0, 0)])
def test_grid_in_place(in_place, p, err, kind, at, device, want):
    assert bool(in_place(p, err, kind, at, device)) == bool(want)
