"""A launch that the device cannot hold at once is refused before anything runs: the caller learns it and no
error is left for the next launch.  The header is compiled into a small library of its own."""
import ctypes as C
import subprocess

import pytest
import torch

from plamatrix_b200 import build

pytestmark = pytest.mark.gpu

SOURCE = """
#include "pm_grid.cuh"
namespace pm { void count_launch() {} void set_last_error(const std::string&) {} }
__global__ void mark(int* at) { if (blockIdx.x == 0 && threadIdx.x == 0) *at += 1; }
extern "C" __attribute__((visibility("default"))) int try_launch(unsigned ctas, int* at)
{
    void* args[] = {&at};
    const bool ran = pm::launch_resident(reinterpret_cast<const void*>(mark), ctas, 1024, args, 0, nullptr);
    return (ran ? 1 : 0) | (cudaGetLastError() == cudaSuccess ? 0 : 2) |
           (cudaStreamSynchronize(nullptr) == cudaSuccess ? 0 : 4);
}
"""


def test_refused_launch(tmp_path):
    source, library = tmp_path / "launch.cu", tmp_path / "launch.so"
    source.write_text(SOURCE)
    subprocess.run([build.NVCC, *build.ARCH, *build.FLAGS, "-shared", "-o", str(library), str(source)], check=True)
    lib = C.CDLL(str(library))
    at = torch.zeros(1, dtype=torch.int32, device="cuda")
    for ctas, ran in ((148, 1), (1 << 20, 0), (1, 1)):
        before = int(at)
        assert lib.try_launch(C.c_uint(ctas), C.c_void_p(at.data_ptr())) == ran
        assert int(at) == before + ran
