"""The source size of a 16-byte copy near and far from the end of its array: never past the end, whole
pieces before it, up to the largest CSR operand (2^31 - 2 nonzeros).  The header is compiled for the host."""
import ctypes as C
import subprocess

import pytest

from plamatrix_b200 import build

FAR = [1 << 27, (1 << 28) - 1, 1 << 28, (1 << 28) + 1, (1 << 29) - 1, 1 << 29, (1 << 29) + 1, 300_000_000,
       (1 << 30) + 3, (1 << 31) - 2]


@pytest.fixture(scope="module")
def piece_bytes(tmp_path_factory):
    folder = tmp_path_factory.mktemp("piece")
    source, library = folder / "piece.cpp", folder / "piece.so"
    source.write_text('#include "pm_piece.h"\n'
                      'extern "C" int piece_bytes(int left, int size) { return pm::piece_bytes(left, size); }\n')
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I", build.CSRC, str(source), "-o", str(library)],
                   check=True)
    return C.CDLL(str(library)).piece_bytes


@pytest.mark.parametrize("size", [4, 8])
@pytest.mark.parametrize("left", [1, 2, 3, 4, 5, 31] + FAR)
def test_source_size(piece_bytes, left, size):
    assert piece_bytes(left, size) == min(16, left * size)
