"""The rows that a CTA of the several-element row solves takes follow the device's
multiprocessors."""
import os
import subprocess

from mpi_b200 import build as B

SRC = """
#include <cstdio>
#include <cstdlib>
#include "helm_multi.cuh"
int main(int argc, char** argv)
{
    for (int i = 1; i + 2 < argc; i += 3)
        std::printf("%d\\n", helm::multi_rows_per_cta(std::atoi(argv[i]), std::atoi(argv[i + 1]), std::atoi(argv[i + 2])));
}
"""


def test_rows_per_cta(tmp_path):
    src, exe = tmp_path / "shape.cpp", tmp_path / "shape"
    src.write_text(SRC)
    cuda = os.path.join(os.path.dirname(os.path.dirname(B.NVCC)), "include")
    subprocess.run(["g++", "-std=c++17", "-I", B.CSRC, "-I", cuda, str(src), "-o", str(exe)], check=True)
    # (rows, elements, multiprocessors) -> two CTAs a multiprocessor, at most 64 vectors each
    cases = {(257, 52, 148): 1, (1056, 25, 148): 2, (2112, 6, 148): 8, (1056, 4, 148): 4, (1056, 4, 74): 8,
             (1056, 4, 16): 16, (5, 2, 148): 1, (100000, 64, 148): 1, (100000, 2, 148): 32}
    out = subprocess.run([str(exe)] + [str(v) for c in cases for v in c], capture_output=True, text=True, check=True)
    assert [int(v) for v in out.stdout.split()] == list(cases.values())
