"""Kernel attributes set once per device: a failed attempt is not remembered."""

import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bldfm_gb300", "csrc")
CUDA_INC = "/usr/local/cuda/include"

PROGRAM = r"""
#include "devattr.h"
#include <stdio.h>
int main()
{
    std::atomic<uint64_t> mask{0};
    int calls = 0;
    cudaError_t next = cudaErrorInvalidValue;
    auto set = [&] { ++calls; return next; };
    printf("%d", set_once(mask, 1, set) == cudaErrorInvalidValue);  // fails: reported
    next = cudaSuccess;
    printf(" %d", set_once(mask, 1, set) == cudaSuccess && calls == 2);  // and tried again
    printf(" %d", set_once(mask, 1, set) == cudaSuccess && calls == 2);  // once it has succeeded, no more
    printf(" %d", set_once(mask, 0, set) == cudaSuccess && calls == 3);  // another device is its own
    next = cudaErrorInvalidValue;
    printf(" %d", set_once(mask, 1, set) == cudaSuccess && calls == 3);  // ... also when that one fails
    next = cudaSuccess;
    set_once(mask, 64, set);
    set_once(mask, 64, set);
    printf(" %d\n", calls == 5);  // no flag for it: set every time
    return 0;
}
"""


@pytest.mark.skipif(not (shutil.which("g++") and os.path.isdir(CUDA_INC)), reason="needs g++ and the CUDA headers")
def test_failed_attribute_is_set_again(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    # the functions that call the CUDA runtime are not used: nothing to link
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, "-I", CUDA_INC, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split() == ["1"] * 6
