"""Kernel attributes are set on every device that is used, not once per process (on the host, with a counterfeit
``cudaGetDevice``)."""

from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "density-functional-theory-on-real-space-grids_b200" / "csrc"

PROGRAM = r"""
#include "per_device.cuh"
#include <stdio.h>
static int current = 0;
extern "C" cudaError_t cudaGetDevice(int* d) {
    if (current < 0) return cudaErrorNoDevice;
    *d = current;
    return cudaSuccess;
}
namespace cdftb { thread_local int g_last_cuda_error = 0; unsigned long long g_launch_count = 0; }
int main() {
    cdftb::OncePerDevice once;
    int calls = 0, status = CDFTB_OK;
    auto on = [&](int device) {
        current = device;
        const int st = once.run([&] { ++calls; return status; });
        printf("%d:%d ", st, calls);
    };
    on(0); on(0);              // set once
    on(1); on(1); on(0);       // and once on another device
    status = CDFTB_ERR_LAUNCH;
    on(2);                     // a failure is not remembered
    status = CDFTB_OK;
    on(2); on(2);
    on(63); on(63); on(64); on(64);
    on(-1);
}
"""


def test_a_setting_is_made_on_each_device(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    gxx = shutil.which("g++")
    include = Path(nvcc).resolve().parents[1] / "include"
    if gxx is None or not (include / "cuda_runtime.h").exists():
        pytest.skip("no g++ or CUDA headers")
    source = tmp_path / "once.cpp"
    source.write_text(PROGRAM)
    subprocess.run([gxx, "-std=c++17", "-I", str(CSRC), "-I", str(include), str(source), "-o", str(tmp_path / "once")],
                   check=True)
    out = subprocess.run([str(tmp_path / "once")], check=True, capture_output=True, text=True).stdout.split()
    # status:calls so far
    assert out == ["0:1", "0:1", "0:2", "0:2", "0:2", "2:3", "0:4", "0:4", "0:5", "0:5", "0:6", "0:7", "2:7"]


@pytest.mark.parametrize("source", sorted(p.name for p in CSRC.glob("*.cu")))
def test_no_attribute_is_set_once_per_process(source):
    text = (CSRC / source).read_text()
    assert "static bool" not in text
