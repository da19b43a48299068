"""The hardware logarithm behind the AL8 codes: the error bound that decides which codes are taken exactly, against every
normal positive binary32 number.  The function and the bound come from the kernel's own header, compiled here."""
import ctypes
import importlib.util
import os
import subprocess

import pytest
import torch

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = r"""
#include "common.cuh"
#include "fullrank_fast.cuh"

// largest |lg2.approx(x) - log2(x)| over its bound, as the bits of a binary64 number (non-negative: they order like it)
__global__ void sweep(unsigned long long *worst, unsigned long long *seen)
{
    double most = 0.0;
    unsigned long long n = 0;
    for (uint32_t b = 0x00800000u + blockIdx.x * blockDim.x + threadIdx.x; b < 0x7f800000u; b += gridDim.x * blockDim.x, ++n) {
        const float x = __uint_as_float(b);
        const double l = log2((double)x), bound = (double)af8::LG2_REL * fabs(l) + (double)af8::LG2_ABS;
        const double ratio = fabs((double)af8::lg2_approx(x) - l) / bound;
        most = ratio <= most ? most : ratio;                       // (a NaN stays)
    }
    atomicMax(worst, (unsigned long long)__double_as_longlong(most));
    atomicAdd(seen, n);
}

extern "C" __attribute__((visibility("default"))) int lg2_sweep(unsigned long long *out, void *stream)
{
    sweep<<<148 * 8, 256, 0, static_cast<cudaStream_t>(stream)>>>(out, out + 1);
    return (int)cudaGetLastError();
}
"""


def test_lg2_approx_stays_within_its_bound_for_every_normal_number(tmp_path):
    spec = importlib.util.spec_from_file_location("af8_build", os.path.join(ROOT, "adafactor-8bit_b200", "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    source, lib = tmp_path / "sweep.cu", tmp_path / "libsweep.so"
    source.write_text(SOURCE)
    subprocess.run([os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")] + build.NVCC_FLAGS + ["-I", build.CSRC, "-I", build.INCLUDE,
                   "-o", str(lib), str(source)], check=True)
    out = torch.zeros(2, dtype=torch.int64, device="cuda")
    assert ctypes.CDLL(str(lib)).lg2_sweep(ctypes.c_void_p(out.data_ptr()), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    worst, seen = out.cpu()
    assert int(seen) == 0x7f800000 - 0x00800000
    assert 0.5 < float(worst.view(torch.float64)) <= 1.0
