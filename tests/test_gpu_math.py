"""The step's short evaluations of the friction power and the Horton
exponential give the full evaluations' F32 bits: every F32 argument of their
ranges, and arguments beyond them (where they hand over to the full one)."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CSRC = Path(__file__).resolve().parents[1] / 'nh-flood-2d_b200' / 'csrc'
SOURCE = r'''
#include <cuda_runtime.h>
#include "%s/nhf_math.cuh"
__device__ unsigned long long differ;
template <int kWhich>
__global__ void k_compare(uint32_t first, uint32_t count)
{
    unsigned long long bad = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        const float x = __uint_as_float(first + i);
        const float a = kWhich ? nhf::horton_exp(x) : nhf::friction_pow(x);
        const float b = kWhich ? nhf::exp_f32(x) : nhf::pow_f32(x, (float)(7.0 / 3.0));
        bad += __float_as_uint(a) != __float_as_uint(b);
    }
    if (bad) atomicAdd(&differ, bad);
}
extern "C" int compare(int which, uint32_t first, uint32_t count, unsigned long long *out)
{
    unsigned long long zero = 0;
    cudaMemcpyToSymbol(differ, &zero, 8);
    if (which) k_compare<1><<<148 * 8, 256>>>(first, count);
    else k_compare<0><<<148 * 8, 256>>>(first, count);
    cudaMemcpyFromSymbol(out, differ, 8);
    return (int)cudaGetLastError();
}
'''


@pytest.fixture(scope='module')
def compare(cuda_available, tmp_path_factory):
    from nhflood.build import ARCH, nvcc
    path = tmp_path_factory.mktemp('math')
    (path / 'math.cu').write_text(SOURCE % CSRC)
    subprocess.run([nvcc(), *ARCH, '-O3', '--fmad=false', '-std=c++17', '-Xcompiler', '-fPIC', '-shared',
                    '-o', str(path / 'math.so'), str(path / 'math.cu')], check=True)
    lib = ctypes.CDLL(str(path / 'math.so'))
    lib.compare.argtypes = [ctypes.c_int, ctypes.c_uint32, ctypes.c_uint32, ctypes.POINTER(ctypes.c_ulonglong)]

    def run(which, low, high):
        a, b = (int(np.float32(v).view(np.uint32)) for v in (low, high))
        out = ctypes.c_ulonglong()
        assert lib.compare(which, a, b - a + 1, ctypes.byref(out)) == 0
        return out.value
    return run


@pytest.mark.parametrize('low, high', [(1e-5, 1.0), (1.0, 2.0 ** 20), (2.0 ** 20, np.inf)])
def test_friction_power_bits(compare, low, high):
    assert compare(0, low, high) == 0


@pytest.mark.parametrize('low, high', [(0.0, -1e-30), (-1e-30, -1.0), (-1.0, -80.0), (-80.0, -np.inf), (-0.0, -0.0)])
def test_horton_exponential_bits(compare, low, high):
    low = -0.0 if low == 0.0 else low
    assert compare(1, low, high) == 0
