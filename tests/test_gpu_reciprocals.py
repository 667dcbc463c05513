"""The kernels' reciprocals and divisions without range tests (rcp_near and div_by,
csrc/shade_common.cuh) against the IEEE routines, bit for bit: every reciprocal of the range, every
pixel of every image size, and a thousand million quotients spread over the range."""
import os
import subprocess

import pytest

import build as vbuild

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <cstdint>
#include "shade_common.cuh"
using namespace vrt;
__device__ unsigned long long checked[3], wrong[3];
__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }
__device__ void count(int what, unsigned n, unsigned bad) { atomicAdd(checked + what, n); if (bad) atomicAdd(wrong + what, bad); }
// block (m, e): 2^13 mantissas of exponent e - 41, both signs
__global__ void reciprocals() {
    unsigned bad = 0, n = 0;
    for (unsigned i = threadIdx.x; i < 8192; i += blockDim.x)
        for (unsigned s = 0; s < 2; s++, n++) {
            const float b = __uint_as_float(s << 31 | (blockIdx.y + 127 - 41) << 23 | blockIdx.x << 13 | i);
            bad += !same(rcp_near(b), frcp(b));
        }
    count(0, n, bad);
}
// block w: an image of width w + 1
__global__ void pixels() {
    unsigned bad = 0, n = 0;
    const float w = (float)(blockIdx.x + 1), inv = frcp(w);
    for (unsigned x = threadIdx.x; x <= blockIdx.x; x += blockDim.x, n++) {
        const float a = (float)(2 * x + 1);
        bad += !same(div_by(a, w, inv), fdiv(a, w));
    }
    count(1, n, bad);
}
__device__ uint64_t mix(uint64_t z) {  // splitmix64
    z += 0x9e3779b97f4a7c15ull;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}
// a = +0 or 2^-60 <= |a| < 2^20, 2^-40 <= |b| <= 2, mantissas of every kind: random, few bits, all but few bits
__global__ void quotients() {
    unsigned bad = 0, n = 0;
    for (unsigned i = 0; i < 1024; i++, n++) {
        const uint64_t r = mix((uint64_t)i << 40 | (uint64_t)blockIdx.x << 10 | threadIdx.x), q = mix(r);
        uint32_t ma = r & 0x7fffff, mb = r >> 23 & 0x7fffff;
        const unsigned kind = q & 15;
        if (kind & 1) ma &= 0x7fffff << (q >> 4 & 31) % 23;
        if (kind & 2) mb &= 0x7fffff << (q >> 9 & 31) % 23;
        if (kind & 4) ma = ~ma & 0x7fffff;
        if (kind & 8) mb = ~mb & 0x7fffff;
        const uint32_t ea = 127 - 60 + (q >> 14 & 127) % 80;
        uint32_t eb = 127 - 40 + (q >> 21 & 63) % 42;
        if (eb == 128) mb = 0;  // 2 itself
        float a = __uint_as_float((uint32_t)(q >> 40 & 1) << 31 | ea << 23 | ma);
        const float b = __uint_as_float((uint32_t)(q >> 41 & 1) << 31 | eb << 23 | mb);
        if ((q >> 42 & 255) == 0) a = 0.0f;
        bad += !same(div_by(a, b, frcp(b)), fdiv(a, b));
    }
    count(2, n, bad);
}
int main() {
    reciprocals<<<dim3(1024, 43), 256>>>();
    pixels<<<32768, 128>>>();
    quotients<<<4096, 256>>>();
    unsigned long long c[3], w[3];
    if (cudaDeviceSynchronize() != cudaSuccess || cudaMemcpyFromSymbol(c, checked, sizeof c) != cudaSuccess ||
        cudaMemcpyFromSymbol(w, wrong, sizeof w) != cudaSuccess)
        return 1;
    for (int i = 0; i < 3; i++) std::printf("%llu %llu\n", c[i], w[i]);
    return 0;
}
"""


def test_reciprocals_and_quotients_round_as_ieee(cuda, tmp_path):
    src, exe = tmp_path / "main.cu", str(tmp_path / "main")
    src.write_text(PROGRAM)
    subprocess.run([vbuild.NVCC] + vbuild.ARCH + ["-O3", "--fmad=false", "-std=c++17", "-I" + vbuild.CSRC,
                                                   "-I" + os.path.join(ROOT, "include"), str(src), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120, check=True).stdout.split()
    n = [int(v) for v in out]
    assert n[0::2] == [43 * (1 << 24), 32768 * 32769 // 2, 4096 * 256 * 1024]
    assert n[1::2] == [0, 0, 0]
