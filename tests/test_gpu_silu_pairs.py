"""The paired SiLU of the large-batch epilogue against the scalar statement, for every one of the 2^32 arguments: the device
functions themselves, compiled from the library's header into a small program.  Every argument that the paired form is for (+0 and
magnitudes of 2^-40 to 80) has the scalar form's bits in either half of a pair; every argument beyond the upper end has to be told
by the look at the largest magnitude, in any place of a group of four.  The lower end is the scales': the smallest products of a
sum and two scales that the epilogue takes the fast way with are checked too."""
import ctypes as C
import subprocess

import pytest

from rknpu2_matmul_open_b200 import build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "w4a8_math.cuh"
using namespace rkb200;
// counts[0]: arguments whose paired value differs; [1]: groups wrongly told to be in range or not; [2]: arguments of the paired form
__global__ void check(unsigned long long* counts)
{
    unsigned long long wrong = 0, misjudged = 0, plain_count = 0;
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < (1ull << 32); i += (unsigned long long)gridDim.x * blockDim.x) {
        const uint32_t u = (uint32_t)i;
        const float g = __uint_as_float(u), magnitude = fabsf(g);
        const bool within = magnitude <= 80.f;                                              // false for NaN
        const bool plain = u == 0u || (magnitude >= 9.094947017729282e-13f && within);      // +0 and 2^-40 .. 80
        // plain neighbours: another exponent, sign and mantissa for every argument
        const uint32_t mix = u * 2654435761u;
        const float n0 = __uint_as_float((mix & 0x807fffffu) | ((100u + (mix >> 9) % 32u) << 23)), n1 = -2.5f, n2 = 0.0625f;
        const float four[4] = {g, n0, n1, n2};
#pragma unroll
        for (int at = 0; at < 4; ++at) {
            const float a = four[at & 3], b = four[(at + 1) & 3], c = four[(at + 2) & 3], d = four[(at + 3) & 3];
            if (silu_fast(max_abs(max_abs(a, b), max_abs(c, d))) != within) ++misjudged;
        }
        // scales of at least 2^-20 (the bits of u spread over the 24 smallest exponents from there on), a sum of one
        const float s0 = __uint_as_float((107u + u % 24u) << 23 | (mix >> 9)), s1 = __uint_as_float((107u + (u >> 16) % 24u) << 23 | (u & 0x7fffffu));
        if (!(__fmul_rn(__fmul_rn(1.f, s0), s1) >= 9.094947017729282e-13f)) ++misjudged;
        if (plain) {
            ++plain_count;
            const uint32_t want = __float_as_uint(silu_poly(g));
            float first, second, other;
            minus_silu_poly2(g, n0, first, other);
            minus_silu_poly2(n0, g, other, second);
            if (__float_as_uint(-first) != want || __float_as_uint(-second) != want) ++wrong;
        }
    }
    atomicAdd(&counts[0], wrong);
    atomicAdd(&counts[1], misjudged);
    atomicAdd(&counts[2], plain_count);
}
extern "C" int run(unsigned long long* out)
{
    unsigned long long* counts = nullptr;
    if (cudaMalloc(&counts, 24) != cudaSuccess || cudaMemset(counts, 0, 24) != cudaSuccess) return 1;
    check<<<148 * 8, 256>>>(counts);
    const cudaError_t e = cudaMemcpy(out, counts, 24, cudaMemcpyDeviceToHost);
    cudaFree(counts);
    return (int)e;
}
"""


def test_every_argument(gpu, tmp_path):
    (tmp_path / "check.cu").write_text(SOURCE)
    flags = [f for f in build.NVCC_FLAGS if f not in ("-Xptxas", "-v", "-lineinfo")]
    subprocess.run([build._nvcc(), *flags, "-shared", f"-I{build.CSRC}", "-o", str(tmp_path / "check.so"), str(tmp_path / "check.cu")], check=True)
    counts = (C.c_ulonglong * 3)()
    assert C.CDLL(str(tmp_path / "check.so")).run(counts) == 0
    wrong, misjudged, plain = counts
    # 2^-40 .. 64 are 46 binades, 64 .. 80 a quarter of one and its end; both signs; and +0
    assert plain == 2 * (46 * 2**23 + 2**21 + 1) + 1
    assert wrong == 0 and misjudged == 0
