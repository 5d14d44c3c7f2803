"""The branch-free FP32 division of the ladder elimination against IEEE
division: the reciprocal for every significand, quotients of random operands
over the range it accepts, subnormal quotients, and every other operand."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "spicier_gb300", "csrc")

SRC = r"""
#include <cstdio>
#include <cstdint>
#include "fpdiv.cuh"
__device__ unsigned long long wrong_rcp, wrong_div, accepted;
__device__ uint32_t mix(uint64_t x) {
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ULL;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebULL;
    return (uint32_t)(x ^ (x >> 31));
}
__global__ void rcp_all() {  // every significand at the ends and the middle of the exponent range, both signs
    const uint32_t m = blockIdx.x * blockDim.x + threadIdx.x;
    const int ex[6] = {127 - 60, 126, 127, 128, 127 + 59, 127 + 33};
    for (int k = 0; k < 6; ++k)
        for (uint32_t s = 0; s < 2; ++s) {
            const float b = __uint_as_float((s << 31) | ((uint32_t)ex[k] << 23) | m);
            if (__float_as_uint(sp::rcp_rn(b)) != __float_as_uint(__fdiv_rn(1.f, b))) atomicAdd(&wrong_rcp, 1ull);
        }
}
__global__ void div_random(int rounds) {
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long bad = 0, took = 0;
    for (int k = 0; k < rounds; ++k) {
        const uint64_t z = (t * rounds + k) * 0x9e3779b97f4a7c15ULL;
        uint32_t ab = mix(z), bb = mix(z + 77);
        if (k % 4 == 1) ab = (ab & 0x807fffffu) | (90u + ab % 57u) << 23, bb = (bb & 0x807fffffu) | (90u + bb % 57u) << 23;  // ordinary size
        if (k % 4 == 2) ab &= 0x81ffffffu, bb = (bb & 0x807fffffu) | (90u + bb % 57u) << 23;  // subnormal quotients
        if (k % 8 == 6) ab &= 0x80000fffu >> (bb % 12u);                         // a few ulps of the smallest number
        if (k % 64 == 3) ab &= 0x80000000u;                                     // zeros
        const float a = __uint_as_float(ab), b = __uint_as_float(bb);
        const uint32_t want = __float_as_uint(__fdiv_rn(a, b));
        const bool nan = (want & 0x7fffffffu) > 0x7f800000u;
        bad += !nan && __float_as_uint(sp::div_careful(a, b)) != want;
        bool mid;
        const float qm = sp::div_mid(a, b, sp::rcp_rn(b), mid);
        bad += mid && __float_as_uint(qm) != want;
        bool ok = true;
        const float q = sp::div_rn(a, b, sp::rcp_rn(b), ok);
        if (!ok) continue;
        ++took;
        bad += __float_as_uint(q) != want;
    }
    atomicAdd(&wrong_div, bad);
    atomicAdd(&accepted, took);
}
int main() {
    rcp_all<<<(1 << 23) / 256, 256>>>();
    div_random<<<4096, 256>>>(1024);
    unsigned long long r = 0, d = 0, n = 0;
    if (cudaDeviceSynchronize() != cudaSuccess) return 2;
    cudaMemcpyFromSymbol(&r, wrong_rcp, 8);
    cudaMemcpyFromSymbol(&d, wrong_div, 8);
    cudaMemcpyFromSymbol(&n, accepted, 8);
    printf("%llu %llu %llu\n", r, d, n);
    return 0;
}
"""


def test_division_matches_ieee(tmp_path):
    src, exe = tmp_path / "div.cu", tmp_path / "div"
    src.write_text(SRC)
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    subprocess.run([nvcc, "-O3", "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", f"-I{CSRC}", str(src),
                    "-o", str(exe)], check=True, capture_output=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=120).stdout.split()
    wrong_rcp, wrong_div, accepted = map(int, out)
    assert wrong_rcp == 0 and wrong_div == 0
    assert accepted > 2 ** 26  # of 2^30 operand pairs, most of them outside the fast range on purpose
