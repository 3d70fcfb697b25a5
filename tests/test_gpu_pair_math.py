"""The splat's paired arithmetic rounds as the plain operations do: inverse
square roots for every significand and both parities of the exponent, at
scales over the whole range of binary32 and for zeros, subnormals, infinities
and NaN, the partial of a square root likewise; sums, differences and products
of pairs over random bit patterns, products not contracted into the sums that
take them."""
import subprocess

import pytest

pytestmark = pytest.mark.gpu

SOURCE = r'''
#include <cstdio>
#include "optics.cuh"
using namespace splat;

__device__ unsigned long long bad[4];

__device__ bool same(float a, float b) {
    return __float_as_uint(a) == __float_as_uint(b) || (isnan(a) && isnan(b));
}
__device__ void check(float x, float y) {
    const float2 g = neg_inv_sqrt2(make_float2(x, y));
    if (!same(g.x, -(1.0f / sqrtf(x)))) atomicAdd(&bad[0], 1ull);
    if (!same(g.y, -(1.0f / sqrtf(y)))) atomicAdd(&bad[0], 1ull);
    const float root = sqrtf(x);  // the reference's partial of a square root
    if (!same(dsqrt(D{x, 1.0f}).d, 1.0f / (2.0f * root))) atomicAdd(&bad[0], 1ull);
}
// i: the significand and the exponent's lowest bit; e: the scale
__global__ void inv_sqrt(int e) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;  // < 2^24
    const unsigned j = (i * 2654435761u) & 0xffffffu;          // another one for the other half
    check(__uint_as_float(((unsigned)e << 23) + i), __uint_as_float(((unsigned)e << 23) + j));
}
__global__ void patterns(unsigned n) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint4 u = philox(make_uint4(i, 0u, 0u, 0u), 5u, 9u);
    // any bit pattern, and for odd i numbers near 1, whose sums keep every bit
    const unsigned keep = i & 1 ? 0x807fffffu : 0xffffffffu, put = i & 1 ? 0x3f800000u : 0u;
    const float2 a = make_float2(__uint_as_float((u.x & keep) | put), __uint_as_float((u.y & keep) | put));
    const float2 b = make_float2(__uint_as_float((u.z & keep) | put), __uint_as_float((u.w & keep) | put));
    check(a.x, a.y);
    const float2 s = add2(a, b), d = sub2(a, b), m = mul2(a, b), f = fma2(a, b, s);
    if (!same(s.x, __fadd_rn(a.x, b.x)) || !same(s.y, __fadd_rn(a.y, b.y))) atomicAdd(&bad[1], 1ull);
    if (!same(d.x, __fsub_rn(a.x, b.x)) || !same(d.y, __fsub_rn(a.y, b.y))) atomicAdd(&bad[2], 1ull);
    const float2 t = add2(mul2(a, b), s), v = sub2(s, mul2(a, b)), w = sub2(mul2(a, b), mul2(s, b));
    if (!same(t.x, __fadd_rn(__fmul_rn(a.x, b.x), s.x)) || !same(t.y, __fadd_rn(__fmul_rn(a.y, b.y), s.y)) ||
        !same(v.x, __fsub_rn(s.x, __fmul_rn(a.x, b.x))) || !same(v.y, __fsub_rn(s.y, __fmul_rn(a.y, b.y))) ||
        !same(w.x, __fsub_rn(__fmul_rn(a.x, b.x), __fmul_rn(s.x, b.x)))) atomicAdd(&bad[2], 1ull);
    if (!same(m.x, __fmul_rn(a.x, b.x)) || !same(m.y, __fmul_rn(a.y, b.y)) ||
        !same(f.x, __fmaf_rn(a.x, b.x, s.x)) || !same(f.y, __fmaf_rn(a.y, b.y, s.y))) atomicAdd(&bad[3], 1ull);
}
int main() {
    // exponents 127 and 128 hold every case; the others the range's ends and beyond
    const int es[] = {127, 0, 25, 26, 27, 28, 60, 126, 200, 226, 227, 228, 229, 253};
    for (int e : es) inv_sqrt<<<(1 << 24) / 256, 256>>>(e);
    patterns<<<(1 << 24) / 256, 256>>>(1u << 24);
    unsigned long long h[4];
    if (cudaMemcpyFromSymbol(h, bad, sizeof(h)) != cudaSuccess) { std::printf("%s\n", cudaGetErrorString(cudaGetLastError())); return 2; }
    std::printf("%llu %llu %llu %llu\n", h[0], h[1], h[2], h[3]);
    return 0;
}
'''


def test_pairs_round_like_single_operations(tmp_path):
    from splat_gb300 import build as B

    src, exe = tmp_path / "pairs.cu", tmp_path / "pairs"
    src.write_text(SOURCE)
    r = subprocess.run([B.nvcc(), *B.ARCH, *B.NVCC_FLAGS, "-I", B.CSRC, str(src), "-o", str(exe)], capture_output=True,
                       text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.strip() == "0 0 0 0", out.stdout + out.stderr
