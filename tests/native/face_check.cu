// Checks of the roots and quotients of gsw_face.cuh against the IEEE operators, run by
// tests/test_face_gpu.py; prints the number of differences of each:
//   sqrt_in and rcp_in: every binary32 in [2^-100, 2^100] (rcp_in: both signs);
//   div_in: every pair of significands whose quotient is nearest to a rounding boundary
//   (a 2^s - b M = c with M odd, |c| <= 8), and random pairs with exponents in [-60, 60].
#include <cstdint>
#include <cstdio>
#include "../../geoswe_b200/csrc/gsw_common.cuh"
#include "../../geoswe_b200/csrc/gsw_face.cuh"

using u64 = unsigned long long;
using namespace gsw;

__global__ void check_roots(u64* bad) {
    const u64 lo = (u64)(127 - 100) << 23, hi = ((u64)(127 + 100) << 23) + 1;
    u64 r = 0, y = 0;
    for (u64 i = lo + blockIdx.x * (u64)blockDim.x + threadIdx.x; i < hi; i += (u64)gridDim.x * blockDim.x) {
        const float x = __uint_as_float((uint32_t)i);
        r += sqrt_in(x) != __fsqrt_rn(x);
        y += (rcp_in(x) != __frcp_rn(x)) + (rcp_in(-x) != __frcp_rn(-x));
    }
    if (r) atomicAdd(bad, r);
    if (y) atomicAdd(bad + 1, y);
}

__global__ void check_hard_quotients(u64* bad, u64* tested) {
    u64 n = 0, wrong = 0;
    for (uint32_t b = (1u << 23) + blockIdx.x * blockDim.x + threadIdx.x; b < (1u << 24); b += gridDim.x * blockDim.x) {
        const int t = __ffs(b) - 1;
        if (t > 3) continue;                       // 2^t would have to divide c
        const uint32_t odd = b >> t;
        uint32_t inv = odd;
        for (int k = 0; k < 5; ++k) inv *= 2u - odd * inv;
        for (int s = 24; s <= 25; ++s)
            for (int c = -8; c <= 8; ++c) {
                if (c == 0 || c % (1 << t) != 0) continue;
                const int co = c / (1 << t);
                const uint32_t mod = 1u << (s - t);
                for (u64 M = ((uint32_t)(-co) * inv) & (mod - 1); M < (1ull << 25); M += mod) {
                    if (M < (1u << 24) || !(M & 1)) continue;
                    const long long num = (long long)odd * (long long)M + co;
                    if (num <= 0 || (num & ((1ll << (s - t)) - 1))) continue;
                    const long long a = num >> (s - t);
                    if (a < (1 << 23) || a >= (1 << 24)) continue;
                    ++n;
                    wrong += div_in((float)a, (float)b, rcp_in((float)b)) != __fdiv_rn((float)a, (float)b);
                }
            }
    }
    atomicAdd(tested, n);
    if (wrong) atomicAdd(bad + 2, wrong);
}

__global__ void check_random_quotients(u64* bad, int reps) {
    u64 st = (blockIdx.x * (u64)blockDim.x + threadIdx.x) * 0x9E3779B97F4A7C15ull + 1, wrong = 0;
    for (int i = 0; i < reps; ++i) {
        st ^= st << 13; st ^= st >> 7; st ^= st << 17;
        const uint32_t p = (uint32_t)st, q = (uint32_t)(st >> 32);
        const float a = __uint_as_float((p & 0x7fffffu) | ((127 - 60 + (p >> 23) % 121) << 23));
        const float b = __uint_as_float((q & 0x7fffffu) | ((127 - 60 + (q >> 23) % 121) << 23));
        wrong += (div_in(a, b, rcp_in(b)) != __fdiv_rn(a, b)) + (div_in(-a, b, rcp_in(b)) != __fdiv_rn(-a, b));
    }
    if (wrong) atomicAdd(bad + 3, wrong);
}

int main() {
    u64* d;
    cudaMalloc(&d, 5 * sizeof(u64));
    cudaMemset(d, 0, 5 * sizeof(u64));
    check_roots<<<1184, 256>>>(d);
    check_hard_quotients<<<1184, 256>>>(d, d + 4);
    check_random_quotients<<<1184, 256>>>(d, 4000);
    u64 h[5];
    if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    printf("%llu %llu %llu %llu %llu\n", h[0], h[1], h[2], h[3], h[4]);
    return 0;
}
