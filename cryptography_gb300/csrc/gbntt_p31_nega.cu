// gbntt_p31_nega.cu — the ends of a negacyclic product (gbntt_negacyclic.cu)
// on the 31-bit primes.
//
// A coefficient of 64 bits is f0 + 2^32 f1, so the product modulo X^N + 1 is
// P0 + 2^32 (P1 - P0 - P2) + 2^64 P2 with the three negacyclic products
// P0 = f0 g0, P1 = (f0 + f1)(g0 + g1), P2 = f1 g1, whose coefficients stay
// below 2^(66 + L) in magnitude: one wave of three products of N = 2^L points
// (N <= 2^24: psi has order 2 N) on primes whose residues take a third of the
// 64-bit primes' instructions.
//   twist:  spectra of f0, f0 + f1, f1 times psi^i, where the first pass reads
//           residues;
//   finish: psi^-i, Garner of the three coefficients to signed integers, and
//           their sum as a signed 256-bit integer.
// Both are bound by memory (8 bytes in and 36 out per coefficient, 36 in and
// 32 out) and by the multiply pipe about equally.
#include "gbntt_p31_garner.cuh"

namespace gbntt {

namespace {

typedef unsigned __int128 u128;

// psi^(+-i), Montgomery form, from the two-level tables of w (order 2^25)
__device__ __forceinline__ uint32_t psi_pow(const P31NegaArgs &a, int k, uint32_t i, uint32_t p, uint32_t pinv)
{
    const uint32_t e = i << a.shift;
    return p31_mont(__ldg(a.hi[k] + (e >> 15)), __ldg(a.lo[k] + (e & 32767u)), p, pinv);
}

__global__ void __launch_bounds__(256) p31_nega_twist_kernel(const __grid_constant__ P31NegaArgs a)
{
    const uint32_t n = (uint32_t)a.n, i = blockIdx.x * 256u + threadIdx.x;
    const int op = blockIdx.y;
    chain_wait();
    if (i >= n) return;
    const uint64_t v = __ldg(a.coef[op] + i);
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const uint32_t p = p31_prime(k), pinv = p31_inv(k);
        const uint32_t w = psi_pow(a, k, i, p, pinv);
        const uint32_t lo = p31_mont((uint32_t)v, w, p, pinv), hi = p31_mont((uint32_t)(v >> 32), w, p, pinv);
        uint32_t *o = a.spec[op][k] + i;
        o[0] = lo;
        o[n] = p31_add(lo, hi, p);
        o[2 * (size_t)n] = hi;
    }
}

// the integer in (-M / 2, M / 2) with the given residues, M = p0 p1 p2
__device__ __forceinline__ __int128 signed_coef(uint32_t r0, uint32_t r1, uint32_t r2)
{
    constexpr u128 M = (u128)kP31[0] * kP31[1] * kP31[2];
    uint32_t w0, w1, w2;
    garner31(r0, r1, r2, w0, w1, w2);
    const u128 c = ((u128)w2 << 64) | ((uint64_t)w1 << 32) | w0;
    return (__int128)(c > M / 2 ? c - M : c);
}

__global__ void __launch_bounds__(256) p31_nega_finish_kernel(const __grid_constant__ P31NegaArgs a)
{
    const uint32_t n = (uint32_t)a.n, i = blockIdx.x * 256u + threadIdx.x;
    chain_wait();
    if (i >= n) return;
    uint32_t r[3][3];   // [product][prime]
#pragma unroll
    for (int k = 0; k < 3; k++)
#pragma unroll
        for (int t = 0; t < 3; t++) r[t][k] = a.spec[0][k][t * (size_t)n + i];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const uint32_t p = p31_prime(k), pinv = p31_inv(k), w = psi_pow(a, k, i, p, pinv);
#pragma unroll
        for (int t = 0; t < 3; t++) r[t][k] = p31_mont(r[t][k], w, p, pinv);
    }
    const __int128 p0 = signed_coef(r[0][0], r[0][1], r[0][2]), p2 = signed_coef(r[2][0], r[2][1], r[2][2]);
    const __int128 mid = signed_coef(r[1][0], r[1][1], r[1][2]) - p0 - p2;
    const uint64_t s0 = (uint64_t)(p0 >> 127), sm = (uint64_t)(mid >> 127), s2 = (uint64_t)(p2 >> 127);
    // words of p0, mid 2^32 and p2 2^64, each sign-extended to 256 bits
    u128 c = (u128)(uint64_t)p0 + ((uint64_t)mid << 32);
    const uint64_t o0 = (uint64_t)c;
    c = (c >> 64) + (uint64_t)(p0 >> 64) + (uint64_t)(mid >> 32) + (uint64_t)p2;
    const uint64_t o1 = (uint64_t)c;
    c = (c >> 64) + s0 + (uint64_t)(mid >> 96) + (uint64_t)(p2 >> 64);
    const uint64_t o2 = (uint64_t)c;
    c = (c >> 64) + s0 + sm + s2;
    ulonglong2 *o = reinterpret_cast<ulonglong2 *>(a.out + 4 * (size_t)i);
    if ((reinterpret_cast<uintptr_t>(o) & 15) == 0) {
        o[0] = make_ulonglong2(o0, o1);
        o[1] = make_ulonglong2(o2, (uint64_t)c);
    } else {
        uint64_t *q = a.out + 4 * (size_t)i;
        q[0] = o0;
        q[1] = o1;
        q[2] = o2;
        q[3] = (uint64_t)c;
    }
}

}  // namespace

cudaError_t launch_p31_nega_twist(int nops, const P31NegaArgs &a, cudaStream_t st)
{
    return launch_chained(p31_nega_twist_kernel, dim3((unsigned)((a.n + 255) / 256), (unsigned)nops), 256, 0, st, a);
}

cudaError_t launch_p31_nega_finish(const P31NegaArgs &a, cudaStream_t st)
{
    return launch_chained(p31_nega_finish_kernel, dim3((unsigned)((a.n + 255) / 256)), 256, 0, st, a);
}

}  // namespace gbntt
