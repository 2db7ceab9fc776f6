// gbntt_p31_radix3.cu — the outer radix-3 stage (gbntt_radix3.cu, where the
// formulas are) for the 31-bit prime set, all three primes in one launch.
#include "gbntt_p31.cuh"

namespace gbntt {

namespace {

constexpr uint32_t kOrder = 3u << kP31MaxLog;   // order of rho

__device__ __forceinline__ uint32_t half(uint32_t x, uint32_t p) { return (x + ((x & 1) ? p : 0u)) >> 1; }

// rho^e, Montgomery form, from rho^(i 2^15) (3 2^10 words) and rho^i (2^15)
__device__ __forceinline__ uint32_t rho_pow(const uint32_t *t, uint32_t e, uint32_t p, uint32_t pinv)
{
    return p31_mont(t[e >> 15], t[(3u << (kP31MaxLog - 15)) + (e & 32767u)], p, pinv);
}

// A thread takes four adjacent j: 16-byte accesses of each sub-array, one
// table look-up for w^j and a Shoup multiply by w from one j to the next. With
// j strided by the grid, 4-byte accesses and one prime per CTA the forward
// stage was bound by latency: 53 us per operand at 3 2^22 points against 37
// now, the inverse 55 against 45 (their traffic takes 27 and 44).
// The forward stage reads a thread's 12 limbs once for all three primes.
__global__ void __launch_bounds__(256) p31_radix3_fwd_kernel(const __grid_constant__ P31R3Args a)
{
    const uint32_t M = (uint32_t)a.M, j = 4u * (blockIdx.x * 256u + threadIdx.x);
    const long long w = blockIdx.y;
    chain_wait();
    const uint32_t *x = a.limb_tab ? a.limb_tab[w] : a.limbs;
    const uint32_t n = (uint32_t)(a.len_tab ? a.len_tab[w] : a.n_limbs);
    if (j >= M) return;
    uint32_t v[3][4];
    const bool aligned = (reinterpret_cast<uintptr_t>(x) & 15) == 0;
#pragma unroll
    for (int r = 0; r < 3; r++) {
        const uint32_t i = j + r * M;
        if (aligned && i + 4 <= n) {
            const uint4 q = __ldg(reinterpret_cast<const uint4 *>(x + i));
            v[r][0] = q.x;
            v[r][1] = q.y;
            v[r][2] = q.z;
            v[r][3] = q.w;
        } else {
#pragma unroll
            for (int u = 0; u < 4; u++) v[r][u] = i + u < n ? __ldg(x + i + u) : 0u;
        }
    }
#pragma unroll 1
    for (int k = 0; k < 3; k++) {
        const uint32_t p = p31_prime(k), pinv = p31_inv(k);
        uint32_t *out = a.spec[k] + w * 3 * a.M + j;
        const ShoupWord c = a.c[k], step = a.step[k];
        uint32_t w1 = rho_pow(a.rho[k], j << a.shift, p, pinv);
        uint32_t y[3][4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const uint32_t x0 = p31_limb(v[0][u], p), x1 = p31_limb(v[1][u], p), x2 = p31_limb(v[2][u], p);
            const uint32_t s = p31_add(x1, x2, p), t = p31_sub(x0, half(s, p), p);
            const uint32_t e = p31_shoup(x1 - x2 + p, c, p), w2 = p31_mont(w1, w1, p, pinv);
            y[0][u] = p31_add(x0, s, p);
            y[1][u] = p31_mont(p31_add(t, e, p), w1, p, pinv);
            y[2][u] = p31_mont(p31_sub(t, e, p), w2, p, pinv);
            if (u < 3) w1 = p31_shoup(w1, step, p);
        }
#pragma unroll
        for (int m = 0; m < 3; m++)
            *reinterpret_cast<uint4 *>(out + m * a.M) = make_uint4(y[m][0], y[m][1], y[m][2], y[m][3]);
    }
}

__global__ void __launch_bounds__(256) p31_radix3_inv_kernel(const __grid_constant__ P31R3Args a)
{
    const int k = blockIdx.x % 3;
    const uint32_t p = p31_prime(k), pinv = p31_inv(k);
    const uint32_t M = (uint32_t)a.M, j = 4u * ((blockIdx.x / 3) * 256u + threadIdx.x);
    uint32_t *z = a.spec[k] + (long long)blockIdx.y * 3 * a.M + j;
    const ShoupWord c = a.c[k], step = a.step[k];
    chain_wait();
    if (j >= M) return;
    uint32_t v[3][4];
#pragma unroll
    for (int m = 0; m < 3; m++) {
        const uint4 q = *reinterpret_cast<const uint4 *>(z + m * a.M);
        v[m][0] = q.x;
        v[m][1] = q.y;
        v[m][2] = q.z;
        v[m][3] = q.w;
    }
    const uint32_t ex = j << a.shift;
    uint32_t w1 = rho_pow(a.rho[k], ex ? kOrder - ex : 0u, p, pinv);   // w^(-j)
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const uint32_t w2 = p31_mont(w1, w1, p, pinv);
        const uint32_t t1 = p31_mont(v[1][u], w1, p, pinv), t2 = p31_mont(v[2][u], w2, p, pinv);
        const uint32_t s = p31_add(t1, t2, p), e = p31_shoup(t1 - t2 + p, c, p);
        const uint32_t t0 = v[0][u], h = p31_sub(t0, half(s, p), p);
        v[0][u] = p31_add(t0, s, p);
        v[1][u] = p31_sub(h, e, p);
        v[2][u] = p31_add(h, e, p);
        if (u < 3) w1 = p31_shoup(w1, step, p);
    }
#pragma unroll
    for (int m = 0; m < 3; m++) *reinterpret_cast<uint4 *>(z + m * a.M) = make_uint4(v[m][0], v[m][1], v[m][2], v[m][3]);
}

}  // namespace

cudaError_t launch_p31_radix3(bool inverse, const P31R3Args &a, cudaStream_t st)
{
    if (a.W < 1 || a.W > 65535 || a.M % 4) return cudaErrorInvalidValue;
    const dim3 grid((unsigned)((inverse ? 3 : 1) * ((a.M / 4 + 255) / 256)), (unsigned)a.W);
    return launch_chained(inverse ? p31_radix3_inv_kernel : p31_radix3_fwd_kernel, grid, 256, 0, st, a);
}

}  // namespace gbntt
