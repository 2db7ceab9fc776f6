// gbntt_p31_radix3.cu — the outer radix-3 stage (gbntt_radix3.cu, where the
// formulas are) for the 31-bit prime set: all three primes in one launch,
// the prime being the fastest block index so that the three CTAs reading the
// same limbs run side by side.
#include "gbntt_p31.cuh"

namespace gbntt {

namespace {

constexpr uint32_t kOrder = 3u << kP31MaxLog;   // order of rho
constexpr int U = kR3Unroll;

__device__ __forceinline__ uint32_t half(uint32_t x, uint32_t p) { return (x + ((x & 1) ? p : 0u)) >> 1; }

// rho^e, Montgomery form, from rho^(i 2^15) (3 2^10 words) and rho^i (2^15)
__device__ __forceinline__ uint32_t rho_pow(const uint32_t *t, uint32_t e, uint32_t p, uint32_t pinv)
{
    return p31_mont(t[e >> 15], t[(3u << (kP31MaxLog - 15)) + (e & 32767u)], p, pinv);
}

// Thread i of a prime's blocks takes j = i, i + G, ... (G = blocks x 256),
// U of them per step with all their loads first; its twiddle w^j comes from
// the tables once and then from one multiply by w^(+-G) per j.
__global__ void __launch_bounds__(256, 4) p31_radix3_fwd_kernel(const __grid_constant__ P31R3Args a)
{
    const int k = blockIdx.x % 3;
    const uint32_t p = p31_prime(k), pinv = p31_inv(k);
    const uint32_t M = (uint32_t)a.M, G = (gridDim.x / 3) * 256u;
    const long long w = blockIdx.y;
    chain_wait();
    const uint32_t *x = a.limb_tab ? a.limb_tab[w] : a.limbs;
    const uint32_t n = (uint32_t)(a.len_tab ? a.len_tab[w] : a.n_limbs);
    uint32_t *out = a.spec[k] + w * 3 * a.M;
    const ShoupWord c = a.c[k], step = a.step[k];
    uint32_t j = (blockIdx.x / 3) * 256u + threadIdx.x;
    if (j >= M) return;
    uint32_t w1 = rho_pow(a.rho[k], j << a.shift, p, pinv);
    for (; j < M; j += U * G) {
        uint32_t v[U][3];
#pragma unroll
        for (int u = 0; u < U; u++)
#pragma unroll
            for (int r = 0; r < 3; r++) {
                const uint32_t jj = j + u * G, i = jj + r * M;
                v[u][r] = (jj < M && i < n) ? __ldg(x + i) : 0u;
            }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const uint32_t jj = j + u * G;
            if (jj < M) {
                const uint32_t x0 = p31_limb(v[u][0], p), x1 = p31_limb(v[u][1], p), x2 = p31_limb(v[u][2], p);
                const uint32_t s = p31_add(x1, x2, p), t = p31_sub(x0, half(s, p), p);
                const uint32_t e = p31_shoup(x1 - x2 + p, c, p), w2 = p31_mont(w1, w1, p, pinv);
                out[jj] = p31_add(x0, s, p);
                out[M + jj] = p31_mont(p31_add(t, e, p), w1, p, pinv);
                out[2 * M + jj] = p31_mont(p31_sub(t, e, p), w2, p, pinv);
            }
            w1 = p31_shoup(w1, step, p);
        }
    }
}

__global__ void __launch_bounds__(256, 4) p31_radix3_inv_kernel(const __grid_constant__ P31R3Args a)
{
    const int k = blockIdx.x % 3;
    const uint32_t p = p31_prime(k), pinv = p31_inv(k);
    const uint32_t M = (uint32_t)a.M, G = (gridDim.x / 3) * 256u;
    uint32_t *z = a.spec[k] + (long long)blockIdx.y * 3 * a.M;
    const ShoupWord c = a.c[k], step = a.step[k];
    uint32_t j = (blockIdx.x / 3) * 256u + threadIdx.x;
    if (j >= M) return;
    const uint32_t ex = j << a.shift;
    uint32_t w1 = rho_pow(a.rho[k], ex ? kOrder - ex : 0u, p, pinv);   // w^(-j)
    chain_wait();
    for (; j < M; j += U * G) {
        uint32_t v[U][3];
#pragma unroll
        for (int u = 0; u < U; u++)
#pragma unroll
            for (int r = 0; r < 3; r++) v[u][r] = j + u * G < M ? z[j + u * G + r * M] : 0u;
#pragma unroll
        for (int u = 0; u < U; u++) {
            const uint32_t jj = j + u * G;
            if (jj < M) {
                const uint32_t w2 = p31_mont(w1, w1, p, pinv);
                const uint32_t t1 = p31_mont(v[u][1], w1, p, pinv), t2 = p31_mont(v[u][2], w2, p, pinv);
                const uint32_t s = p31_add(t1, t2, p), e = p31_shoup(t1 - t2 + p, c, p);
                const uint32_t t0 = v[u][0], h = p31_sub(t0, half(s, p), p);
                z[jj] = p31_add(t0, s, p);
                z[M + jj] = p31_sub(h, e, p);
                z[2 * M + jj] = p31_add(h, e, p);
            }
            w1 = p31_shoup(w1, step, p);
        }
    }
}

}  // namespace

cudaError_t launch_p31_radix3(bool inverse, const P31R3Args &a, cudaStream_t st)
{
    if (a.W < 1 || a.W > 65535 || a.blocks < 1) return cudaErrorInvalidValue;
    const dim3 grid((unsigned)(3 * a.blocks), (unsigned)a.W);
    return launch_chained(inverse ? p31_radix3_inv_kernel : p31_radix3_fwd_kernel, grid, 256, 0, st, a);
}

}  // namespace gbntt
