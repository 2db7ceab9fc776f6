// gbntt_p31_pass.cu — strided NTT passes of the 31-bit prime set (the pass
// structure of gbntt_pass.cuh: DIF forward, transposed inverse, in place).
//
// A thread loads its 2^ceil(l/2) rows straight into registers (4 G bytes
// contiguous per row over a warp), exchanges once through shared memory and
// stores from registers: two shared-memory accesses per residue instead of
// the six of a staged tile, which together with the arithmetic (see
// gbntt_p31.cuh) is what the pass spends its time on. The pass is bound by
// the multiply pipe; pass twiddles are Montgomery words (4 bytes) because
// the outermost table comes from HBM once per residue.
#include "gbntt_p31.cuh"

namespace gbntt {

namespace {

// w^e (Montgomery form), e < 2^25, from the two-level tables
__device__ __forceinline__ uint32_t p31_tw(const P31PassArgs &a, int k, uint32_t e, uint32_t p, uint32_t pinv)
{
    return p31_mont(__ldg(a.hi[k] + (e >> 15)), __ldg(a.lo[k] + (e & 32767u)), p, pinv);
}

template <int LOG_L, int DIR, bool LIMBS>
__global__ void __launch_bounds__(P31Shape<LOG_L>::T, LOG_L >= 9 ? 3 : LOG_L == 5 ? 10 : 5)
p31_pass_kernel(const __grid_constant__ P31PassArgs a)
{
    using S = P31Shape<LOG_L>;
    constexpr int A = S::A, B = S::B, G = S::G;
    __shared__ uint32_t sm[S::WORDS_S];
    const int k = blockIdx.x % 3, op = blockIdx.y;
    const long long col0 = (long long)(blockIdx.x / 3) * G;
    const uint32_t p = p31_prime(k), pinv = p31_inv(k);
    const int t = threadIdx.x, g = t & (G - 1), q = t >> S::LOG_G;
    const int log_s = a.log_s;
    const uint32_t sub0 = (uint32_t)((col0 >> log_s) << a.log_m);            // first element of the sub-problem
    const uint32_t j = (uint32_t)(col0 & ((1LL << log_s) - 1)) + g;           // this thread's column
    uint32_t *data = a.data[op][k];
    // byte offsets: elements stay below 2^30 per prime
    const uint32_t step = (uint32_t)B << (log_s + 2);
    const uint32_t off0 = (sub0 + j + ((uint32_t)q << log_s)) << 2;
    uint32_t x[A];
    if (LIMBS) {
        // the sub-problem is one product: its operand starts at sub0
        const uint32_t *limbs;
        long long n;
        if (a.limb_tab[op]) {
            const long long b = (long long)(sub0 >> a.log_prod);
            limbs = a.limb_tab[op][b];
            n = a.len_tab[op][b];
        } else {
            limbs = a.limbs[op];
            n = a.n_limbs[op];
        }
        const uint32_t nn = (uint32_t)n, r0 = j + ((uint32_t)q << log_s), rs = (uint32_t)B << log_s;
#pragma unroll
        for (int i = 0; i < A; i++) {
            const uint32_t r = r0 + i * rs;
            x[i] = r < nn ? __ldg(limbs + r) : 0u;
        }
#pragma unroll
        for (int i = 0; i < A; i++) x[i] = p31_limb(x[i], p);
    } else {
#pragma unroll
        for (int i = 0; i < A; i++) x[i] = ld_off(data, off0 + i * step);
    }
    const uint32_t *ptw = a.ptw[k];
    // table address such that an element's own offset indexes it
    const char *tb = reinterpret_cast<const char *>(reinterpret_cast<uintptr_t>(ptw) - ((uintptr_t)sub0 << 2));
    if (DIR == 1) {
        if (ptw) {
            uint32_t tw[A];
#pragma unroll
            for (int i = 0; i < A; i++) tw[i] = __ldg(reinterpret_cast<const uint32_t *>(tb + (off0 + i * step)));
#pragma unroll
            for (int i = 0; i < A; i++) x[i] = p31_mont(x[i], tw[i], p, pinv);
        } else {
            const int sh = kP31MaxLog - a.log_m;
            const uint32_t sc = a.scale[k];
#pragma unroll
            for (int i = 0; i < A; i++) {
                uint32_t w = p31_tw(a, k, (uint32_t)(((uint64_t)(i * B + q) * j) << sh), p, pinv);
                if (a.use_scale) w = p31_mont(w, sc, p, pinv);
                x[i] = p31_mont(x[i], w, p, pinv);
            }
        }
    }
    p31_tile_fwd<LOG_L, true>(x, sm, g, q, c_p31_roots.v[k][DIR], a.st[k] + (S::L - 32), p);
    const uint32_t row = 4u << log_s;
    if (DIR == 0) {
        if (ptw) {
#pragma unroll
            for (int r = 0; r < S::R; r++) {
#pragma unroll
                for (int kb = 0; kb < B; kb++) {
                    const uint32_t off = off0 + (r * B + A * kb) * row;
                    const uint32_t tw = __ldg(reinterpret_cast<const uint32_t *>(tb + off));
                    st_off(data, off, p31_mont(x[r * B + kb], tw, p, pinv));
                }
            }
        } else {
            const int sh = kP31MaxLog - a.log_m;
#pragma unroll
            for (int r = 0; r < S::R; r++) {
#pragma unroll
                for (int kb = 0; kb < B; kb++) {
                    const int m = q + r * B + A * kb;
                    const uint32_t w = p31_tw(a, k, (uint32_t)(((uint64_t)m * j) << sh), p, pinv);
                    st_off(data, off0 + (r * B + A * kb) * row, p31_mont(x[r * B + kb], w, p, pinv));
                }
            }
        }
    } else {
#pragma unroll
        for (int r = 0; r < S::R; r++) {
#pragma unroll
            for (int kb = 0; kb < B; kb++) st_off(data, off0 + (r * B + A * kb) * row, x[r * B + kb]);
        }
    }
}

template <int LOG_L>
cudaError_t launch_l(int dir, bool limbs, int nops, const P31PassArgs &a, cudaStream_t st)
{
    using S = P31Shape<LOG_L>;
    const dim3 grid((unsigned)(3 * (a.ncols / S::G)), (unsigned)nops);
    if (dir == 1) p31_pass_kernel<LOG_L, 1, false><<<grid, S::T, 0, st>>>(a);
    else if (limbs) p31_pass_kernel<LOG_L, 0, true><<<grid, S::T, 0, st>>>(a);
    else p31_pass_kernel<LOG_L, 0, false><<<grid, S::T, 0, st>>>(a);
    return cudaGetLastError();
}

__global__ void p31_table_kernel(int k, uint32_t *table, const uint32_t *hi, const uint32_t *lo, int log_m, int log_s,
                                 int use_scale, uint32_t scale)
{
    const uint32_t p = p31_prime(k), pinv = p31_inv(k);
    const long long M = 1LL << log_m;
    const int sh = kP31MaxLog - log_m;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < M; e += (long long)gridDim.x * blockDim.x) {
        const uint64_t m = (uint64_t)e >> log_s, j = (uint64_t)e & ((1ull << log_s) - 1);
        const uint32_t x = (uint32_t)((m * j) << sh);
        uint32_t w = p31_mont(hi[x >> 15], lo[x & 32767u], p, pinv);
        if (use_scale) w = p31_mont(w, scale, p, pinv);
        table[e] = w;
    }
}

}  // namespace

cudaError_t launch_p31_pass(int log_l, int dir, bool limbs, int nops, const P31PassArgs &a, cudaStream_t st)
{
    switch (log_l) {
    case 5: return launch_l<5>(dir, limbs, nops, a, st);
    case 6: return launch_l<6>(dir, limbs, nops, a, st);
    case 7: return launch_l<7>(dir, limbs, nops, a, st);
    case 8: return launch_l<8>(dir, limbs, nops, a, st);
    case 9: return launch_l<9>(dir, limbs, nops, a, st);
    case 10: return launch_l<10>(dir, limbs, nops, a, st);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_p31_build_table(int prime, uint32_t *table, const uint32_t *hi, const uint32_t *lo, int log_m,
                                   int log_s, int use_scale, uint32_t scale, cudaStream_t st)
{
    const long long M = 1LL << log_m;
    const long long grid = (M + 255) / 256;
    p31_table_kernel<<<(unsigned)(grid > 152 * 16 ? 152 * 16 : grid), 256, 0, st>>>(prime, table, hi, lo, log_m, log_s,
                                                                                     use_scale, scale);
    return cudaGetLastError();
}

}  // namespace gbntt
