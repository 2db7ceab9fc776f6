// gbntt_p31.cuh — arithmetic, register DFTs and tile transforms of the
// 31-bit prime set.
//
// A product coefficient of 32-bit limbs is below min(n_a, n_b) 2^64, so three
// primes just below 2^31 (product 2^92.64) carry every product whose shorter
// operand has at most 2^28 limbs. Against q0 (64 bits) with p3 (32 bits) the
// modulus per residue word is the same, but a residue below 2^31 leaves the
// 32-bit word a spare bit: a modular addition is an add and a minimum (two
// instructions, VIADDMNMX on the ALU pipe), and a product by a known factor
// is one high and two low multiplies (Shoup) with no carries. Measured on
// GB300 (cycles per warp instruction and SM sub-partition): add or minimum 2,
// 32-bit multiply-add 2, high or wide multiply 4; a butterfly with a twiddle
// takes 10.1, without one 4.6. q0 and p3 together execute about 33
// instructions per coefficient and radix-2 level, this set about 20.
//
// All three primes have 2-adicity of at least 25 and p - 1 divisible by 3:
//   15 2^27 + 1, 27 2^26 + 1, 63 2^25 + 1,
// so transforms have up to 2^25 points, or 3 2^k with k <= 25. Longer
// products (up to 2^29 coefficients) are put together from up to 16
// transforms of 2^25 points (gbntt_p31_outer.cu); beyond that the modulus is
// too small and the 64-bit prime sets take over.
//
// One launch covers all three primes (the prime is the fastest block index,
// so the CTAs that read the same limbs or tile run side by side), and both
// operands where they have the same shape (blockIdx.y).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "gbntt_internal.h"

namespace gbntt {

constexpr uint32_t kP31[3] = {2013265921u, 1811939329u, 2113929217u};
constexpr uint32_t kP31Inv[3] = {2281701377u, 2483027969u, 2181038081u};   // p^-1 mod 2^32
constexpr uint32_t kP31Gen[3] = {31u, 13u, 5u};                            // primitive roots
constexpr int kP31MaxLog = 25;

constexpr uint64_t p31_pow(uint64_t b, uint64_t e, uint64_t p)
{
    uint64_t r = 1;
    b %= p;
    while (e) {
        if (e & 1) r = r * b % p;
        b = b * b % p;
        e >>= 1;
    }
    return r;
}

// A factor w with floor(w 2^32 / p) beside it.
struct ShoupWord {
    uint32_t w, q;
};
constexpr ShoupWord shoup_word(uint64_t w, uint64_t p) { return {(uint32_t)w, (uint32_t)((w << 32) / p)}; }

// t[i] = w^i in Montgomery form, i < n: each length's powers from the first
// half's times one factor (Shoup).
static inline void p31_powers(uint32_t *t, size_t n, uint64_t w, uint64_t p)
{
    const uint32_t q = (uint32_t)p;
    t[0] = (uint32_t)(((uint64_t)1 << 32) % p);
    for (size_t m = 1; m < n; m *= 2, w = w * w % p) {
        const ShoupWord f = shoup_word(w, p);   // w^m
        const uint32_t *__restrict__ a = t;
        uint32_t *__restrict__ b = t + m;
        const size_t end = n - m < m ? n - m : m;
        for (size_t i = 0; i < end; i++) {
            const uint32_t r = a[i] * f.w - (uint32_t)(((uint64_t)a[i] * f.q) >> 32) * q, s = r - q;
            b[i] = s < r ? s : r;   // (r < 2 p)
        }
    }
}

// w_32^i per prime and direction: the constants of the register DFTs.
struct P31Roots {
    ShoupWord v[3][2][16];
};
constexpr P31Roots p31_roots()
{
    P31Roots t{};
    for (int k = 0; k < 3; k++) {
        const uint64_t p = kP31[k];
        const uint64_t w = p31_pow(kP31Gen[k], (p - 1) / 32, p);
        for (int d = 0; d < 2; d++) {
            const uint64_t wd = d ? p31_pow(w, p - 2, p) : w;
            uint64_t x = 1;
            for (int i = 0; i < 16; i++) {
                t.v[k][d][i] = shoup_word(x, p);
                x = x * wd % p;
            }
        }
    }
    return t;
}

#ifdef __CUDACC__
// Launches of a product follow each other with nothing to do on the host
// between them, so the next one is set up while the one before it runs
// (programmatic dependent launch) and waits in chain_wait until the memory
// of every earlier launch is complete. Every kernel that launch_chained
// starts calls chain_wait before it touches memory that an earlier launch
// writes or reads. No kernel lets its successor start early: CTAs of the
// next launch that come up during the last wave of this one take places
// unevenly (2^24 points 770 us so, 788 us with plain launches and 858 us with
// an early start; 2^17 points 19.5, 26.9 and 27.1 us; 2^13 12.4, 20.7 and
// 13.4 us).
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
template <class Args>
static inline cudaError_t launch_chained(void (*fn)(Args), dim3 grid, int threads, size_t smem, cudaStream_t st,
                                         const Args &args, int cluster = 1)
{
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = grid;
    c.blockDim = dim3((unsigned)threads);
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = at;
    c.numAttrs = 1;
    if (cluster > 1) {
        at[1].id = cudaLaunchAttributeClusterDimension;
        at[1].val.clusterDim.x = (unsigned)cluster;
        at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
        c.numAttrs = 2;
    }
    return cudaLaunchKernelEx(&c, fn, args);
}

static __constant__ const P31Roots c_p31_roots = p31_roots();

__device__ __forceinline__ uint32_t p31_prime(int k)
{
    constexpr uint32_t p0 = kP31[0], p1 = kP31[1], p2 = kP31[2];
    return k == 0 ? p0 : k == 1 ? p1 : p2;
}
__device__ __forceinline__ uint32_t p31_inv(int k)
{
    constexpr uint32_t i0 = kP31Inv[0], i1 = kP31Inv[1], i2 = kP31Inv[2];
    return k == 0 ? i0 : k == 1 ? i1 : i2;
}

// Canonical operands and results in [0, p), p < 2^31.
__device__ __forceinline__ uint32_t p31_add(uint32_t a, uint32_t b, uint32_t p)
{
    const uint32_t s = a + b;
    return __viaddmin_u32(s, 0u - p, s);
}
__device__ __forceinline__ uint32_t p31_sub(uint32_t a, uint32_t b, uint32_t p)
{
    const uint32_t d = a - b;
    return __viaddmin_u32(d, p, d);
}
// x w mod p in [0, 2 p) for any x (Shoup; the quotient is at most one short)
__device__ __forceinline__ uint32_t p31_shoup_lazy(uint32_t x, ShoupWord w, uint32_t p)
{
    return x * w.w - __umulhi(x, w.q) * p;
}
__device__ __forceinline__ uint32_t p31_shoup(uint32_t x, ShoupWord w, uint32_t p)
{
    const uint32_t r = p31_shoup_lazy(x, w, p);
    return __viaddmin_u32(r, 0u - p, r);
}
// x t 2^-32 mod p for any x and t < p (Montgomery)
__device__ __forceinline__ uint32_t p31_mont(uint32_t x, uint32_t t, uint32_t p, uint32_t pinv)
{
    const uint64_t z = (uint64_t)x * t;
    const uint32_t m = (uint32_t)z * pinv;
    const uint32_t d = (uint32_t)(z >> 32) - __umulhi(m, p);
    return __viaddmin_u32(d, p, d);
}
// a 32-bit limb (< 2^32 < 3 p)
__device__ __forceinline__ uint32_t p31_limb(uint32_t v, uint32_t p)
{
    v = __viaddmin_u32(v, 0u - 2u * p, v);
    return __viaddmin_u32(v, 0u - p, v);
}

constexpr int p31_bitrev(int x, int bits)
{
    int r = 0;
    for (int i = 0; i < bits; i++) r = (r << 1) | ((x >> i) & 1);
    return r;
}

// Radix-2 DIF DFT of 2^LOG_R points in registers: X[k] ends in
// x[bitrev(k)]. roots: w_32^i of the prime and direction. upper_zero: the
// upper half of x is zero and not read (a first pass over an operand of at
// most half the transform's length).
template <int LOG_R>
__device__ __forceinline__ void p31_dft(uint32_t *x, const ShoupWord *roots, uint32_t p, bool upper_zero = false)
{
    constexpr int R = 1 << LOG_R;
    if (upper_zero) {
        x[R / 2] = x[0];
#pragma unroll
        for (int i = 1; i < R / 2; i++) x[R / 2 + i] = p31_shoup(x[i], roots[i * (32 / R)], p);
    }
#pragma unroll
    for (int s = R / 2; s >= 1; s >>= 1) {
        if (s == R / 2 && upper_zero) continue;
#pragma unroll
        for (int blk = 0; blk < R; blk += 2 * s) {
#pragma unroll
            for (int i = 0; i < s; i++) {
                const uint32_t u = x[blk + i], v = x[blk + i + s];
                x[blk + i] = p31_add(u, v, p);
                if (i == 0) x[blk + i + s] = p31_sub(u, v, p);
                else x[blk + i + s] = p31_shoup(u - v + p, roots[i * (16 / s)], p);
            }
        }
    }
}

// Shape of a tile: G columns of 2^l points, A x B with A = 2^ceil(l/2)
// points per thread and B threads per column. Threads whose column index is
// the fast one (strided tiles) read and write 4 G contiguous bytes per row;
// in contiguous tiles the B threads of a column are adjacent. Row and column
// strides of the exchange buffer keep both its accesses free of bank
// conflicts for every l.
template <int LOG_L>
struct P31Shape {
    static constexpr int L = 1 << LOG_L;
    static constexpr int LOG_A = (LOG_L + 1) / 2, LOG_B = LOG_L / 2;
    static constexpr int A = 1 << LOG_A, B = 1 << LOG_B, R = A / B;
    static constexpr int T = LOG_L == 5 ? 128 : 256;
    static constexpr int G = T / B;
    static constexpr int LOG_G = LOG_L == 5 ? 5 : 8 - LOG_B;
    static constexpr int RS_C = B + 1;                                         // contiguous: g GS_C + ka RS_C + b
    static constexpr int GS_C = A * RS_C + (LOG_L == 5 ? 4 : LOG_L == 7 ? 8 : LOG_L == 9 ? 16 : 0);
    static constexpr int WORDS_C = G * GS_C;
};

// The forward DFT of one column, spread over B threads. In: thread (g, b)
// holds x[i] = element i B + b. Out: thread (g, q) holds element (q + r B) +
// A kb in x[r B + kb]. st: step table w_L^(ka b) at [ka B + b]. Starts and
// ends without a barrier; the buffer may be reused after one.
template <int LOG_L>
__device__ __forceinline__ void p31_tile_fwd(uint32_t *x, uint32_t *sm, int g, int q, const ShoupWord *roots,
                                             const ShoupWord *__restrict__ st, uint32_t p)
{
    using S = P31Shape<LOG_L>;
    constexpr int A = S::A, B = S::B;
    p31_dft<S::LOG_A>(x, roots, p);
    constexpr int RS = S::RS_C;
    uint32_t *w = sm + g * S::GS_C + q;
#pragma unroll
    for (int ka = 0; ka < A; ka++) {
        const uint32_t v = x[p31_bitrev(ka, S::LOG_A)];
        w[ka * RS] = ka == 0 ? v : p31_shoup(v, st[ka * B + q], p);
    }
    __syncthreads();
    const uint32_t *r0 = sm + g * S::GS_C + q * RS;
#pragma unroll
    for (int r = 0; r < S::R; r++) {
        uint32_t y[B];
#pragma unroll
        for (int b = 0; b < B; b++) y[b] = r0[r * B * RS + b];
        p31_dft<S::LOG_B>(y, roots, p);
#pragma unroll
        for (int kb = 0; kb < B; kb++) x[r * B + kb] = y[p31_bitrev(kb, S::LOG_B)];
    }
}

// The inverse DFT (unscaled) from the layout p31_tile_fwd leaves back to the
// one it takes (contiguous tiles). st: w_L^(-ka b) at [b A + ka].
template <int LOG_L>
__device__ __forceinline__ void p31_tile_inv(uint32_t *x, uint32_t *sm, int g, int q, const ShoupWord *roots,
                                             const ShoupWord *__restrict__ st, uint32_t p)
{
    using S = P31Shape<LOG_L>;
    constexpr int A = S::A, B = S::B, RS = S::RS_C;
    uint32_t *w = sm + g * S::GS_C + q * RS;
#pragma unroll
    for (int r = 0; r < S::R; r++) {
        uint32_t y[B];
#pragma unroll
        for (int kb = 0; kb < B; kb++) y[kb] = x[r * B + kb];
        p31_dft<S::LOG_B>(y, roots, p);
#pragma unroll
        for (int b = 0; b < B; b++) {
            const uint32_t v = y[p31_bitrev(b, S::LOG_B)];
            w[r * B * RS + b] = b == 0 ? v : p31_shoup(v, st[b * A + q + r * B], p);
        }
    }
    __syncthreads();
    const uint32_t *r0 = sm + g * S::GS_C + q;
#pragma unroll
    for (int ka = 0; ka < A; ka++) x[ka] = r0[ka * RS];
    p31_dft<S::LOG_A>(x, roots, p);
    uint32_t y[A];
#pragma unroll
    for (int i = 0; i < A; i++) y[i] = x[p31_bitrev(i, S::LOG_A)];
#pragma unroll
    for (int i = 0; i < A; i++) x[i] = y[i];
}

#endif  // __CUDACC__

// Step tables of one prime and direction: for pass size 2^l the A x B block
// at 2^l - 32 holds w_L^(ka b) at [ka B + b]; the second half (at
// kStep1Words) the same at [b A + ka]. After them the tables of the strided
// 2^9-point passes' three steps: w_512^(k0 c) at [64 k0 + c], then
// w_64^(k1 m0) at [8 k1 + m0].
constexpr int kP31Step9 = 2 * kStep1Words;
constexpr int kP31StepWords = kP31Step9 + 512 + 64;

struct P31PassArgs {
    uint32_t *data[2][3];               // per operand (blockIdx.y) and prime
    const uint32_t *limbs[2];           // first pass of one product
    long long n_limbs[2];
    const uint32_t *const *limb_tab[2]; // first pass of a wave: product b's limbs
    const long long *len_tab[2];
    const uint32_t *ptw[3];             // pass twiddles w_M^(+-j m) at j + m S, Montgomery form, or null
    const ShoupWord *st[3];             // step tables (this direction)
    const uint32_t *hi[3], *lo[3];      // two-level tables: w^(i 2^15), w^i, Montgomery form, w of order 2^25
    uint32_t scale[3];                  // inverse, no table: factor of the outermost pass (Montgomery form of it)
    int use_scale;
    int log_m, log_s;                   // sub-problem and column-stride logs
    int log_prod;                       // log2 of a product's coefficients (first pass)
    long long ncols;                    // columns per operand
    int by_table;                       // the outermost pass: order the CTAs by their part of the table
};

struct P31InnerArgs {
    uint32_t *data[3];                  // first spectra, product in place
    const uint32_t *other[3];           // second spectra (null: a square)
    const ShoupWord *st[3], *sti[3];    // step tables, forward and inverse
    uint32_t scale[3];                  // single-pass transforms: factor (Montgomery form)
    int use_scale;
    int other_done;                     // the second spectra have had their innermost pass
    int log_prod;                       // log2 of a (sub-)transform's points
    int shared, paired, r3;             // second spectra shared by all products / by pairs; sub-transforms of 3 2^k
    long long ncols;
    unsigned *zero;                     // carry control words to clear: zero[0], zero[2 .. 2 + nzero)
    long long nzero;
};

// Outer radix-3 stage of W products: product w's three 2^k-point spectra at
// spec[prime] + w 3 M + m M.
struct P31R3Args {
    uint32_t *spec[3];
    long long M, W;                     // 2^k, products (<= 65535)
    int shift;                          // 25 - k: w_N^j = rho^(j << shift)
    const uint32_t *limbs;              // forward input of a single product, or of W products
    long long n_limbs;
    const uint32_t *const *limb_tab;
    const long long *len_tab;
    const uint32_t *rho[3];             // two-level tables of rho (order 3 2^25)
    ShoupWord c[3], step[3];            // (om - om^2) / 2; w (forward) or w^-1 (inverse)
};
cudaError_t launch_p31_radix3(bool inverse, const P31R3Args &a, cudaStream_t st);

// Outer stage of a product of up to R 2^25 coefficients (R = 2, 4 .. 16):
// spectrum m at spec[prime] + m 2^25.
constexpr int kP31MaxOuter = 16;
struct P31OuterArgs {
    uint32_t *spec[3];
    const uint32_t *limbs;              // forward input
    long long n_limbs;
    int blocks;                         // ceil(n_limbs / 2^25), at most R
    const uint32_t *g[3];               // two-level tables of g (forward) or g^-1: 2^10 words g^(i 2^15), 2^15 words g^i
    const uint32_t *gh[3];              // the same of g^(d / 2) (primes whose d is even)
};
cudaError_t launch_p31_outer(int R, bool inverse, const P31OuterArgs &a, cudaStream_t st);
uint64_t p31_outer_root(int k);         // g of prime k
uint64_t p31_outer_half(int k);         // g^(d / 2)
cudaError_t p31_outer_init();

// A whole product of up to 2^kP31BlockLog coefficients in one CTA or a cluster
// of three (W of them: the tables).
constexpr int kP31BlockLog = 12;
struct P31BlockArgs {
    const uint32_t *limbs[2];
    long long n_limbs[2];
    uint32_t *out;
    long long n_out;
    const uint32_t *const *limb_tab[2];
    const long long *len_tab[2];
    uint32_t *const *out_tab;
    const long long *nout_tab;
    int shared, paired;                 // second operands: entry 0 for all, entry b / 2
    const uint32_t *tw[3][2];           // step tables per prime and direction (p31_block_tables)
    ShoupWord scale[3];                 // 2^32 / N
    unsigned *error;
    unsigned *sticky;                   // or null: error bits moved from here to *error (one product)
};
cudaError_t launch_p31_block(int log_n, const P31BlockArgs &a, long long W, cudaStream_t st);
// Fills the step tables of 2^log_n points for a root w of that order (at
// most 2^(log_n + 1) words) and returns their size.
int p31_block_tables(int log_n, uint32_t *dst, uint64_t w, uint64_t p);

// Negacyclic products of N = 2^L 64-bit coefficients, L < kP31MaxLog: three
// products' spectra of N words, one after the other, per prime and operand.
struct P31NegaArgs {
    uint32_t *spec[2][3];
    const uint64_t *coef[2];            // twist
    const uint32_t *hi[3], *lo[3];      // two-level tables of w (order 2^25) or w^-1
    int shift;                          // psi^i = w^(i << shift)
    long long n;                        // N
    uint64_t *out;                      // finish: 4 N words
};
cudaError_t launch_p31_nega_twist(int nops, const P31NegaArgs &a, cudaStream_t st);
cudaError_t launch_p31_nega_finish(const P31NegaArgs &a, cudaStream_t st);

cudaError_t launch_p31_pass(int log_l, int dir, bool limbs, int nops, const P31PassArgs &a, cudaStream_t st);
cudaError_t launch_p31_contig_fwd(int log_l, const P31InnerArgs &a, cudaStream_t st);
cudaError_t launch_p31_inner(int log_l, const P31InnerArgs &a, cudaStream_t st);
// Powers of w in Montgomery form on the device: t[i] = w^i, i < n, prime k
// (w: 2^32 times the root).
constexpr int kP31MaxPowers = 48;
struct P31PowersArgs {
    struct {
        uint32_t *t;
        uint32_t n, w;
        int k;
    } job[kP31MaxPowers];
    int njobs;
};
cudaError_t launch_p31_powers(const P31PowersArgs &a, cudaStream_t st);
cudaError_t launch_p31_build_table(int prime, uint32_t *table, const uint32_t *hi, const uint32_t *lo, int log_m,
                                   int log_s, int use_scale, uint32_t scale, cudaStream_t st);

}  // namespace gbntt
