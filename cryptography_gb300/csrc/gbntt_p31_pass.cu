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

// Residues of one prime in a launch from which threads take two columns.
// Measured per product, one column and two: 2^19 points 50.6 and 51.0 us (2^20
// residues for both operands), 2^21 128 and 121 us, 2^23 447 and 410 us; at
// 2^17 points the halved number of tiles costs more, 27.0 and 35.1 us.
constexpr long long kTwoColumns = 1LL << 20;

// ... and four of them in 2^9-point passes (2^17 points 18.5 us per product
// with one, 22.4 with four).
constexpr long long kFourColumns = 1LL << 21;

// First column, prime and operand of a CTA. Launches over many sub-problems
// with a large table (by_table) take the CTAs that read the same part of the
// table one after the other, so that it comes from HBM once: grid (prime and
// operand, sub-problem, tile of columns); the others count tiles through.
// Outermost passes over 16 sub-problems of 2^25 points: 6.51 -> 6.04 ms forward,
// 3.09 -> 2.90 ms inverse; over 3 of 2^22 141 -> 129 and 74 -> 61 us.
struct PassTile {
    int k, op;
    long long col0;
};
template <int G>
__device__ __forceinline__ PassTile pass_tile_of(const P31PassArgs &a)
{
    if (a.by_table)
        return {(int)(blockIdx.x % 3), (int)(blockIdx.x / 3),
                ((long long)blockIdx.y << a.log_s) + (long long)blockIdx.z * G};
    return {(int)(blockIdx.x % 3), (int)blockIdx.y, (long long)(blockIdx.x / 3) * G};
}
template <int G>
dim3 pass_grid(P31PassArgs &a, int nops)
{
    const long long subs = a.ncols >> a.log_s, tiles = (1LL << a.log_s) / G;
    a.by_table = a.by_table && subs * nops > 1 && subs <= 65535 && tiles <= 65535;
    if (a.by_table) return dim3((unsigned)(3 * nops), (unsigned)subs, (unsigned)tiles);
    return dim3((unsigned)(3 * (a.ncols / G)), (unsigned)nops);
}

// word at byte offset off of a base address
template <class Word>
__device__ __forceinline__ Word ld_off(const void *base, uint32_t off)
{
    return *reinterpret_cast<const Word *>(reinterpret_cast<const char *>(base) + off);
}
template <class Word>
__device__ __forceinline__ Word ldg_off(const void *base, uint32_t off)
{
    return __ldg(reinterpret_cast<const Word *>(reinterpret_cast<const char *>(base) + off));
}
template <class Word>
__device__ __forceinline__ void st_off(void *base, uint32_t off, Word v)
{
    *reinterpret_cast<Word *>(reinterpret_cast<char *>(base) + off) = v;
}

// w^e (Montgomery form), e < 2^25, from the two-level tables
__device__ __forceinline__ uint32_t p31_tw(const P31PassArgs &a, int k, uint32_t e, uint32_t p, uint32_t pinv)
{
    return p31_mont(__ldg(a.hi[k] + (e >> 15)), __ldg(a.lo[k] + (e & 32767u)), p, pinv);
}

// Shape of a strided tile with V adjacent columns per thread: GP threads
// side by side, G = V GP columns. Exchange words are V residues wide, at
// ka RS + b GP + gp.
template <int LOG_L, int V, int DIR, bool LIMBS = false>
struct P31StridedShape {
    using S = P31Shape<LOG_L>;
    static constexpr int B = S::B;
    static constexpr int GP = V == 1 ? S::G : 16;
    static constexpr int LOG_GP = GP == 8 ? 3 : GP == 16 ? 4 : 5;
    static constexpr int G = V * GP;
    static constexpr int T = GP * B;
    static constexpr int LANES = 32 / V;   // threads served by one shared-memory access
    static constexpr int RS = B * GP + (GP < LANES ? GP : 0);
    static constexpr int MIN_BLOCKS = V == 1 ? (LOG_L >= 9 ? 3 : LOG_L == 5 ? 10 : 5)
                                             : (LOG_L == 8 ? 3 + (DIR || LIMBS) : LOG_L == 5 ? 10 : 6);
};
template <int V>
struct Residues;
template <>
struct Residues<1> {
    typedef uint32_t T;
    static __device__ __forceinline__ uint32_t get(uint32_t x, int) { return x; }
    static __device__ __forceinline__ uint32_t make(const uint32_t *x, int) { return x[0]; }
};
template <>
struct Residues<2> {
    typedef uint2 T;
    static __device__ __forceinline__ uint32_t get(uint2 x, int v) { return v ? x.y : x.x; }
    static __device__ __forceinline__ uint2 make(const uint32_t *x, int n) { return make_uint2(x[0], x[n]); }
};

// One pass over V adjacent columns per thread. With two, the addresses, the
// step twiddles' loads and the memory instructions are shared by two
// residues: 42.5 instead of 50.9 instructions per residue of a 2^8-point
// pass. A forward 2^8-point pass over 6 2^25 residues takes 317 us instead of
// 352, an inverse one over half of them 156 instead of 180 (FMA-heavy pipe
// 76 and 74%, issue 0.69 and 0.70, DRAM 61 and 60%). It wants twice the tiles
// to fill the GPU (launch_l).
template <int LOG_L, int DIR, bool LIMBS, int V>
__global__ void __launch_bounds__(P31StridedShape<LOG_L, V, DIR, LIMBS>::T, P31StridedShape<LOG_L, V, DIR, LIMBS>::MIN_BLOCKS)
p31_pass_kernel(const __grid_constant__ P31PassArgs a)
{
    using S = P31Shape<LOG_L>;
    using H = P31StridedShape<LOG_L, V, DIR, LIMBS>;
    using W = Residues<V>;
    typedef typename W::T Word;
    constexpr int A = S::A, B = S::B, GP = H::GP, RS = H::RS;
    __shared__ Word sm[A * RS];
    const PassTile at = pass_tile_of<H::G>(a);
    const int k = at.k, op = at.op;
    const long long col0 = at.col0;
    const uint32_t p = p31_prime(k), pinv = p31_inv(k);
    const int t = threadIdx.x, gp = t & (GP - 1), q = t >> H::LOG_GP;
    const int log_s = a.log_s;
    const uint32_t sub0 = (uint32_t)((col0 >> log_s) << a.log_m);            // first element of the sub-problem
    const uint32_t j = (uint32_t)(col0 & ((1LL << log_s) - 1)) + V * gp;      // this thread's (first) column
    uint32_t *data = a.data[op][k];
    // byte offsets: elements stay below 2^30 per prime
    const uint32_t step = (uint32_t)B << (log_s + 2);
    const uint32_t off0 = (sub0 + j + ((uint32_t)q << log_s)) << 2;
    uint32_t x[V * A];   // column v's values at x[v A ..]
    chain_wait();
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
        for (int i = 0; i < A; i++)
#pragma unroll
            for (int v = 0; v < V; v++) {
                const uint32_t r = r0 + i * rs + v;
                x[v * A + i] = r < nn ? __ldg(limbs + r) : 0u;
            }
#pragma unroll
        for (int i = 0; i < V * A; i++) x[i] = p31_limb(x[i], p);
    } else {
#pragma unroll
        for (int i = 0; i < A; i++) {
            const Word w = ld_off<Word>(data, off0 + i * step);
#pragma unroll
            for (int v = 0; v < V; v++) x[v * A + i] = W::get(w, v);
        }
    }
    const uint32_t *ptw = a.ptw[k];
    // table address such that an element's own offset indexes it
    const void *tb = reinterpret_cast<const void *>(reinterpret_cast<uintptr_t>(ptw) - ((uintptr_t)sub0 << 2));
    if (DIR == 1) {
        if (ptw) {
            Word tw[A];
#pragma unroll
            for (int i = 0; i < A; i++) tw[i] = ldg_off<Word>(tb, off0 + i * step);
#pragma unroll
            for (int i = 0; i < A; i++)
#pragma unroll
                for (int v = 0; v < V; v++) x[v * A + i] = p31_mont(x[v * A + i], W::get(tw[i], v), p, pinv);
        } else {
            const int sh = kP31MaxLog - a.log_m;
            const uint32_t sc = a.scale[k];
#pragma unroll
            for (int i = 0; i < A; i++)
#pragma unroll
                for (int v = 0; v < V; v++) {
                    uint32_t w = p31_tw(a, k, (uint32_t)(((uint64_t)(i * B + q) * (j + v)) << sh), p, pinv);
                    if (a.use_scale) w = p31_mont(w, sc, p, pinv);
                    x[v * A + i] = p31_mont(x[v * A + i], w, p, pinv);
                }
        }
    }
    // step 1: DFTs over the high digit, step twiddles, exchange
    const ShoupWord *roots = c_p31_roots.v[k][DIR], *__restrict__ st = a.st[k] + (S::L - 32);
#pragma unroll
    for (int v = 0; v < V; v++) p31_dft<S::LOG_A>(x + v * A, roots, p);
    {
        Word *w = sm + q * GP + gp;
#pragma unroll
        for (int ka = 0; ka < A; ka++) {
            uint32_t y[V];
            const int at = p31_bitrev(ka, S::LOG_A);
            if (ka == 0) {
#pragma unroll
                for (int v = 0; v < V; v++) y[v] = x[v * A + at];
            } else {
                const ShoupWord f = st[ka * B + q];
#pragma unroll
                for (int v = 0; v < V; v++) y[v] = p31_shoup(x[v * A + at], f, p);
            }
            w[ka * RS] = W::make(y, 1);
        }
    }
    __syncthreads();
    // step 2: DFTs over the low digit, pass twiddles, store
    const uint32_t row = 4u << log_s;
    const Word *r0 = sm + q * RS + gp;
#pragma unroll
    for (int r = 0; r < S::R; r++) {
        uint32_t y[V * B];
#pragma unroll
        for (int b = 0; b < B; b++) {
            const Word w = r0[r * B * RS + b * GP];
#pragma unroll
            for (int v = 0; v < V; v++) y[v * B + b] = W::get(w, v);
        }
        // twiddles in groups, a group's loads all in flight; with two columns the
        // first group's are issued before the DFT
        constexpr int C = V == 1 ? (B < 16 ? B : 16) : (B < 8 ? B : 8);
        Word tw0[C];
        if (V == 2 && DIR == 0 && ptw) {
#pragma unroll
            for (int c = 0; c < C; c++) tw0[c] = ldg_off<Word>(tb, off0 + (r * B + A * c) * row);
        }
#pragma unroll
        for (int v = 0; v < V; v++) p31_dft<S::LOG_B>(y + v * B, roots, p);
#pragma unroll
        for (int k0 = 0; k0 < B; k0 += C) {
            Word tw[C];
            if (DIR == 0 && ptw) {
#pragma unroll
                for (int c = 0; c < C; c++)
                    tw[c] = V == 2 && k0 == 0 ? tw0[c] : ldg_off<Word>(tb, off0 + (r * B + A * (k0 + c)) * row);
            }
#pragma unroll
            for (int c = 0; c < C; c++) {
                const int kb = k0 + c;
                uint32_t z[V];
#pragma unroll
                for (int v = 0; v < V; v++) z[v] = y[v * B + p31_bitrev(kb, S::LOG_B)];
                if (DIR == 0) {
                    if (ptw) {
#pragma unroll
                        for (int v = 0; v < V; v++) z[v] = p31_mont(z[v], W::get(tw[c], v), p, pinv);
                    } else {
                        const int sh = kP31MaxLog - a.log_m, m = q + r * B + A * kb;
#pragma unroll
                        for (int v = 0; v < V; v++)
                            z[v] = p31_mont(z[v], p31_tw(a, k, (uint32_t)(((uint64_t)m * (j + v)) << sh), p, pinv), p, pinv);
                    }
                }
                st_off<Word>(data, off0 + (r * B + A * kb) * row, W::make(z, 1));
            }
        }
    }
}

// Passes of 2^9 points: three steps of 8-point DFTs over four adjacent
// columns per thread, 32 columns per CTA (rows of 128 bytes). As 32 x 16
// points a thread holds 32 residues of one column, pays for its own addresses
// and loads (62 instructions per residue of a first pass, 54 of an inverse
// one; here 53 and 43) and reads rows of 64 bytes. An operand of at most half
// the transform's length leaves the upper half of step 1 zero. Measured at
// 2^25 points: first pass of both operands 444 -> 416 us, inverse 222 -> 207
// us; two columns of 64-byte rows with the same steps were slower (565 and
// 248 us), and so was skipping the zero half in 2^8-point passes.
// Row m = 64 m2 + 8 m1 + m0; step 1 transforms over m2 (k0 comes out), step 2
// over m1 (k1), step 3 over m0 (k2); the output row is k0 + 8 k1 + 64 k2.
// Exchange word (16 bytes) (k0, m1 | k1, m0) at ((8 k0 + m1) 8 + m0) GP + gp:
// the 8 threads that one access serves are adjacent.
__device__ __forceinline__ uint32_t word4(const uint4 &w, int v)
{
    return v == 0 ? w.x : v == 1 ? w.y : v == 2 ? w.z : w.w;
}

template <int DIR, bool LIMBS>
__global__ void __launch_bounds__(512, 2) p31_pass9_kernel(const __grid_constant__ P31PassArgs a)
{
    constexpr int GP = 8, V = 4;
    extern __shared__ uint4 sm9[];
    const PassTile at = pass_tile_of<V * GP>(a);
    const int k = at.k, op = at.op;
    const long long col0 = at.col0;
    const uint32_t p = p31_prime(k), pinv = p31_inv(k);
    const int t = threadIdx.x, gp = t & (GP - 1), q = t >> 3;
    const int log_s = a.log_s;
    const uint32_t sub0 = (uint32_t)((col0 >> log_s) << a.log_m);
    const uint32_t j = (uint32_t)(col0 & ((1LL << log_s) - 1)) + V * gp;
    uint32_t *data = a.data[op][k];
    const uint32_t step = 256u << log_s;   // 64 rows, in bytes
    const uint32_t off0 = (sub0 + j + ((uint32_t)q << log_s)) << 2;
    uint32_t x[V][8];
    bool upper_zero = false;
    chain_wait();
    if (LIMBS) {
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
        const uint32_t nn = (uint32_t)n, r0 = j + ((uint32_t)q << log_s);
        upper_zero = 2 * n <= 1LL << a.log_m;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            if (h == 1 && upper_zero) break;
#pragma unroll
            for (int i = 4 * h; i < 4 * h + 4; i++)
#pragma unroll
                for (int v = 0; v < V; v++) {
                    const uint32_t r = r0 + ((uint32_t)(64 * i) << log_s) + v;
                    x[v][i] = r < nn ? __ldg(limbs + r) : 0u;
                }
#pragma unroll
            for (int i = 4 * h; i < 4 * h + 4; i++)
#pragma unroll
                for (int v = 0; v < V; v++) x[v][i] = p31_limb(x[v][i], p);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const uint4 w = ld_off<uint4>(data, off0 + i * step);
#pragma unroll
            for (int v = 0; v < V; v++) x[v][i] = word4(w, v);
        }
    }
    const uint32_t *ptw = a.ptw[k];
    const void *tb = reinterpret_cast<const void *>(reinterpret_cast<uintptr_t>(ptw) - ((uintptr_t)sub0 << 2));
    const int sh = kP31MaxLog - a.log_m;
    // pass twiddles of rows r0 + 64 i at byte offset off + i step
    auto twiddle = [&](uint32_t off, int r0) {
        if (ptw) {
#pragma unroll
            for (int i0 = 0; i0 < 8; i0 += 4) {
                uint4 tw[4];
#pragma unroll
                for (int i = 0; i < 4; i++) tw[i] = ldg_off<uint4>(tb, off + (i0 + i) * step);
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int v = 0; v < V; v++) x[v][i0 + i] = p31_mont(x[v][i0 + i], word4(tw[i], v), p, pinv);
            }
        } else {
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int v = 0; v < V; v++) {
                    uint32_t w = p31_tw(a, k, (uint32_t)(((uint64_t)(r0 + 64 * i) * (j + v)) << sh), p, pinv);
                    if (DIR == 1 && a.use_scale) w = p31_mont(w, a.scale[k], p, pinv);
                    x[v][i] = p31_mont(x[v][i], w, p, pinv);
                }
        }
    };
    if (DIR == 1) twiddle(off0, q);
    const ShoupWord *roots = c_p31_roots.v[k][DIR];
    const ShoupWord *__restrict__ st = a.st[k] + kP31Step9;   // w_512^(k0 c) at [64 k0 + c], then w_64^(k1 m0) at [8 k1 + m0]
    // one step's DFTs with its twiddles f[k by], results to w[k stride]
    auto dfts = [&](bool zero) {
#pragma unroll
        for (int v = 0; v < V; v++) p31_dft<3>(x[v], roots, p, zero);
    };
    auto put = [&](uint4 *w, int stride, const ShoupWord *f, int by) {
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int at = p31_bitrev(i, 3);
            uint4 y = make_uint4(x[0][at], x[1][at], x[2][at], x[3][at]);
            if (i > 0) {
                const ShoupWord s = f[i * by];
                y = make_uint4(p31_shoup(y.x, s, p), p31_shoup(y.y, s, p), p31_shoup(y.z, s, p), p31_shoup(y.w, s, p));
            }
            w[i * stride] = y;
        }
    };
    auto get = [&](const uint4 *w, int stride) {
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const uint4 y = w[i * stride];
#pragma unroll
            for (int v = 0; v < V; v++) x[v][i] = word4(y, v);
        }
    };
    dfts(LIMBS && upper_zero);
    put(sm9 + q * GP + gp, 64 * GP, st + q, 64);
    __syncthreads();
    uint4 *const w2 = sm9 + ((q >> 3) * 64 + (q & 7)) * GP + gp;   // (k0, m0)
    get(w2, 8 * GP);
    dfts(false);
    put(w2, 8 * GP, st + 512 + (q & 7), 8);
    __syncthreads();
    get(sm9 + q * 8 * GP + gp, GP);   // (k0, k1) = (q >> 3, q & 7)
    const int row = (q >> 3) + 8 * (q & 7);
    const uint32_t out0 = (sub0 + j + ((uint32_t)row << log_s)) << 2;
    dfts(false);
    {
        uint32_t y[V][8];
#pragma unroll
        for (int v = 0; v < V; v++)
#pragma unroll
            for (int i = 0; i < 8; i++) y[v][i] = x[v][p31_bitrev(i, 3)];
#pragma unroll
        for (int v = 0; v < V; v++)
#pragma unroll
            for (int i = 0; i < 8; i++) x[v][i] = y[v][i];
    }
    if (DIR == 0) twiddle(out0, row);
#pragma unroll
    for (int i = 0; i < 8; i++)
        st_off<uint4>(data, out0 + i * step, make_uint4(x[0][i], x[1][i], x[2][i], x[3][i]));
}

cudaError_t launch_9(int dir, bool limbs, int nops, P31PassArgs &a, cudaStream_t st)
{
    constexpr size_t smem = 64 * 64 * sizeof(uint4);
    static const cudaError_t attr[3] = {
        cudaFuncSetAttribute(p31_pass9_kernel<0, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
        cudaFuncSetAttribute(p31_pass9_kernel<0, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
        cudaFuncSetAttribute(p31_pass9_kernel<1, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)};
    for (const cudaError_t e : attr)
        if (e != cudaSuccess) return e;
    return launch_chained(dir == 1 ? p31_pass9_kernel<1, false>
                          : limbs  ? p31_pass9_kernel<0, true>
                                   : p31_pass9_kernel<0, false>,
                          pass_grid<32>(a, nops), 512, smem, st, a);
}

template <int LOG_L, int V>
cudaError_t launch_v(int dir, bool limbs, int nops, P31PassArgs &a, cudaStream_t st)
{
    using H = P31StridedShape<LOG_L, V, 0>;
    const dim3 grid = pass_grid<H::G>(a, nops);
    return launch_chained(dir == 1 ? p31_pass_kernel<LOG_L, 1, false, V>
                          : limbs  ? p31_pass_kernel<LOG_L, 0, true, V>
                                   : p31_pass_kernel<LOG_L, 0, false, V>,
                          grid, H::T, 0, st, a);
}

template <int LOG_L>
cudaError_t launch_l(int dir, bool limbs, int nops, P31PassArgs &a, cudaStream_t st)
{
    if constexpr (LOG_L <= 8) {   // (more points leave too few warps: 32 or more residues per column in registers)
        if ((a.ncols << LOG_L) * nops >= kTwoColumns) return launch_v<LOG_L, 2>(dir, limbs, nops, a, st);
    }
    return launch_v<LOG_L, 1>(dir, limbs, nops, a, st);
}

// One table per blockIdx.y, a word per thread by repeated squaring (15 steps at
// most): 18 tables, or 42 with the outer stage's, of up to 2^15 words. Bound by
// nothing at this size; it takes the place of 7 ms of host arithmetic.
__global__ void p31_powers_kernel(const __grid_constant__ P31PowersArgs a)
{
    const auto &j = a.job[blockIdx.y];
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= j.n) return;
    const uint32_t p = p31_prime(j.k), pinv = p31_inv(j.k);
    uint32_t x = 0u - 2u * p < p ? 0u - 2u * p : 0u - 3u * p;   // 2^32 mod p, 2 p < 2^32 < 4 p
    uint32_t b = j.w;
    for (uint32_t e = i; e; e >>= 1) {
        if (e & 1) x = p31_mont(x, b, p, pinv);
        b = p31_mont(b, b, p, pinv);
    }
    j.t[i] = x;
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

cudaError_t launch_p31_pass(int log_l, int dir, bool limbs, int nops, const P31PassArgs &args, cudaStream_t st)
{
    P31PassArgs a = args;
    switch (log_l) {
    case 5: return launch_l<5>(dir, limbs, nops, a, st);
    case 6: return launch_l<6>(dir, limbs, nops, a, st);
    case 7: return launch_l<7>(dir, limbs, nops, a, st);
    case 8: return launch_l<8>(dir, limbs, nops, a, st);
    case 9: return (a.ncols << 9) * nops >= kFourColumns ? launch_9(dir, limbs, nops, a, st) : launch_l<9>(dir, limbs, nops, a, st);
    case 10: return launch_l<10>(dir, limbs, nops, a, st);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_p31_powers(const P31PowersArgs &a, cudaStream_t st)
{
    uint32_t n = 0;
    for (int i = 0; i < a.njobs; i++) n = n > a.job[i].n ? n : a.job[i].n;
    if (a.njobs < 1 || a.njobs > kP31MaxPowers || n == 0) return cudaErrorInvalidValue;
    p31_powers_kernel<<<dim3((n + 255) / 256, (unsigned)a.njobs), 256, 0, st>>>(a);
    return cudaGetLastError();
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
