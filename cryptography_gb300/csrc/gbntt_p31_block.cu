// gbntt_p31_block.cu — whole products of up to 2^12 coefficients in one CTA:
// limbs in, product limbs out, one launch for a product or for a wave of
// them (one CTA each).
//
// A product this short is bound by launches and by the latency of each
// step's dependent chain, not by any pipe: the pass chain needs at least a
// first pass, the fused innermost pass, an inverse pass and the carry
// kernel, each a launch that waits for the one before it. Here the spectra
// of the three 31-bit primes stay in shared memory, groups of threads take
// one (prime, operand) each, and Garner and the carries follow in the same
// CTA. Above 2^12 points the six spectra no longer fit beside a second CTA.
#include <cooperative_groups.h>
#include "gbntt_carry.cuh"
#include "gbntt_p31.cuh"
#include "gbntt_p31_garner.cuh"

namespace gbntt {

namespace {

namespace cg = cooperative_groups;

// Up to this many products of 2^10 points and more take a cluster of three
// CTAs each, one per prime (3 kClusterW CTAs fill the GPU once). Measured, one
// CTA and three: one product of 2^12 points 20.1 and 10.5 us, of 2^11 11.9 and
// 8.2, of 2^10 7.0 and 6.6; a wave of 50 24.6 and 22.2, 16.5 and 14.9, 12.3 and
// 12.0; of 152 24.8 and 38.1, 16.5 and 20.8, 11.6 and 13.4.
constexpr long long kClusterW = 50;

// N = 2^LOG_N points, E per thread, in steps of radix E (the last one of
// what is left): N / E threads per transform. Up to 2^11 points the two
// operands are transformed by different threads.
template <int LOG_N, bool CL>
struct BlockShape {
    static constexpr int N = 1 << LOG_N;
    static constexpr int PRIMES = CL ? 1 : 3;              // primes per CTA
    static constexpr int LOG_E = LOG_N >= 10 ? 4 : LOG_N >= 8 ? 3 : 2;
    static constexpr int E = 1 << LOG_E;
    static constexpr int TP = N / E;                       // threads per transform
    static constexpr int OPS = PRIMES * 2 * TP > 1024 ? 1 : 2;   // operands side by side
    static constexpr int T = (PRIMES * OPS * TP + 31) / 32 * 32;
    static constexpr int STEPS = (LOG_N + LOG_E - 1) / LOG_E;
    static constexpr int NP = N + N / 16;                  // words of a spectrum with its padding
    static constexpr int K = ((CL ? (N + 5) / 3 : N + 3) + T - 1) / T;   // product limbs per thread
    static constexpr int SPAN = K * T;                     // ... and per CTA
    static constexpr int WP = SPAN + 2 + (SPAN + 2) / 16 + 1;   // words of a CTA's coefficients, padded
    static constexpr size_t SMEM = (CL ? NP + (NP > 3 * WP ? NP : 3 * WP) : 6 * (size_t)NP) * sizeof(uint32_t);
    static constexpr int log_r(int step) { return step < STEPS - 1 ? LOG_E : LOG_N - LOG_E * (STEPS - 1); }
    static constexpr int log_m(int step) { return LOG_N - LOG_E * step; }
};

__device__ __forceinline__ int bpad(int i) { return i + (i >> 4); }

// One forward step (radix 2^LOG_R on sub-blocks of 2^LOG_M points) of the
// transform in s: thread t takes E / R of its DFTs, in place. FIRST: values
// come from limbs; LAST: results stay in x.
template <class S_, int STEP>
struct BlockStep {
    using S = S_;
    static constexpr int LOG_R = S::log_r(STEP), R = 1 << LOG_R, LOG_M = S::log_m(STEP), LOG_S = LOG_M - LOG_R;
    static constexpr int D = S::E / R;
    static __device__ __forceinline__ int base(int t, int r)
    {
        const int d = t + r * S::TP;
        return ((d >> LOG_S) << LOG_M) + (d & ((1 << LOG_S) - 1));
    }
    static __device__ __forceinline__ int column(int t, int r) { return (t + r * S::TP) & ((1 << LOG_S) - 1); }
};

// Twiddles of a step: w_M^(+-j k) in Montgomery form at [k S + j] of the
// step's M-word table.
template <class S, int STEP>
__device__ __forceinline__ const uint32_t *step_table(const uint32_t *tw)
{
    int off = 0;
#pragma unroll
    for (int s = 0; s < STEP; s++) off += 1 << S::log_m(s);
    return tw + off;
}

template <class S, int STEP>
__device__ __forceinline__ void fwd_step(uint32_t *x, uint32_t *s, int t, const uint32_t *tw, const ShoupWord *roots,
                                         uint32_t p, uint32_t pinv)
{
    using B = BlockStep<S, STEP>;
    constexpr bool last = STEP == S::STEPS - 1;
    const uint32_t *tab = step_table<S, STEP>(tw);
#pragma unroll
    for (int r = 0; r < B::D; r++) {
        uint32_t *y = x + r * B::R;
        const int b = B::base(t, r), j = B::column(t, r);
        if (STEP > 0) {
#pragma unroll
            for (int i = 0; i < B::R; i++) y[i] = s[bpad(b + (i << B::LOG_S))];
        }
        p31_dft<B::LOG_R>(y, roots, p);
        if (!last) {
#pragma unroll
            for (int k = 0; k < B::R; k++) {
                uint32_t v = y[p31_bitrev(k, B::LOG_R)];
                if (k > 0) v = p31_mont(v, __ldg(tab + (k << B::LOG_S) + j), p, pinv);
                s[bpad(b + (k << B::LOG_S))] = v;
            }
        }
    }
}

template <class S, int STEP>
__device__ __forceinline__ void inv_step(uint32_t *x, uint32_t *s, int t, const uint32_t *tw, const ShoupWord *roots,
                                         uint32_t p, uint32_t pinv)
{
    using B = BlockStep<S, STEP>;
    constexpr bool first = STEP == S::STEPS - 1;
    const uint32_t *tab = step_table<S, STEP>(tw);
#pragma unroll
    for (int r = 0; r < B::D; r++) {
        uint32_t y[B::R];
        const int b = B::base(t, r), j = B::column(t, r);
        if (first) {   // from the registers of the last forward step
#pragma unroll
            for (int k = 0; k < B::R; k++) y[k] = x[r * B::R + p31_bitrev(k, B::LOG_R)];
        } else {
#pragma unroll
            for (int k = 0; k < B::R; k++) {
                uint32_t v = s[bpad(b + (k << B::LOG_S))];
                if (k > 0) v = p31_mont(v, __ldg(tab + (k << B::LOG_S) + j), p, pinv);
                y[k] = v;
            }
        }
        p31_dft<B::LOG_R>(y, roots, p);
#pragma unroll
        for (int i = 0; i < B::R; i++) s[bpad(b + (i << B::LOG_S))] = y[p31_bitrev(i, B::LOG_R)];
    }
}

// steps 1 .. STEPS - 1 of a forward transform, a barrier before each
template <class S, int STEP>
__device__ __forceinline__ void fwd_rest(bool on, uint32_t *x, uint32_t *s, int t, const uint32_t *tw,
                                         const ShoupWord *roots, uint32_t p, uint32_t pinv)
{
    if constexpr (STEP < S::STEPS) {
        __syncthreads();
        if (on) fwd_step<S, STEP>(x, s, t, tw, roots, p, pinv);
        fwd_rest<S, STEP + 1>(on, x, s, t, tw, roots, p, pinv);
    }
}
// steps STEP .. 0 of an inverse transform, a barrier after each
template <class S, int STEP>
__device__ __forceinline__ void inv_rest(bool on, uint32_t *x, uint32_t *s, int t, const uint32_t *tw,
                                         const ShoupWord *roots, uint32_t p, uint32_t pinv)
{
    if constexpr (STEP >= 0) {
        if (on) inv_step<S, STEP>(x, s, t, tw, roots, p, pinv);
        __syncthreads();
        inv_rest<S, STEP - 1>(on, x, s, t, tw, roots, p, pinv);
    }
}

template <int LOG_N, bool CL>
__global__ void __launch_bounds__(BlockShape<LOG_N, CL>::T) p31_block_kernel(const __grid_constant__ P31BlockArgs a)
{
    using S = BlockShape<LOG_N, CL>;
    constexpr int PRIMES = S::PRIMES;
    constexpr int N = S::N, E = S::E, TP = S::TP, OPS = S::OPS, T = S::T, K = S::K, NP = S::NP;
    extern __shared__ uint32_t sm[];   // spectra of the first operand (PRIMES x NP words), then of the second
    __shared__ unsigned s_warp[T / 32];
    const int tid = threadIdx.x;
    const uint32_t *in[2];
    long long len[2];
    uint32_t *out;
    long long n_out;
    const int rank = CL ? (int)(blockIdx.x % 3) : 0;   // CTA of its cluster: the prime, and the third of the limbs
    const long long b = CL ? blockIdx.x / 3 : blockIdx.x;
    chain_wait();
    if (a.limb_tab[0]) {
        const long long bb = a.shared ? 0 : a.paired ? b >> 1 : b;
        in[0] = a.limb_tab[0][b];
        len[0] = a.len_tab[0][b];
        in[1] = a.limb_tab[1][bb];
        len[1] = a.len_tab[1][bb];
        out = a.out_tab[b];
        n_out = a.nout_tab[b];
    } else {
        in[0] = a.limbs[0];
        in[1] = a.limbs[1];
        len[0] = a.n_limbs[0];
        len[1] = a.n_limbs[1];
        out = a.out;
        n_out = a.n_out;
    }
    const bool square = in[0] == in[1] && len[0] == len[1];
    const int grp = tid / TP, t = tid - grp * TP;
    const int k = CL ? rank : grp % 3, slot = CL ? 0 : k, op0 = grp / PRIMES;   // op0 >= OPS: a thread that only fills the last warp
    const bool on = op0 < OPS;
    const uint32_t p = p31_prime(k), pinv = p31_inv(k);
    const ShoupWord *wf = c_p31_roots.v[k][0], *wi = c_p31_roots.v[k][1];
    const uint32_t *tf = a.tw[k][0], *ti = a.tw[k][1];
    uint32_t x[E];
    using First = BlockStep<S, 0>;
    // forward: with OPS == 2 each group its operand, else the second operand
    // and then the first, whose spectrum is left in registers
#pragma unroll
    for (int pass = 0; pass < 3 - OPS; pass++) {
        const int op = OPS == 2 ? op0 : 1 - pass;
        uint32_t *s = sm + (op * PRIMES + slot) * NP;
        const bool go = on && !(op == 1 && square);
        if (go) {
            const uint32_t *v = in[op];
            const long long n = len[op];
#pragma unroll
            for (int r = 0; r < First::D; r++)
#pragma unroll
                for (int i = 0; i < First::R; i++) {
                    const int e = First::base(t, r) + (i << First::LOG_S);
                    x[r * First::R + i] = e < n ? __ldg(v + e) : 0u;
                }
#pragma unroll
            for (int i = 0; i < E; i++) x[i] = p31_limb(x[i], p);
            fwd_step<S, 0>(x, s, t, tf, wf, p, pinv);
        }
        fwd_rest<S, 1>(go, x, s, t, tf, wf, p, pinv);
        if (go && op == 1) {   // the second operand's spectrum goes where the first one's threads read it
            using Last = BlockStep<S, S::STEPS - 1>;
#pragma unroll
            for (int r = 0; r < Last::D; r++)
#pragma unroll
                for (int i = 0; i < Last::R; i++) s[bpad(Last::base(t, r) + i)] = x[r * Last::R + i];
        }
    }
    __syncthreads();
    const bool first = on && (OPS == 1 || op0 == 0);
    uint32_t *s = sm + slot * NP;
    if (first) {
        // pointwise product times the factor 2^32 / N (the Montgomery
        // product and the scale)
        using Last = BlockStep<S, S::STEPS - 1>;
        const uint32_t *o = s + PRIMES * NP;
        const ShoupWord sc = a.scale[k];
#pragma unroll
        for (int r = 0; r < Last::D; r++)
#pragma unroll
            for (int i = 0; i < Last::R; i++) {
                uint32_t &v = x[r * Last::R + i];
                v = p31_mont(p31_shoup_lazy(v, sc, p), square ? v : o[bpad(Last::base(t, r) + i)], p, pinv);
            }
    }
    __syncthreads();   // the last forward step's reads of s are done before the inverse steps write it
    inv_rest<S, S::STEPS - 1>(first, x, s, t, ti, wi, p, pinv);

    unsigned err = 0;
    if constexpr (CL) {
        // this CTA's limbs [first, first + SPAN), from coefficients first - 2
        // on: the other primes' residues come from the other CTAs, the
        // carry into the span from their transfer functions
        cg::cluster_group cluster = cg::this_cluster();
        __shared__ unsigned s_agg[2];
        const int first_limb = rank * S::SPAN;
        uint32_t *W0 = sm + NP, *W1 = W0 + S::WP, *W2 = W1 + S::WP;
        const uint32_t *res[3];
#pragma unroll
        for (int q = 0; q < 3; q++) res[q] = cluster.map_shared_rank(sm, q);
        cluster.sync();   // every CTA's residues are in place
        for (int i = tid; i < S::SPAN + 2; i += T) {
            const int j = first_limb - 2 + i;
            uint32_t w0 = 0, w1 = 0, w2 = 0;
            if (j >= 0 && j < N) garner31(res[0][bpad(j)], res[1][bpad(j)], res[2][bpad(j)], w0, w1, w2);
            if (w2 >= (uint32_t)N) err |= ERR_GARNER_DIGIT;
            W0[bpad(i)] = w0;
            W1[bpad(i)] = w1;
            W2[bpad(i)] = w2;
        }
        __syncthreads();
        uint64_t sum[K];
#pragma unroll
        for (int i = 0; i < K; i++) {
            const int q = tid * K + i;
            sum[i] = (uint64_t)W0[bpad(q + 2)] + W1[bpad(q + 1)] + W2[bpad(q)];
        }
        unsigned agg;
        const unsigned before = block_scan_transfer<T>(run_transfer<K>(sum), s_warp, &agg);
        if (tid > rank && tid < 3) *cluster.map_shared_rank(&s_agg[rank < 2 ? rank : 0], tid) = agg;
        cluster.sync();   // residues read by all, transfer functions of the lower CTAs here
        unsigned cin = 0;
        for (int q = 0; q < rank; q++) cin = fn_apply(s_agg[q], cin);
        uint64_t c = fn_apply(before, cin);
#pragma unroll
        for (int i = 0; i < K; i++) {
            const uint64_t v = sum[i] + c;
            c = v >> 32;
            W0[tid * K + i] = (uint32_t)v;   // the words are dead (every thread has its sums)
        }
        __syncthreads();
        for (int j = tid; j < S::SPAN; j += T)
            if (first_limb + j < n_out) out[first_limb + j] = W0[j];
    } else {
        // Garner: the words of every coefficient into the second operand's area
        uint32_t *W0 = sm + 3 * NP, *W1 = W0 + NP, *W2 = W1 + NP;
        for (int j = tid; j < N; j += T) {
            uint32_t w0, w1, w2;
            garner31(sm[bpad(j)], sm[NP + bpad(j)], sm[2 * NP + bpad(j)], w0, w1, w2);
            if (w2 >= (uint32_t)N) err |= ERR_GARNER_DIGIT;
            W0[bpad(j)] = w0;
            W1[bpad(j)] = w1;
            W2[bpad(j)] = w2;
        }
        __syncthreads();
        // limb sums, carries, store (limbs through shared memory)
        uint64_t sum[K];
    #pragma unroll
        for (int i = 0; i < K; i++) {
            const int j = tid * K + i;
            sum[i] = (uint64_t)(j < N ? W0[bpad(j)] : 0u) + (j >= 1 && j - 1 < N ? W1[bpad(j - 1)] : 0u) +
                     (j >= 2 && j - 2 < N ? W2[bpad(j - 2)] : 0u);
        }
        unsigned agg;
        const unsigned before = block_scan_transfer<T>(run_transfer<K>(sum), s_warp, &agg);
        uint64_t c = fn_apply(before, 0);
    #pragma unroll
        for (int i = 0; i < K; i++) {
            const uint64_t v = sum[i] + c;
            c = v >> 32;
            sm[tid * K + i] = (uint32_t)v;   // the residues are dead; K T <= 3 NP
        }
        __syncthreads();
        for (int j = tid; j < K * T; j += T)
            if (j < n_out) out[j] = sm[j];
    }
    if (a.sticky && tid == 0 && rank == 0) err |= atomicExch(a.sticky, 0u);
    if (err) atomicOr(a.error, err);
}

template <int LOG_N, bool CL>
cudaError_t launch_n(const P31BlockArgs &a, long long W, cudaStream_t st)
{
    using S = BlockShape<LOG_N, CL>;
    static_assert(CL ? 3 * S::SPAN >= S::N + 3 : S::SPAN <= 3 * S::NP && S::SPAN >= S::N + 3, "limb staging");
    auto fn = p31_block_kernel<LOG_N, CL>;
    if (S::SMEM > 48 * 1024) {
        static const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM);
        if (e != cudaSuccess) return e;
    }
    return launch_chained(fn, dim3((unsigned)(CL ? 3 * W : W)), S::T, S::SMEM, st, a, CL ? 3 : 1);
}

template <int LOG_N>
int fill_tables(uint32_t *dst, uint64_t w, uint64_t p)   // w of order N; returns the words
{
    using S = BlockShape<LOG_N, false>;   // (the steps are the same for clusters)
    int off = 0;
    for (int s = 0; s < S::STEPS - 1; s++) {
        const int lm = S::log_m(s), ls = lm - S::log_r(s);
        const uint64_t wm = p31_pow(w, 1ull << (LOG_N - lm), p);
        for (int k = 0; k < 1 << S::log_r(s); k++) {
            p31_powers(dst + off + (k << ls), (size_t)1 << ls, p31_pow(wm, (uint64_t)k, p), p);
        }
        off += 1 << lm;
    }
    return off;
}

}  // namespace

cudaError_t launch_p31_block(int log_n, const P31BlockArgs &a, long long W, cudaStream_t st)
{
    const bool cl = log_n >= 10 && W <= kClusterW;
    switch (log_n) {
    case 5: return launch_n<5, false>(a, W, st);
    case 6: return launch_n<6, false>(a, W, st);
    case 7: return launch_n<7, false>(a, W, st);
    case 8: return launch_n<8, false>(a, W, st);
    case 9: return launch_n<9, false>(a, W, st);
    case 10: return cl ? launch_n<10, true>(a, W, st) : launch_n<10, false>(a, W, st);
    case 11: return cl ? launch_n<11, true>(a, W, st) : launch_n<11, false>(a, W, st);
    case 12: return cl ? launch_n<12, true>(a, W, st) : launch_n<12, false>(a, W, st);
    default: return cudaErrorInvalidValue;
    }
}

// The step tables of 2^log_n points for the root w of that order.
int p31_block_tables(int log_n, uint32_t *dst, uint64_t w, uint64_t p)
{
    switch (log_n) {
    case 5: return fill_tables<5>(dst, w, p);
    case 6: return fill_tables<6>(dst, w, p);
    case 7: return fill_tables<7>(dst, w, p);
    case 8: return fill_tables<8>(dst, w, p);
    case 9: return fill_tables<9>(dst, w, p);
    case 10: return fill_tables<10>(dst, w, p);
    case 11: return fill_tables<11>(dst, w, p);
    default: return fill_tables<12>(dst, w, p);
    }
}

}  // namespace gbntt
