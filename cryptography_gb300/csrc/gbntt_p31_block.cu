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
#include "gbntt_carry.cuh"
#include "gbntt_p31.cuh"
#include "gbntt_p31_garner.cuh"

namespace gbntt {

namespace {

// N = 2^LOG_N points, E per thread, in steps of radix E (the last one of
// what is left): N / E threads per transform. Up to 2^11 points the two
// operands are transformed by different threads.
template <int LOG_N>
struct BlockShape {
    static constexpr int N = 1 << LOG_N;
    static constexpr int LOG_E = LOG_N >= 10 ? 4 : LOG_N >= 8 ? 3 : 2;
    static constexpr int E = 1 << LOG_E;
    static constexpr int TP = N / E;                       // threads per transform
    static constexpr int OPS = LOG_N == 12 ? 1 : 2;        // operands side by side
    static constexpr int T = (3 * OPS * TP + 31) / 32 * 32;
    static constexpr int STEPS = (LOG_N + LOG_E - 1) / LOG_E;
    static constexpr int NP = N + N / 16;                  // words of a spectrum with its padding
    static constexpr int K = (N + 3 + T - 1) / T;          // product limbs per thread
    static constexpr size_t SMEM = 6 * (size_t)NP * sizeof(uint32_t);
    static constexpr int log_r(int step) { return step < STEPS - 1 ? LOG_E : LOG_N - LOG_E * (STEPS - 1); }
    static constexpr int log_m(int step) { return LOG_N - LOG_E * step; }
};

__device__ __forceinline__ int bpad(int i) { return i + (i >> 4); }

// One forward step (radix 2^LOG_R on sub-blocks of 2^LOG_M points) of the
// transform in s: thread t takes E / R of its DFTs, in place. FIRST: values
// come from limbs; LAST: results stay in x.
template <int LOG_N, int STEP>
struct BlockStep {
    using S = BlockShape<LOG_N>;
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
template <int LOG_N, int STEP>
__device__ __forceinline__ const uint32_t *step_table(const uint32_t *tw)
{
    int off = 0;
#pragma unroll
    for (int s = 0; s < STEP; s++) off += 1 << BlockShape<LOG_N>::log_m(s);
    return tw + off;
}

template <int LOG_N, int STEP>
__device__ __forceinline__ void fwd_step(uint32_t *x, uint32_t *s, int t, const uint32_t *tw, const ShoupWord *roots,
                                         uint32_t p, uint32_t pinv)
{
    using B = BlockStep<LOG_N, STEP>;
    constexpr bool last = STEP == BlockShape<LOG_N>::STEPS - 1;
    const uint32_t *tab = step_table<LOG_N, STEP>(tw);
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

template <int LOG_N, int STEP>
__device__ __forceinline__ void inv_step(uint32_t *x, uint32_t *s, int t, const uint32_t *tw, const ShoupWord *roots,
                                         uint32_t p, uint32_t pinv)
{
    using B = BlockStep<LOG_N, STEP>;
    constexpr bool first = STEP == BlockShape<LOG_N>::STEPS - 1;
    const uint32_t *tab = step_table<LOG_N, STEP>(tw);
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
template <int LOG_N, int STEP>
__device__ __forceinline__ void fwd_rest(bool on, uint32_t *x, uint32_t *s, int t, const uint32_t *tw,
                                         const ShoupWord *roots, uint32_t p, uint32_t pinv)
{
    if constexpr (STEP < BlockShape<LOG_N>::STEPS) {
        __syncthreads();
        if (on) fwd_step<LOG_N, STEP>(x, s, t, tw, roots, p, pinv);
        fwd_rest<LOG_N, STEP + 1>(on, x, s, t, tw, roots, p, pinv);
    }
}
// steps STEP .. 0 of an inverse transform, a barrier after each
template <int LOG_N, int STEP>
__device__ __forceinline__ void inv_rest(bool on, uint32_t *x, uint32_t *s, int t, const uint32_t *tw,
                                         const ShoupWord *roots, uint32_t p, uint32_t pinv)
{
    if constexpr (STEP >= 0) {
        if (on) inv_step<LOG_N, STEP>(x, s, t, tw, roots, p, pinv);
        __syncthreads();
        inv_rest<LOG_N, STEP - 1>(on, x, s, t, tw, roots, p, pinv);
    }
}

template <int LOG_N>
__global__ void __launch_bounds__(BlockShape<LOG_N>::T) p31_block_kernel(const __grid_constant__ P31BlockArgs a)
{
    using S = BlockShape<LOG_N>;
    constexpr int N = S::N, E = S::E, TP = S::TP, OPS = S::OPS, T = S::T, K = S::K, NP = S::NP;
    extern __shared__ uint32_t sm[];   // spectra of the first operand (3 NP words), then of the second
    __shared__ unsigned s_warp[T / 32];
    const int tid = threadIdx.x;
    const uint32_t *in[2];
    long long len[2];
    uint32_t *out;
    long long n_out;
    const long long b = blockIdx.x;
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
    const int k = grp % 3, op0 = grp / 3;   // op0 >= OPS: a thread that only fills the last warp
    const bool on = op0 < OPS;
    const uint32_t p = p31_prime(k), pinv = p31_inv(k);
    const ShoupWord *wf = c_p31_roots.v[k][0], *wi = c_p31_roots.v[k][1];
    const uint32_t *tf = a.tw[k][0], *ti = a.tw[k][1];
    uint32_t x[E];
    using First = BlockStep<LOG_N, 0>;
    // forward: with OPS == 2 each group its operand, else the second operand
    // and then the first, whose spectrum is left in registers
#pragma unroll
    for (int pass = 0; pass < 3 - OPS; pass++) {
        const int op = OPS == 2 ? op0 : 1 - pass;
        uint32_t *s = sm + (op * 3 + k) * NP;
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
            fwd_step<LOG_N, 0>(x, s, t, tf, wf, p, pinv);
        }
        fwd_rest<LOG_N, 1>(go, x, s, t, tf, wf, p, pinv);
        if (go && op == 1) {   // the second operand's spectrum goes where the first one's threads read it
            using Last = BlockStep<LOG_N, S::STEPS - 1>;
#pragma unroll
            for (int r = 0; r < Last::D; r++)
#pragma unroll
                for (int i = 0; i < Last::R; i++) s[bpad(Last::base(t, r) + i)] = x[r * Last::R + i];
        }
    }
    __syncthreads();
    const bool first = on && (OPS == 1 || op0 == 0);
    uint32_t *s = sm + k * NP;
    if (first) {
        // pointwise product times the factor 2^32 / N (the Montgomery
        // product and the scale)
        using Last = BlockStep<LOG_N, S::STEPS - 1>;
        const uint32_t *o = s + 3 * NP;
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
    inv_rest<LOG_N, S::STEPS - 1>(first, x, s, t, ti, wi, p, pinv);

    // Garner: the words of every coefficient into the second operand's area
    uint32_t *W0 = sm + 3 * NP, *W1 = W0 + NP, *W2 = W1 + NP;
    unsigned err = 0;
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
    if (a.sticky && tid == 0) err |= atomicExch(a.sticky, 0u);
    if (err) atomicOr(a.error, err);
}

template <int LOG_N>
cudaError_t launch_n(const P31BlockArgs &a, long long W, cudaStream_t st)
{
    using S = BlockShape<LOG_N>;
    static_assert(S::K * S::T <= 3 * S::NP && S::K * S::T >= S::N + 3, "limb staging");
    auto fn = p31_block_kernel<LOG_N>;
    if (S::SMEM > 48 * 1024) {
        static const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM);
        if (e != cudaSuccess) return e;
    }
    return launch_chained(fn, dim3((unsigned)W), S::T, S::SMEM, st, a);
}

template <int LOG_N>
int fill_tables(uint32_t *dst, uint64_t w, uint64_t p)   // w of order N; returns the words
{
    using S = BlockShape<LOG_N>;
    int off = 0;
    for (int s = 0; s < S::STEPS - 1; s++) {
        const int lm = S::log_m(s), ls = lm - S::log_r(s);
        const uint64_t wm = p31_pow(w, 1ull << (LOG_N - lm), p);
        for (int k = 0; k < 1 << S::log_r(s); k++) {
            const uint64_t wk = p31_pow(wm, (uint64_t)k, p);
            uint64_t x = 1;
            for (int j = 0; j < 1 << ls; j++) {
                dst[off + (k << ls) + j] = (uint32_t)((x << 32) % p);
                x = x * wk % p;
            }
        }
        off += 1 << lm;
    }
    return off;
}

}  // namespace

cudaError_t launch_p31_block(int log_n, const P31BlockArgs &a, long long W, cudaStream_t st)
{
    switch (log_n) {
    case 5: return launch_n<5>(a, W, st);
    case 6: return launch_n<6>(a, W, st);
    case 7: return launch_n<7>(a, W, st);
    case 8: return launch_n<8>(a, W, st);
    case 9: return launch_n<9>(a, W, st);
    case 10: return launch_n<10>(a, W, st);
    case 11: return launch_n<11>(a, W, st);
    case 12: return launch_n<12>(a, W, st);
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
