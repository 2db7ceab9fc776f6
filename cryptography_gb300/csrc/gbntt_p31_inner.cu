// gbntt_p31_inner.cu — innermost passes of the 31-bit prime set: contiguous
// blocks of 2^l points. The fused kernel runs the innermost forward pass of
// both operands, the pointwise product and the innermost inverse pass, all
// between one load of each spectrum and one store of the product; a block's
// values stay in registers but for one exchange through shared memory per
// transform (the inverse starts from the layout the forward transforms
// leave). It also clears the carry kernel's control words, which would
// otherwise be two more launches.
#include "gbntt_p31.cuh"

namespace gbntt {

namespace {

// Position of the second spectrum of (sub-)transform s: one shared spectrum,
// one per pair of products, or the same; transforms of 3 2^k points share
// per sub-transform.
__device__ __forceinline__ long long p31_other(const P31InnerArgs &a, long long s)
{
    if (!a.shared && !a.paired) return s;
    const long long prod = a.r3 ? s / 3 : s, m = a.r3 ? s - 3 * prod : 0;
    const long long o = a.shared ? 0 : prod >> 1;
    return a.r3 ? 3 * o + m : o;
}

template <int LOG_L, bool SQUARE, bool DONE>
__global__ void __launch_bounds__(P31Shape<LOG_L>::T, LOG_L >= 9 ? 2 : LOG_L == 5 ? 8 : 4)
p31_inner_kernel(const __grid_constant__ P31InnerArgs a)
{
    using S = P31Shape<LOG_L>;
    constexpr int A = S::A, B = S::B, G = S::G, L = S::L;
    __shared__ uint32_t sm[S::WORDS_C];
    const int k = blockIdx.x % 3;
    const long long col0 = (long long)(blockIdx.x / 3) * G;
    const uint32_t p = p31_prime(k), pinv = p31_inv(k);
    const int t = threadIdx.x, q = t & (B - 1), g = t >> S::LOG_B;
    const bool live = col0 + g < a.ncols;
    const long long col = live ? col0 + g : 0;   // columns beyond the last one load zeros and store nothing
    chain_wait();
    if (a.zero && k == 0) {
        const long long n = a.nzero, at = (long long)(blockIdx.x / 3) * S::T + t, by = (long long)(gridDim.x / 3) * S::T;
        if (at == 0) a.zero[0] = 0;
        for (long long i = at; i < n; i += by) a.zero[2 + i] = 0;
    }
    uint32_t *d = a.data[k] + (col << LOG_L) + q;
    uint32_t x[A], y[A];
#pragma unroll
    for (int i = 0; i < A; i++) x[i] = live ? d[i * B] : 0u;
    if (!SQUARE) {
        const int lc = a.log_prod - LOG_L;   // columns per (sub-)transform, log
        const long long oc = (p31_other(a, col >> lc) << lc) + (col & ((1LL << lc) - 1));
        const uint32_t *o = a.other[k] + (oc << LOG_L) + q;
        if (DONE) {
#pragma unroll
            for (int r = 0; r < S::R; r++)
#pragma unroll
                for (int kb = 0; kb < B; kb++) y[r * B + kb] = live ? o[r * B + A * kb] : 0u;
        } else {
#pragma unroll
            for (int i = 0; i < A; i++) y[i] = live ? o[i * B] : 0u;
        }
    }
    const ShoupWord *st = a.st[k] + (L - 32), *sti = a.sti[k] + kStep1Words + (L - 32);
    const ShoupWord *wf = c_p31_roots.v[k][0], *wi = c_p31_roots.v[k][1];
    p31_tile_fwd<LOG_L>(x, sm, g, q, wf, st, p);
    if (!SQUARE && !DONE) {
        __syncthreads();
        p31_tile_fwd<LOG_L>(y, sm, g, q, wf, st, p);
    }
#pragma unroll
    for (int i = 0; i < A; i++) x[i] = p31_mont(x[i], SQUARE ? x[i] : y[i], p, pinv);
    __syncthreads();
    p31_tile_inv<LOG_L>(x, sm, g, q, wi, sti, p);
    if (a.use_scale) {
        const uint32_t sc = a.scale[k];
#pragma unroll
        for (int i = 0; i < A; i++) x[i] = p31_mont(x[i], sc, p, pinv);
    }
    if (live) {
#pragma unroll
        for (int i = 0; i < A; i++) d[i * B] = x[i];
    }
}

// The innermost forward pass alone, in place: a right operand that a whole
// wave shares.
template <int LOG_L>
__global__ void __launch_bounds__(P31Shape<LOG_L>::T) p31_contig_fwd_kernel(const __grid_constant__ P31InnerArgs a)
{
    using S = P31Shape<LOG_L>;
    constexpr int A = S::A, B = S::B, G = S::G, L = S::L;
    __shared__ uint32_t sm[S::WORDS_C];
    const int k = blockIdx.x % 3;
    const long long col0 = (long long)(blockIdx.x / 3) * G;
    const uint32_t p = p31_prime(k);
    const int t = threadIdx.x, q = t & (B - 1), g = t >> S::LOG_B;
    const bool live = col0 + g < a.ncols;
    uint32_t *d = a.data[k] + ((live ? col0 + g : 0) << LOG_L) + q;
    uint32_t x[A];
    chain_wait();
#pragma unroll
    for (int i = 0; i < A; i++) x[i] = live ? d[i * B] : 0u;
    p31_tile_fwd<LOG_L>(x, sm, g, q, c_p31_roots.v[k][0], a.st[k] + (L - 32), p);
    if (live) {
#pragma unroll
        for (int r = 0; r < S::R; r++)
#pragma unroll
            for (int kb = 0; kb < B; kb++) d[r * B + A * kb] = x[r * B + kb];
    }
}

template <int LOG_L>
cudaError_t launch_inner_l(const P31InnerArgs &a, cudaStream_t st)
{
    using S = P31Shape<LOG_L>;
    const unsigned grid = (unsigned)(3 * ((a.ncols + S::G - 1) / S::G));
    return launch_chained(!a.other[0]    ? p31_inner_kernel<LOG_L, true, false>
                          : a.other_done ? p31_inner_kernel<LOG_L, false, true>
                                         : p31_inner_kernel<LOG_L, false, false>,
                          dim3(grid), S::T, 0, st, a);
}

template <int LOG_L>
cudaError_t launch_contig_l(const P31InnerArgs &a, cudaStream_t st)
{
    using S = P31Shape<LOG_L>;
    return launch_chained(p31_contig_fwd_kernel<LOG_L>, dim3((unsigned)(3 * ((a.ncols + S::G - 1) / S::G))), S::T, 0, st, a);
}

}  // namespace

cudaError_t launch_p31_inner(int log_l, const P31InnerArgs &a, cudaStream_t st)
{
    switch (log_l) {
    case 5: return launch_inner_l<5>(a, st);
    case 6: return launch_inner_l<6>(a, st);
    case 7: return launch_inner_l<7>(a, st);
    case 8: return launch_inner_l<8>(a, st);
    case 9: return launch_inner_l<9>(a, st);
    case 10: return launch_inner_l<10>(a, st);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_p31_contig_fwd(int log_l, const P31InnerArgs &a, cudaStream_t st)
{
    switch (log_l) {
    case 5: return launch_contig_l<5>(a, st);
    case 6: return launch_contig_l<6>(a, st);
    case 7: return launch_contig_l<7>(a, st);
    case 8: return launch_contig_l<8>(a, st);
    case 9: return launch_contig_l<9>(a, st);
    case 10: return launch_contig_l<10>(a, st);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace gbntt
