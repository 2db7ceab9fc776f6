// gbntt_p31_outer.cu — products of more than 2^25 coefficients on the 31-bit
// primes.
//
// The primes' roots of unity end at 2^25, so a product of up to R M
// coefficients (M = 2^25; R = 2, 4 .. 16, 3 M points being the radix-3
// stage's) is computed modulo R polynomials X^M - c_m that do have M-th roots
// of c_m: c_m = gamma^m, gamma = g^M, for a g of order d M with d = (p - 1) / M
// = 60, 54 and 63 in the three primes (gamma has order d >= R, so the c_m
// differ).
//   forward  y_m[j] = g^(jm) sum_r x[j + r M] gamma^(rm)     (A mod X^M - c_m
//            under X -> g^m X, a cyclic convolution of length M)
//   inverse  t_m = z_m[j] g^(-jm), x[j + r M] = sum_m V^-1[r][m] t_m with the
//            Vandermonde matrix V[m][r] = gamma^(rm).
// Two of the primes have -1 among the M-th powers (d even): there, for even
// R, the c_m are pairs +-gamma^i, and the even- and odd-indexed blocks are
// two sums of half the length, added and subtracted (forward 80 to 60, inverse
// 112 to 80 cycles per residue, warp and SM sub-partition at R = 16).
// A dense R x R product instead of log2 R radix-2 levels: one wide multiply
// per term, the high word folded every second term, one Montgomery reduction
// per sum. It costs about as much as 8 levels of the pass chain at R = 16 (of
// 25), against the 64-bit primes' doubled arithmetic on every level; and R
// need not be a power of two. The shorter operand may have 2^28 limbs (the
// modulus is 2^92.64).
#include <vector>
#include "gbntt_p31.cuh"

namespace gbntt {

namespace {

constexpr int kMaxR = kP31MaxOuter;
constexpr uint32_t kM = 1u << kP31MaxLog;

constexpr uint64_t outer_order(int k) { return (kP31[k] - 1ull) / kM; }   // d
static_assert(outer_order(0) >= kMaxR && outer_order(1) >= kMaxR && outer_order(2) >= kMaxR, "distinct c_m");
constexpr uint64_t outer_g(int k) { return kP31Gen[k]; }   // of order d M = p - 1

// gamma^(rm) per prime, Montgomery form, row m
struct ForwardMatrix {
    uint32_t v[3][kMaxR][kMaxR];
};
constexpr ForwardMatrix forward_matrix()
{
    ForwardMatrix f{};
    for (int k = 0; k < 3; k++) {
        const uint64_t p = kP31[k], gamma = p31_pow(outer_g(k), kM, p);
        for (int m = 0; m < kMaxR; m++) {
            const uint64_t cm = p31_pow(gamma, (uint64_t)m, p);
            uint64_t x = 1;
            for (int r = 0; r < kMaxR; r++) {
                f.v[k][m][r] = (uint32_t)((x << 32) % p);
                x = x * cm % p;
            }
        }
    }
    return f;
}
__constant__ const ForwardMatrix c_fwd = forward_matrix();
// V^-1 for each R, Montgomery form, row r at [R][k][r kMaxR + m]; for paired
// points the two matrices of R / 2 rows that take the pairs' sums to the
// even blocks ([s kMaxR + i]) and their differences to the odd ones
// ([s kMaxR + kMaxR / 2 + i])
__constant__ uint32_t c_inv[kMaxR + 1][3][kMaxR * kMaxR];

struct Acc {
    uint64_t s = 0;
    __device__ __forceinline__ void add(uint32_t a, uint32_t b) { s += (uint64_t)a * b; }
    // the high word back below p (after at most two products)
    __device__ __forceinline__ void fold(uint32_t p)
    {
        const uint32_t h = (uint32_t)(s >> 32);
        s = ((uint64_t)__viaddmin_u32(h, 0u - p, h) << 32) | (uint32_t)s;
    }
    __device__ __forceinline__ uint32_t reduce(uint32_t p, uint32_t pinv) const
    {
        const uint32_t m = (uint32_t)s * pinv;
        const uint32_t d = (uint32_t)(s >> 32) - __umulhi(m, p);
        return __viaddmin_u32(d, p, d);
    }
};

__host__ __device__ constexpr bool outer_paired(int R, int k) { return R % 2 == 0 && k < 2; }

// g^(+-j), Montgomery form
__device__ __forceinline__ uint32_t g_pow(const uint32_t *t, uint32_t j, uint32_t p, uint32_t pinv)
{
    return p31_mont(__ldg(t + (j >> 15)), __ldg(t + (kM >> 15) + (j & 32767u)), p, pinv);
}

// The R residues modulo prime k of column j, from its limbs in ni blocks.
template <int R>
__device__ __forceinline__ void outer_fwd(const P31OuterArgs &a, int k, uint32_t j, int ni, const uint32_t (&limb)[R])
{
    const uint32_t p = p31_prime(k), pinv = p31_inv(k);
    uint32_t x[R];
#pragma unroll
    for (int r = 0; r < R; r++) x[r] = p31_limb(limb[r], p);
    const uint32_t w1 = g_pow(a.g[k], j, p, pinv);
    uint32_t w = w1;
    uint32_t *out = a.spec[k] + j;
    if (outer_paired(R, k)) {
        const uint32_t h = g_pow(a.gh[k], j, p, pinv);   // g^(j d / 2): the twist between a pair's points
#pragma unroll
        for (int i = 0; i < R / 2; i++) {
            Acc even, odd;
#pragma unroll
            for (int r0 = 0; r0 < R; r0 += 4)
                if (r0 == 0 || r0 < ni) {
#pragma unroll
                    for (int r = r0; r < r0 + 4 && r < R; r += 2) {
                        even.add(x[r], c_fwd.v[k][i][r]);
                        odd.add(x[r + 1], c_fwd.v[k][i][r + 1]);
                    }
                    even.fold(p);
                    odd.fold(p);
                }
            const uint32_t e = even.reduce(p, pinv), o = odd.reduce(p, pinv);
            const uint32_t y0 = p31_add(e, o, p), y1 = p31_sub(e, o, p);
            if (i == 0) {
                out[0] = y0;
                out[kM] = p31_mont(y1, h, p, pinv);
            } else {
                out[(size_t)(2 * i) * kM] = p31_mont(y0, w, p, pinv);
                out[(size_t)(2 * i + 1) * kM] = p31_mont(y1, p31_mont(w, h, p, pinv), p, pinv);
                if (i < R / 2 - 1) w = p31_mont(w, w1, p, pinv);
            }
        }
        return;
    }
#pragma unroll
    for (int m = 0; m < R; m++) {
        Acc s;
#pragma unroll
        for (int r0 = 0; r0 < R; r0 += 4)
            if (r0 == 0 || r0 < ni) {
#pragma unroll
                for (int r = r0; r < r0 + 4 && r < R; r++) {
                    s.add(x[r], c_fwd.v[k][m][r]);
                    if ((r & 1) || r == R - 1) s.fold(p);
                }
            }
        uint32_t y = s.reduce(p, pinv);
        if (m > 0) {
            y = p31_mont(y, w, p, pinv);
            if (m < R - 1) w = p31_mont(w, w1, p, pinv);
        }
        out[(size_t)m * kM] = y;
    }
}

// One CTA takes its 256 columns for all three primes, so that each limb is
// read once: that is what the host link needs when the operand is in pinned
// memory, and it is faster in device memory too (R = 16 2.90 -> 2.66 ms, R = 2
// 0.37 -> 0.30 ms against a CTA per prime).
template <int R>
__global__ void __launch_bounds__(256) p31_outer_fwd_kernel(const __grid_constant__ P31OuterArgs a)
{
    const uint32_t j = blockIdx.x * 256u + threadIdx.x;
    const uint32_t n = (uint32_t)a.n_limbs;
    const int ni = a.blocks;   // nonzero blocks of M limbs, at most R
    uint32_t x[R];
    chain_wait();
#pragma unroll
    for (int r = 0; r < R; r++) {
        const uint32_t i = j + r * kM;
        x[r] = r < ni && i < n ? __ldg(a.limbs + i) : 0u;
    }
#pragma unroll 1
    for (int k = 0; k < 3; k++) outer_fwd<R>(a, k, j, ni, x);
}

template <int R>
__global__ void __launch_bounds__(256) p31_outer_inv_kernel(const __grid_constant__ P31OuterArgs a)
{
    const int k = blockIdx.x % 3;
    const uint32_t p = p31_prime(k), pinv = p31_inv(k);
    const uint32_t j = (blockIdx.x / 3) * 256u + threadIdx.x;
    uint32_t *z = a.spec[k] + j;
    uint32_t t[R];
    const uint32_t w1 = g_pow(a.g[k], j, p, pinv);
    chain_wait();
#pragma unroll
    for (int m = 0; m < R; m++) t[m] = z[(size_t)m * kM];
    uint32_t w = w1;
    if (outer_paired(R, k)) {
        const uint32_t h = g_pow(a.gh[k], j, p, pinv);
#pragma unroll
        for (int i = 0; i < R / 2; i++) {
            const uint32_t y0 = i ? p31_mont(t[2 * i], w, p, pinv) : t[0];
            const uint32_t y1 = p31_mont(t[2 * i + 1], i ? p31_mont(w, h, p, pinv) : h, p, pinv);
            if (i > 0 && i < R / 2 - 1) w = p31_mont(w, w1, p, pinv);
            t[2 * i] = p31_add(y0, y1, p);
            t[2 * i + 1] = p31_sub(y0, y1, p);
        }
#pragma unroll
        for (int r = 0; r < R; r++) {
            Acc s;
#pragma unroll
            for (int i = 0; i < R / 2; i++) {
                s.add(t[2 * i + (r & 1)], c_inv[R][k][(r / 2) * kMaxR + (r & 1) * (kMaxR / 2) + i]);
                if ((i & 1) || i == R / 2 - 1) s.fold(p);
            }
            z[(size_t)r * kM] = s.reduce(p, pinv);
        }
        return;
    }
#pragma unroll
    for (int m = 1; m < R; m++) {
        t[m] = p31_mont(t[m], w, p, pinv);
        if (m < R - 1) w = p31_mont(w, w1, p, pinv);
    }
#pragma unroll
    for (int r = 0; r < R; r++) {
        Acc s;
#pragma unroll
        for (int m = 0; m < R; m++) {
            s.add(t[m], c_inv[R][k][r * kMaxR + m]);
            if ((m & 1) || m == R - 1) s.fold(p);
        }
        z[(size_t)r * kM] = s.reduce(p, pinv);
    }
}

template <int R>
cudaError_t launch_r(bool inverse, const P31OuterArgs &a, cudaStream_t st)
{
    if (inverse) return launch_chained(p31_outer_inv_kernel<R>, dim3(3 * (kM / 256)), 256, 0, st, a);
    return launch_chained(p31_outer_fwd_kernel<R>, dim3(kM / 256), 256, 0, st, a);
}

}  // namespace

cudaError_t launch_p31_outer(int R, bool inverse, const P31OuterArgs &a, cudaStream_t st)
{
    switch (R) {
    case 2: return launch_r<2>(inverse, a, st);
    case 4: return launch_r<4>(inverse, a, st);
    case 5: return launch_r<5>(inverse, a, st);
    case 6: return launch_r<6>(inverse, a, st);
    case 7: return launch_r<7>(inverse, a, st);
    case 8: return launch_r<8>(inverse, a, st);
    case 9: return launch_r<9>(inverse, a, st);
    case 10: return launch_r<10>(inverse, a, st);
    case 11: return launch_r<11>(inverse, a, st);
    case 12: return launch_r<12>(inverse, a, st);
    case 13: return launch_r<13>(inverse, a, st);
    case 14: return launch_r<14>(inverse, a, st);
    case 15: return launch_r<15>(inverse, a, st);
    case 16: return launch_r<16>(inverse, a, st);
    default: return cudaErrorInvalidValue;
    }
}

uint64_t p31_outer_root(int k) { return outer_g(k); }
uint64_t p31_outer_half(int k) { return k < 2 ? p31_pow(outer_g(k), outer_order(k) / 2, kP31[k]) : 1; }

// V^-1 for the n points c mod p: row r, column m is the X^r coefficient of
// the Lagrange polynomial prod_(i != m) (X - c_i) / (c_m - c_i).
static std::vector<uint64_t> vandermonde_inverse(const std::vector<uint64_t> &c, uint64_t p)
{
    const int n = (int)c.size();
    std::vector<uint64_t> all(n + 1, 0), v((size_t)n * n);
    all[0] = 1;   // prod (X - c_i), all[d] the X^d coefficient
    for (int m = 0; m < n; m++)
        for (int d = m + 1; d >= 0; d--) all[d] = ((d ? all[d - 1] : 0) + all[d] * (p - c[m])) % p;
    for (int m = 0; m < n; m++) {
        std::vector<uint64_t> q(n);   // divided by X - c_m
        uint64_t carry = 0, denom = 1;
        for (int d = n; d >= 1; d--) q[d - 1] = carry = (all[d] + carry * c[m]) % p;
        for (int i = 0; i < n; i++)
            if (i != m) denom = denom * ((c[m] + p - c[i]) % p) % p;
        const uint64_t inv = p31_pow(denom, p - 2, p);
        for (int r = 0; r < n; r++) v[(size_t)r * n + m] = q[r] * inv % p;
    }
    return v;
}

cudaError_t p31_outer_init()
{
    std::vector<uint32_t> h((size_t)(kMaxR + 1) * 3 * kMaxR * kMaxR, 0);
    for (int R = 2; R <= kMaxR; R++)
        for (int k = 0; k < 3 && R != 3; k++) {
            const uint64_t p = kP31[k], gamma = p31_pow(outer_g(k), kM, p);
            uint32_t *dst = h.data() + ((size_t)R * 3 + k) * kMaxR * kMaxR;
            auto mont = [&](uint64_t x) { return (uint32_t)((x << 32) % p); };
            const bool paired = outer_paired(R, k);
            const int n = paired ? R / 2 : R;
            std::vector<uint64_t> c(n);
            for (int m = 0; m < n; m++) c[m] = p31_pow(gamma, (uint64_t)m * (paired ? 2 : 1), p);
            const std::vector<uint64_t> v = vandermonde_inverse(c, p);
            for (int m = 0; m < n; m++) {
                const uint64_t odd = p31_pow(p31_pow(gamma, (uint64_t)m, p), p - 2, p);
                for (int r = 0; r < n; r++) {
                    const uint64_t x = v[(size_t)r * n + m], half = x * ((p + 1) / 2) % p;
                    dst[r * kMaxR + m] = mont(paired ? half : x);
                    if (paired)   // the differences are 2 gamma^m times the odd blocks' polynomial
                        dst[r * kMaxR + kMaxR / 2 + m] = mont(half * odd % p);
                }
            }
        }
    return cudaMemcpyToSymbol(c_inv, h.data(), h.size() * sizeof(uint32_t));
}

}  // namespace gbntt
