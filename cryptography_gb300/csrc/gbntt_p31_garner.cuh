// gbntt_p31_garner.cuh — Garner reconstruction for the 31-bit prime set.
#pragma once
#include "gbntt_p31.cuh"

namespace gbntt {

// c = a0 + p0 a1 + p0 p1 a2 < 2^93 from canonical residues; three 32-bit
// words ((0, 0, 0) gives 0).
__device__ __forceinline__ void garner31(uint32_t r0, uint32_t r1, uint32_t r2, uint32_t &w0, uint32_t &w1, uint32_t &w2)
{
    constexpr uint32_t p0 = kP31[0], p1 = kP31[1], p2 = kP31[2];
    constexpr uint64_t p01 = (uint64_t)p0 * p1;
    constexpr ShoupWord i01 = shoup_word(p31_pow(p0, p1 - 2, p1), p1);        // p0^-1 mod p1
    constexpr ShoupWord i012 = shoup_word(p31_pow(p01 % p2, p2 - 2, p2), p2); // (p0 p1)^-1 mod p2
    constexpr ShoupWord i12 = shoup_word(p31_pow(p1, p2 - 2, p2), p2);        // p1^-1 mod p2
    const uint32_t b1 = __viaddmin_u32(r0, 0u - p1, r0), b2 = __viaddmin_u32(r0, 0u - p2, r0);
    const uint32_t a1 = p31_shoup(r1 - b1 + p1, i01, p1);
    const uint32_t a2 = p31_sub(p31_shoup(r2 - b2 + p2, i012, p2), p31_shoup(a1, i12, p2), p2);
    const uint64_t x = (uint64_t)p0 * a1 + r0 + (uint64_t)(uint32_t)p01 * a2;   // < 2^62 + 2^63
    const uint64_t y = (x >> 32) + (uint64_t)(uint32_t)(p01 >> 32) * a2;
    w0 = (uint32_t)x;
    w1 = (uint32_t)y;
    w2 = (uint32_t)(y >> 32);
}

}  // namespace gbntt
