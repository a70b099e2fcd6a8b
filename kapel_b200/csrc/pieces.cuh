// A 32-bit value as the sum of three bfloat16 pieces, x = x1 + x2 + x3: three times eight bits are the 24 of a float and bfloat16 has its
// exponents, so the pieces hold the value exactly (down to 2^-133: of values below 2^-110 they keep that much and no more. Products therefore cut
// their inputs times PIECE_SCALE, where every float has pieces that are not even subnormal; what that takes beyond the largest float comes
// out as no finite number, which those kernels compute again by multiply-adds). A second piece is at most 2^-8 of the value, a third 2^-17: of the nine
// products of two values' pieces the three that are left out are together at most 2^-24 of the whole, as much as the rounding of one 32-bit
// product, and mostly far less. Added up from the small ones to the large ones (`piece_a`, `piece_b`) a product of 32-bit values is as exact on the tensor
// cores as by multiply-adds, as long as the sums in the tensor cores are short: they add in 32 bits and round towards zero.
#pragma once
#include "common.cuh"

namespace kb {

constexpr int PIECE_PRODUCTS = 6;
constexpr float PIECE_SCALE = 16777216.f;                          // 2^24: the last bit of the smallest subnormal becomes 2^-125
__host__ __device__ constexpr int piece_a(int i) { return i == 0 ? 2 : i == 2 || i == 3 ? 1 : 0; }        // 2 0 1 1 0 0
__host__ __device__ constexpr int piece_b(int i) { return i == 1 ? 2 : i == 2 || i == 4 ? 1 : 0; }        // 0 2 1 0 1 0

#ifdef __CUDACC__
// Two neighbouring values cut: a word of each piece, `x` in its lower half. x and y come back as what the first two pieces leave, the third's value:
// NaN where a value is no finite number or rounds to infinity in bfloat16.
__device__ __forceinline__ void cut_pair(float& x, float& y, uint32_t& one, uint32_t& two, uint32_t& three) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(x, y);
    one = *reinterpret_cast<const uint32_t*>(&p);
    x -= __uint_as_float(one << 16), y -= __uint_as_float(one & 0xffff0000u);
    const __nv_bfloat162 q = __floats2bfloat162_rn(x, y);
    two = *reinterpret_cast<const uint32_t*>(&q);
    x -= __uint_as_float(two << 16), y -= __uint_as_float(two & 0xffff0000u);
    const __nv_bfloat162 r = __floats2bfloat162_rn(x, y);
    three = *reinterpret_cast<const uint32_t*>(&r);
}
#endif

}  // namespace kb
