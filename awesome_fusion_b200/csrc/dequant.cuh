// In-register unpack of packed int8 / int4 weights to exact bf16 pairs.
//
// The reference kernel splices each byte into the mantissa of 2^23 and subtracts
// 2^23 + 128 in fp32 (bf16gemm_kernel_gfx90a.s:18-27, constants :204-210).  Here the splice costs nothing: a bf16 whose upper
// byte is zero is its lower byte times 2^-133 (denormals, and up to 255 the binade above them, have the same step), so an
// unsigned weight u merely zero-extended to 16 bits already IS the bf16 u * 2^-133, and ONE packed fused multiply-add,
//     fma(u * 2^-133, 2^127, -(128 + zero) * 2^-6)  =  (u - 128 - zero) * 2^-6,
// makes two exact weights of it (both operands and the result have at most 8 significant bits).  An int4 weight in the upper
// half of a byte is 16 u * 2^-133 and takes 2^123.  Zero-points and the storage encoding live in the constants.
// Every routine returns the weights times kUnpackFactor = 2^-6; the kernels multiply the finished fp32 sums by 64, and only then by a
// channel's scale (64 * scale overflows from 2^122 on).  Powers of two: no bit of a result depends on it while the products of weight
// and activation stay in the normal range of fp32 with the factor, that is above 2^-120 (with folded group scales 2^-116).  Group scales
// below 2^-100 are not folded; their weights q * scale * 2^-10 lose bits once q * scale is below 2^-116.  Cost per 4 int8 weights: 1 xor + 2 permutes + 2 fma (splice, sign and add: 8 in natural
// order, 7 strided); per 8 int4 weights 10 in natural order, 9 strided (13, 11).  The unpack is what the decode kernels and the
// converter warps of the prefill kernels issue most; see the figures there.
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>
#include "afb_capi.h"

namespace afb {

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}
// (a & b) ^ c
__device__ __forceinline__ uint32_t lop3_and_xor(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, 0x6A;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ uint32_t bf16x2_mul(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}

__device__ __forceinline__ uint32_t bf16x2_fma(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}

// What the unpack adds and multiplies.  kUnpackFactor * 64 = 1.
constexpr float kUnpackInverse = 64.f;
__device__ __forceinline__ float unscaled(float sum, float scale) { return (sum * kUnpackInverse) * scale; }
constexpr uint32_t kMulByte = 0x7F007F00u;       // 2^127 in both halves: weights in the low bits of their byte
constexpr uint32_t kMulHighNibble = 0x7D007D00u; // 2^123: weights in bits [4,8) of their byte
constexpr uint32_t kMulNibblePair = 0x7D007F00u; // low half from bits [0,4), high half from bits [4,8)

// Stored integers to unsigned ones (value + 128 / value + 8): one xor per word, nothing to flip when they are stored that way.
__host__ __device__ __forceinline__ uint32_t flip8(uint32_t enc) { return enc == AFB_ENC_OFFSET_BINARY ? 0u : 0x80808080u; }
__host__ __device__ __forceinline__ uint32_t flip4(uint32_t enc) { return enc == AFB_ENC_OFFSET_BINARY ? 0u : 0x88888888u; }

__device__ __forceinline__ uint32_t bf16_dup(uint16_t s) { return (uint32_t)s * 0x00010001u; }
__device__ __forceinline__ uint32_t bf16_dup_rn(float v) { return bf16_dup(__bfloat16_as_ushort(__float2bfloat16_rn(v))); }

// The addend for a zero-point byte in the weights' own encoding (without zero-points: the byte that decodes to 0).
__device__ __forceinline__ int decode_zero8(uint32_t zbyte, uint32_t enc) { return enc == AFB_ENC_OFFSET_BINARY ? (int)zbyte - 128 : (int)(int8_t)zbyte; }
__device__ __forceinline__ int decode_zero4(uint32_t zbyte, uint32_t enc) {
    const int nib = (int)(zbyte & 0xFu);
    return enc == AFB_ENC_OFFSET_BINARY ? nib - 8 : ((nib ^ 8) - 8);
}
__device__ __forceinline__ uint32_t unpack_add(int bits, int zero) { return bf16_dup_rn((float)(-(bits == 8 ? 128 : 8) - zero) * 0.015625f); }

// Two of the four bytes of `t` (flipped to unsigned) as bf16 pairs; the selectors say which: {k0,k1},{k2,k3} of a plain word, or
// {b0,b2},{b1,b3}: the pre-packed order [k0,k2,k1,k3] read as consecutive k, or a plain word in strided pairs.
constexpr uint32_t kSel8Natural01 = 0x4140u, kSel8Natural23 = 0x4342u, kSel8Strided02 = 0x4240u, kSel8Strided13 = 0x4341u;
__device__ __forceinline__ void s8x4_to_bf16(uint32_t w, uint32_t flip, uint32_t sel0, uint32_t sel1, uint32_t mul, uint32_t add, uint32_t& p0, uint32_t& p1) {
    const uint32_t t = w ^ flip;
    p0 = bf16x2_fma(prmt(t, 0u, sel0), mul, add);
    p1 = bf16x2_fma(prmt(t, 0u, sel1), mul, add);
}

// Eight nibbles of w in strided pairs: {n0,n4},{n1,n5},{n2,n6},{n3,n7} (consecutive k of a pre-packed word).
__device__ __forceinline__ void s4x8_to_bf16_strided(uint32_t w, uint32_t flip, uint32_t add, uint32_t p[4]) {
    const uint32_t h = w >> 8;
    p[0] = bf16x2_fma(lop3_and_xor(w, 0x000f000fu, flip & 0x000f000fu), kMulByte, add);
    p[1] = bf16x2_fma(lop3_and_xor(w, 0x00f000f0u, flip & 0x00f000f0u), kMulHighNibble, add);
    p[2] = bf16x2_fma(lop3_and_xor(h, 0x000f000fu, flip & 0x000f000fu), kMulByte, add);
    p[3] = bf16x2_fma(lop3_and_xor(h, 0x00f000f0u, flip & 0x00f000f0u), kMulHighNibble, add);
}
// Eight nibbles of w in either order, chosen by the constants of Nibbles: even nibbles and odd nibbles are masked out of the word
// once each (odd ones stay in the upper half of their bytes) and a permute pairs the bytes; its sign-replicating selectors supply
// the zero bytes (an even nibble's byte never has its top bit set).
struct Nibbles { uint32_t sel[4], mul[2]; };
__device__ __forceinline__ Nibbles nibbles(bool packed) {
    Nibbles q;
    q.sel[0] = packed ? 0x8280u : 0x8480u;   // {n0,n4} / {n0,n1}
    q.sel[1] = packed ? 0x8684u : 0x9591u;   // {n1,n5} / {n2,n3}
    q.sel[2] = packed ? 0x8381u : 0xA6A2u;   // {n2,n6} / {n4,n5}
    q.sel[3] = packed ? 0x8785u : 0xB7B3u;   // {n3,n7} / {n6,n7}
    q.mul[0] = packed ? kMulByte : kMulNibblePair;         // of pairs 0 and 2
    q.mul[1] = packed ? kMulHighNibble : kMulNibblePair;   // of pairs 1 and 3
    return q;
}
__device__ __forceinline__ void s4x8_to_bf16(uint32_t w, uint32_t flip, const Nibbles& q, uint32_t mul0, uint32_t mul1, uint32_t add, uint32_t p[4]) {
    const uint32_t e = lop3_and_xor(w, 0x0f0f0f0fu, flip & 0x0f0f0f0fu), o = lop3_and_xor(w, 0xf0f0f0f0u, flip & 0xf0f0f0f0u);
    p[0] = bf16x2_fma(prmt(e, o, q.sel[0]), mul0, add);
    p[1] = bf16x2_fma(prmt(e, o, q.sel[1]), mul1, add);
    p[2] = bf16x2_fma(prmt(e, o, q.sel[2]), mul0, add);
    p[3] = bf16x2_fma(prmt(e, o, q.sel[3]), mul1, add);
}

// Group scales on weights that go to the tensor cores as bf16_rn(q * scale): the scale rides on the same multiply-add,
//     fma(u * 2^-133, scale * 2^123, -128 * scale * 2^-10)  =  bf16_rn((u - 128) * scale) * 2^-10,
// one rounding of the exact product, as a separate multiplication of the exact weight would round it.  Needs both constants to be
// exact: 2^-100 < scale < 16 (or 0) and no zero-point ((128 + zero) * scale can have 16 significant bits); negative scales stay out
// so that a zero weight keeps the sign that the product gives it.  Otherwise the weight
// is unpacked as above and multiplied by scale * 2^-4, with the same factor of 2^-10 in the result.
constexpr float kGroupInverse = 1024.f;
struct GroupUnpack {
    uint32_t mul0, mul1;   // multipliers of the unpack (int8 uses mul0)
    uint32_t add;
    uint32_t scale;        // scale * 2^-4 in both halves: second step when not folded, and the two-term mode
};
__device__ __forceinline__ bool group_folds(uint16_t s, bool has_zero) {
    const float f = __uint_as_float((uint32_t)s << 16);
    return !has_zero && ((f < 16.f && f > 7.9e-31f) || s == 0);
}
__device__ __forceinline__ GroupUnpack group_unpack(int bits, uint16_t s, int zero, bool folded, const Nibbles& q) {
    const float f = __uint_as_float((uint32_t)s << 16);
    GroupUnpack u;
    u.scale = bf16_dup_rn(f * 0.0625f);
    u.mul0 = bits == 8 ? kMulByte : q.mul[0];
    u.mul1 = bits == 8 ? kMulByte : q.mul[1];
    if (folded) {   // the multipliers above divided by 16, times the scale
        const uint32_t lo = __bfloat16_as_ushort(__float2bfloat16_rn(f * 0x1p123f)), hi = __bfloat16_as_ushort(__float2bfloat16_rn(f * 0x1p119f));
        u.mul0 = ((u.mul0 & 0xffffu) == 0x7F00u ? lo : hi) | ((u.mul0 >> 16) == 0x7F00u ? lo : hi) << 16;
        u.mul1 = ((u.mul1 & 0xffffu) == 0x7F00u ? lo : hi) | ((u.mul1 >> 16) == 0x7F00u ? lo : hi) << 16;
        u.add = bf16_dup_rn(f * (bits == 8 ? -0.125f : -0.0078125f));   // -128 * 2^-10, -8 * 2^-10
    } else {
        u.add = unpack_add(bits, zero);
    }
    return u;
}

// The folded constants of one group from those of all groups: a scale that folds is 0 or a positive normal number, so its products with
// powers of two are integer additions to the exponent fields (6 instructions instead of 30).
struct GroupFold { uint32_t mul0, mul1, add; };
__device__ __forceinline__ GroupFold group_fold(int bits, const Nibbles& q) {
    const uint32_t m0 = bits == 8 ? kMulByte : q.mul[0], m1 = bits == 8 ? kMulByte : q.mul[1];
    const uint32_t sixteenth = 0x3F803F80u + 0x02000200u;   // the multipliers divided by 16, less the exponent of 1
    return {m0 - sixteenth, m1 - sixteenth, 0x80008000u - (bits == 8 ? 0x01800180u : 0x03800380u)};   // -2^-3, -2^-7
}
__device__ __forceinline__ void group_folded(const GroupFold& f, uint16_t s, GroupUnpack& u) {
    const uint32_t two = bf16_dup(s);
    u.mul0 = s ? two + f.mul0 : 0u;
    u.mul1 = s ? two + f.mul1 : 0u;
    u.add = s ? two + f.add : 0x80008000u;
}

// Place of weight k inside its word in the pre-packed layout (int8: bytes [k0,k2,k1,k3]; int4: nibbles [k0,k2,k4,k6,k1,k3,k5,k7]).
__host__ __device__ __forceinline__ uint32_t packed_pos(uint32_t bits, uint32_t k) {
    if (bits == 8) { const uint32_t i = k & 3u; return (k & ~3u) | ((i >> 1) | ((i & 1u) << 1)); }
    const uint32_t i = k & 7u;
    return (k & ~7u) | ((i >> 1) | ((i & 1u) << 2));
}

}  // namespace afb
