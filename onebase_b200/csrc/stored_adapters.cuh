// Adapters stored in a low-precision format -> bf16 operand tiles in shared memory, shared by the kernels that multiply them
// on the tensor cores.
#pragma once
#include "ob_common.cuh"
#include "ob_ptx.cuh"

namespace ob {

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    __nv_bfloat162 b = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&b);
}

__device__ __forceinline__ float stored_e4m3_value(uint32_t code) {
    uint32_t h2;
    asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h2) : "h"((uint16_t)code));
    return __half2float(__ushort_as_half((unsigned short)(h2 & 0xFFFFu)));
}
__device__ __forceinline__ float2 stored_e4m3x2_values(uint32_t two_codes) {
    uint32_t h2;
    asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h2) : "h"((uint16_t)two_codes));
    return __half22float2(*reinterpret_cast<__half2*>(&h2));
}

// Four e2m1 codes (the nibbles of the low 16 bits of w4) -> four bf16 values of bf16(value * block scale * global), through
// byte tables of the block's eight magnitudes: two byte permutes pick the low and the high bytes of the four results,
// two more interleave them, the codes' sign bits are ORed in.
__device__ __forceinline__ void e2m1x4_lookup(uint32_t w4, const uint32_t (&lo)[2], const uint32_t (&hi)[2], uint32_t& out01, uint32_t& out23) {
    const uint32_t sel = w4 & 0x7777u;
    const uint32_t L = __byte_perm(lo[0], lo[1], sel), H = __byte_perm(hi[0], hi[1], sel);
    out01 = __byte_perm(L, H, 0x5140u) | ((w4 & 0x8u) << 12) | ((w4 & 0x80u) << 24);
    out23 = __byte_perm(L, H, 0x7362u) | ((w4 & 0x800u) << 4) | ((w4 & 0x8000u) << 16);
}

// 16 e4m3 codes -> 16 bf16 values bf16(code * sc), one rounding (none with sc = 1: every e4m3 value is a bf16 value).
__device__ __forceinline__ void e4m3x16_to_bf16(const uint4& c, float sc, uint32_t (&o)[8]) {
    const uint32_t w[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float2 a = stored_e4m3x2_values(w[q] & 0xFFFFu), b = stored_e4m3x2_values(w[q] >> 16);
        o[2 * q] = pack_bf16x2(a.x * sc, a.y * sc);
        o[2 * q + 1] = pack_bf16x2(b.x * sc, b.y * sc);
    }
}

// A block of 16 e2m1 codes (x: codes 0..7, y: 8..15) and its ue4m3 scale byte -> 16 bf16 values bf16((value * block scale) *
// sc): the reference's order of the two products, one fp32 rounding (none with sc = 1: at most six significant bits).
__device__ __forceinline__ void e2m1x16_to_bf16(uint32_t x, uint32_t y, uint32_t scale_byte, float sc, uint32_t (&o)[8]) {
    const float sf = stored_e4m3_value(scale_byte);
    const uint32_t m01 = pack_bf16x2(0.0f, (0.5f * sf) * sc), m23 = pack_bf16x2((1.0f * sf) * sc, (1.5f * sf) * sc);
    const uint32_t m45 = pack_bf16x2((2.0f * sf) * sc, (3.0f * sf) * sc), m67 = pack_bf16x2((4.0f * sf) * sc, (6.0f * sf) * sc);
    const uint32_t lo[2] = {__byte_perm(m01, m23, 0x6420u), __byte_perm(m45, m67, 0x6420u)};
    const uint32_t hi[2] = {__byte_perm(m01, m23, 0x7531u), __byte_perm(m45, m67, 0x7531u)};
    e2m1x4_lookup(x, lo, hi, o[0], o[1]);   // element 2q in the low nibble of byte q: nibble order = element order
    e2m1x4_lookup(x >> 16, lo, hi, o[2], o[3]);
    e2m1x4_lookup(y, lo, hi, o[4], o[5]);
    e2m1x4_lookup(y >> 16, lo, hi, o[6], o[7]);
}

}  // namespace ob
