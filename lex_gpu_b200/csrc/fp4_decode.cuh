// Bit-exact NVFP4 decode for sm_100a: E2M1 code x E4M3 group scale x f32 row scale -> f16.
//
// The value every kernel in this library multiplies by is the one lex's reference
// interpreter stages (crates/lex-front/src/interp.rs:643-657, then :500-507):
//
//     w32 = fl32( fl32( e2m1(code) * e4m3(scale) ) * wg[row] )     left to right
//     w16 = round_to_nearest_even_f16( w32 )
//
// The first product is exact (at most 6 significant bits), so only the multiply by
// the row scale and the conversion round.  The reference's own GPU kernels fold the
// group scale into the row scale first (crates/lex-msl/src/gemm.rs:254-255,
// crates/lex-msl/src/dialect.rs:768-791), which rounds differently in about one
// weight in 10^5 and turns the NaN scale bytes into +-480; this file follows the
// interpreter instead.
//
// Two methods, the same bits.
//
// Products (the usual one).  Up to its sign and a power of two, a weight is A = f16(fl32(s * wg)) (magnitudes 0.5, 1, 2, 4)
// or B = f16(fl32(1.5 s * wg)) (1.5, 3, 6): scaling by a power of two commutes with both roundings while nothing is
// subnormal or overflows.  B is not f16(1.5 A), but it lies at most 1.5 units in the last place of A (call it u) from
// 1.5 A, so one f16 fused multiply-add gives every weight of the group:
//     w = fma(e, A - u, e * (u + d))     e = the code's value, d = 0 if B == 1.5 A, else 3/8 u with the sign of B - 1.5 A
// (e = 0.5, 1, 2, 4: e A + e d rounds to e A, because |e d| is less than half a unit of e A; e = 1.5, 3, 6: e A is within
// 1.5 units of B and e d decides between its two neighbours the right way; the u taken off and put back keeps the
// addend's sign that of the code, so that code 8 gives -0.)  e * (u + d) is exact in f16 for A >= 2^-10.  Checked against
// the table method for every mantissa of wg, all scale bytes and codes, once; tests/test_fp4_products.py restates it for a
// spread of mantissas and those beside a tie.  Per weight: half a conversion of two codes
// (`cvt.rn.f16x2.e2m1x2`, integer pipe) and one FP16 multiply and one fused multiply-add per two weights (the FP16
// pipe, idle otherwise), 2.4 instructions in all with the factors, where the table takes 5.7, most of them in the integer
// pipe.  Measured, 16 warps that store what they decode to shared memory: 33 weights per clock and SM with the choice
// between the methods in place (49, what the stores allow, without it) against 21.5 by the table.
//
// Table (when a scale or row scale is outside the range of the products: see RowScale).  A group of 16 weights
// shares its scale, so it has only 8 distinct magnitudes.  They are computed once per group (16 f32 multiplies, 4 packed
// f32->f16x2 conversions) and kept as a register table split into a low-byte plane
// and a high-byte plane; each weight is then one byte-permute lookup per plane,
// selected by its 3 magnitude bits, and the sign bit of the code is XORed in.
#pragma once
#include <cuda_fp16.h>
#include <stdint.h>

namespace lexb {

// Two OCP e4m3fn bytes -> two f32, exact for all 256 byte values: the hardware conversion to f16 is
// exact (every E4M3 value, subnormals included, is an f16 value) and maps the two NaN bytes
// (exponent 15, mantissa 7; interp.rs:41-42) to NaN; f16 -> f32 is exact as well.
__device__ __forceinline__ float2 e4m3x2_to_f32(uint32_t two_bytes) {
    uint32_t h2;
    asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h2) : "h"(static_cast<unsigned short>(two_bytes)));
    return __half22float2(*reinterpret_cast<const __half2*>(&h2));
}
__device__ __forceinline__ float e4m3_to_f32(uint32_t b) { return e4m3x2_to_f32(b & 0xFFu).x; }

__device__ __forceinline__ uint32_t pack_f16x2_rn(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
    return r;
}

// The 8 magnitudes of one group as f16, split into byte planes:
// lo.x/lo.y hold the low bytes of entries 0-3 / 4-7, hi.x/hi.y the high bytes.
struct GroupTable {
    uint32_t lo0, lo1, hi0, hi1;
};

__device__ __forceinline__ GroupTable make_group_table_f32(float s, float wg) {
    // (e2m1 * s) is exact; __fmul_rn keeps the compiler from reassociating or contracting.
    const float p0 = __fmul_rn(__fmul_rn(0.0f, s), wg);
    const float p1 = __fmul_rn(__fmul_rn(0.5f, s), wg);
    const float p2 = __fmul_rn(s, wg);
    const float p3 = __fmul_rn(__fmul_rn(1.5f, s), wg);
    const float p4 = __fmul_rn(__fmul_rn(2.0f, s), wg);
    const float p5 = __fmul_rn(__fmul_rn(3.0f, s), wg);
    const float p6 = __fmul_rn(__fmul_rn(4.0f, s), wg);
    const float p7 = __fmul_rn(__fmul_rn(6.0f, s), wg);
    const uint32_t h01 = pack_f16x2_rn(p0, p1);
    const uint32_t h23 = pack_f16x2_rn(p2, p3);
    const uint32_t h45 = pack_f16x2_rn(p4, p5);
    const uint32_t h67 = pack_f16x2_rn(p6, p7);
    GroupTable t;
    t.lo0 = prmt(h01, h23, 0x6420u);
    t.lo1 = prmt(h45, h67, 0x6420u);
    t.hi0 = prmt(h01, h23, 0x7531u);
    t.hi1 = prmt(h45, h67, 0x7531u);
    return t;
}

__device__ __forceinline__ GroupTable make_group_table(uint32_t scale_byte, float wg) {
    return make_group_table_f32(e4m3_to_f32(scale_byte), wg);
}

// d = a ^ (b & c) in one logic instruction
__device__ __forceinline__ uint32_t xor_and(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0x78;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
}

// Eight codes (one 32-bit word of wq: code j in bits 4j..4j+3, i.e. column order) ->
// eight f16 in column order, packed as four f16x2 words.
// The decode is bound by the integer pipe (64 lanes a clock against the FP32 pipe's 128), so the two shifts are
// written as multiplies, which the FP32 pipe's integer multiply-add takes, and each sign is folded into its
// lookup with one three-input logic instruction.
__device__ __forceinline__ void decode8(const GroupTable& t, uint32_t w, uint32_t& o0, uint32_t& o1,
                                        uint32_t& o2, uint32_t& o3) {
    const uint32_t mag = w & 0x77777777u;     // selector nibbles: bit 3 must be clear for prmt
    const uint32_t mag_hi = __umulhi(mag, 0x10000u);      // mag >> 16
    const uint32_t w4 = w * 16u;                          // w << 4
    // sign bytes: prmt's replicate-msb mode (selector bit 3) turns the sign bit of a code
    // into 0x00 / 0xff.  Codes 0..3 live in bytes 0,1 of w (odd codes: bit 7 of the byte)
    // and of w4 (even codes: bit 3 of w's byte moved up to bit 7).
    const uint32_t sgn_a = prmt(w4, w, 0xD9C8u);          // codes 0,1,2,3
    const uint32_t sgn_b = prmt(w4, w, 0xFBEAu);          // codes 4,5,6,7
    const uint32_t lo_a = prmt(t.lo0, t.lo1, mag);
    const uint32_t hi_a = xor_and(prmt(t.hi0, t.hi1, mag), sgn_a, 0x80808080u);
    const uint32_t lo_b = prmt(t.lo0, t.lo1, mag_hi);
    const uint32_t hi_b = xor_and(prmt(t.hi0, t.hi1, mag_hi), sgn_b, 0x80808080u);
    o0 = prmt(lo_a, hi_a, 0x5140u);
    o1 = prmt(lo_a, hi_a, 0x7362u);
    o2 = prmt(lo_b, hi_b, 0x5140u);
    o3 = prmt(lo_b, hi_b, 0x7362u);
}

__device__ __forceinline__ uint32_t h_mul2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t h_fma2(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ uint32_t h_clamp2(uint32_t v, uint32_t limit) {      // to [-limit, limit], limit >= 0
    uint32_t d;
    asm("{\n\t.reg .b32 t;\n\tmin.f16x2 t, %1, %2;\n\tmax.f16x2 %0, t, %3;\n\t}" : "=r"(d) : "r"(v), "r"(limit), "r"(limit ^ 0x80008000u));
    return d;
}

// A row's scale with what the product method needs: `up` = wg * 2^120 (a scale byte shifted to bit 20 is, as f32, its
// value times 2^-120), and the scale bytes it may be used with - those with 2^-10 <= s * wg < 2^12, and 0 - as two
// addends that carry a byte outside [lowest, highest] into its top bit (four bytes at a time).
struct RowScale {
    float wg, up;
    uint32_t below, above;
};
__device__ __forceinline__ RowScale make_row_scale(float wg) {
    RowScale r;
    r.wg = wg;
    r.up = __fmul_rn(wg, __uint_as_float((127u + 120u) << 23));
    r.below = 0x7F7F7F7Fu;                                       // +0: every scale but the NaN bytes
    r.above = 0x01010101u;
    const uint32_t bits = __float_as_uint(wg);
    if (bits != 0u) {
        const int e = static_cast<int>(bits >> 23) - 127;       // (a set sign bit puts it out of range)
        const int e_lo = -10 - e, e_hi = 11 - e;                 // exponents of s that keep s * wg in range
        if (e_lo > 8 || e_hi < -6 || e > 6) {                    // (past e = 6 `up` overflows)
            r.above = 0x80808080u;                               // no byte: the table
        } else {
            const uint32_t lowest = e_lo >= -6 ? static_cast<uint32_t>(e_lo + 7) << 3 : (e_lo >= -9 ? 1u << (e_lo + 9) : 1u);
            const uint32_t highest = e_hi >= 8 ? 0x7Eu : (static_cast<uint32_t>(e_hi + 7) << 3) | 7u;
            r.below = (0x80u - lowest) * 0x01010101u;
            r.above = (0x7Fu - highest) * 0x01010101u;
        }
    }
    return r;
}
// four scale bytes of rows whose addends are `below` / `above`: can all four groups take the products?
__device__ __forceinline__ bool products_ok(uint32_t scales, uint32_t below, uint32_t above) {
    const uint32_t nonzero = scales + 0x7F7F7F7Fu, not_low = scales + below, high = scales + above;
    return ((((nonzero & ~not_low) | high) | scales) & 0x80808080u) == 0u;
}

// The factors of two groups of one row, one in each half: base = A - u, extra = u + d.  Each scale byte comes at bits
// 20-26 of its word; the other bits are ignored.
struct GroupFactors {
    uint32_t base, extra;
};
__device__ __forceinline__ GroupFactors group_factors(uint32_t s0_at_20, uint32_t s1_at_20, float up) {
    const float x0 = __uint_as_float(s0_at_20 & 0x07F00000u), x1 = __uint_as_float(s1_at_20 & 0x07F00000u);
    const uint32_t A = pack_f16x2_rn(__fmul_rn(x0, up), __fmul_rn(x1, up));
    const uint32_t B = pack_f16x2_rn(__fmul_rn(__fmul_rn(x0, 1.5f), up), __fmul_rn(__fmul_rn(x1, 1.5f), up));
    const uint32_t diff = h_fma2(A, 0xBE00BE00u, B);             // B - 1.5 A: 0 or at least u / 2 in magnitude
    const uint32_t pow2 = A & 0x7C007C00u;                       // u * 2^10
    const uint32_t d = h_clamp2(diff, h_mul2(pow2, 0x0E000E00u));        // 3/8 * 2^-10
    GroupFactors f;
    f.base = h_fma2(pow2, 0x94009400u, A);
    f.extra = h_fma2(pow2, 0x14001400u, d);
    return f;
}
// eight codes of one group (its factors in both halves) -> eight f16 in column order
__device__ __forceinline__ void multiply8(uint32_t w, uint32_t base, uint32_t extra, uint32_t& o0, uint32_t& o1, uint32_t& o2, uint32_t& o3) {
    uint32_t e0, e1, e2, e3;
    asm("{\n\t.reg .b8 a, b, c, d;\n\tmov.b32 {a, b, c, d}, %4;\n\t"
        "cvt.rn.f16x2.e2m1x2 %0, a;\n\tcvt.rn.f16x2.e2m1x2 %1, b;\n\tcvt.rn.f16x2.e2m1x2 %2, c;\n\tcvt.rn.f16x2.e2m1x2 %3, d;\n\t}"
        : "=r"(e0), "=r"(e1), "=r"(e2), "=r"(e3)
        : "r"(w));
    o0 = h_fma2(e0, base, h_mul2(e0, extra));
    o1 = h_fma2(e1, base, h_mul2(e1, extra));
    o2 = h_fma2(e2, base, h_mul2(e2, extra));
    o3 = h_fma2(e3, base, h_mul2(e3, extra));
}
// (written as moves of halves, which the multiplies' operand selection can take in; a byte permute is an instruction of its own)
__device__ __forceinline__ uint32_t low_half_twice(uint32_t v) {
    uint32_t d;
    asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %1;\n\tmov.b32 %0, {l, l};\n\t}" : "=r"(d) : "r"(v));
    return d;
}
__device__ __forceinline__ uint32_t high_half_twice(uint32_t v) {
    uint32_t d;
    asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %1;\n\tmov.b32 %0, {h, h};\n\t}" : "=r"(d) : "r"(v));
    return d;
}

// One group of 16 weights by the table: q = its 8 packed bytes (q.x = columns 0-7, q.y = columns 8-15).
__device__ __forceinline__ void table_group16(uint2 q, uint32_t scale_byte, float wg, uint4& out_lo, uint4& out_hi) {
    const GroupTable t = make_group_table(scale_byte, wg);
    decode8(t, q.x, out_lo.x, out_lo.y, out_lo.z, out_lo.w);
    decode8(t, q.y, out_hi.x, out_hi.y, out_hi.z, out_hi.w);
}
__device__ __forceinline__ void multiply_group16(uint2 q, uint32_t base, uint32_t extra, uint4& out_lo, uint4& out_hi) {
    multiply8(q.x, base, extra, out_lo.x, out_lo.y, out_lo.z, out_lo.w);
    multiply8(q.y, base, extra, out_hi.x, out_hi.y, out_hi.z, out_hi.w);
}
// One group on its own.
__device__ __forceinline__ void decode_group16(uint2 q, uint32_t scale_byte, const RowScale& row, uint4& out_lo, uint4& out_hi) {
    if (products_ok(scale_byte, row.below, row.above)) {
        const GroupFactors f = group_factors(scale_byte << 20, scale_byte << 20, row.up);
        multiply_group16(q, f.base, f.extra, out_lo, out_hi);
    } else {
        table_group16(q, scale_byte, row.wg, out_lo, out_hi);
    }
}
// Two / four consecutive groups of one row (32 / 64 columns), their scale bytes in `sc` from the low byte up.  Whole warp:
// the method is chosen for all lanes together.
__device__ __forceinline__ void decode_row32(const uint4& q, uint32_t sc, const RowScale& row, uint4 (&o)[4]) {
    sc &= 0xFFFFu;
    if (__all_sync(0xFFFFFFFFu, products_ok(sc, row.below, row.above))) {
        const GroupFactors f = group_factors(sc << 20, sc << 12, row.up);
        multiply_group16(make_uint2(q.x, q.y), low_half_twice(f.base), low_half_twice(f.extra), o[0], o[1]);
        multiply_group16(make_uint2(q.z, q.w), high_half_twice(f.base), high_half_twice(f.extra), o[2], o[3]);
    } else {
        table_group16(make_uint2(q.x, q.y), sc & 0xFFu, row.wg, o[0], o[1]);
        table_group16(make_uint2(q.z, q.w), sc >> 8, row.wg, o[2], o[3]);
    }
}
__device__ __forceinline__ void decode_row64(const uint4& q0, const uint4& q1, uint32_t sc, const RowScale& row, uint4 (&o)[8]) {
    if (__all_sync(0xFFFFFFFFu, products_ok(sc, row.below, row.above))) {
        const GroupFactors f = group_factors(sc << 20, sc << 12, row.up), g = group_factors(sc << 4, sc >> 4, row.up);
        multiply_group16(make_uint2(q0.x, q0.y), low_half_twice(f.base), low_half_twice(f.extra), o[0], o[1]);
        multiply_group16(make_uint2(q0.z, q0.w), high_half_twice(f.base), high_half_twice(f.extra), o[2], o[3]);
        multiply_group16(make_uint2(q1.x, q1.y), low_half_twice(g.base), low_half_twice(g.extra), o[4], o[5]);
        multiply_group16(make_uint2(q1.z, q1.w), high_half_twice(g.base), high_half_twice(g.extra), o[6], o[7]);
    } else {
        table_group16(make_uint2(q0.x, q0.y), sc & 0xFFu, row.wg, o[0], o[1]);
        table_group16(make_uint2(q0.z, q0.w), (sc >> 8) & 0xFFu, row.wg, o[2], o[3]);
        table_group16(make_uint2(q1.x, q1.y), (sc >> 16) & 0xFFu, row.wg, o[4], o[5]);
        table_group16(make_uint2(q1.z, q1.w), sc >> 24, row.wg, o[6], o[7]);
    }
}

}  // namespace lexb
