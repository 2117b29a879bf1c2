// cell.cuh -- the combing rule for 32-bit strands (src/lcs_residual_fixup.hpp:49-54):
// swap the strands h and v when the symbols match or when h > v.
#pragma once

#include "slcs_internal.cuh"

namespace slcs {

// Symbols as floats.  A symbol s of a or b becomes the float with bits
// 0x43000000 | s << 16 (128 + s up to 127, 2 s above: distinct symbols are at
// least 1 apart, and one byte permute makes it); masked rows and columns hold
// floats far from every symbol and from each other.
__device__ __forceinline__ uint32_t symbol_code(uint32_t word, int j)
{
    return __byte_perm(word, 0x43000000u, 0x7044u | (uint32_t(j) << 8));
}
constexpr uint32_t MASKED_ROW = 0xF149F2CAu;    // -1e30f
constexpr uint32_t MASKED_COLUMN = 0x7149F2CAu; // 1e30f

// The cell rule.  With far = fma.sat(d, -d, 1), d = a - b: far holds the bits
// of 1.0f (0x3F800000) when the symbols match and 0 otherwise, so that
//   h' = min(h + far, v)   (v on a match, min(h, v) otherwise)
//   v' = max(v - far, h)   (h on a match, max(h, v) otherwise)
// for 0 <= h, v < FAST_IDS: 4 instructions, two of them on the FMA pipe.  A
// comb is bound by instruction issue and the integer pipe, a lone warp by the
// chain through h and v.  In cycles per warp and cell (4 columns per step, 16
// rows per lane): compare, compare and two selects 6.76 with 4 warps on a
// sub-partition and 10.0 with one, this 4.61 and 5.45; v' = h + v - h' instead
// of the max (h' is then in v's chain) 4.58 and 7.92.
// Masked rows hold h = -1 and masked columns v = INT_MAX; neither ever
// matches, so neither swaps.  WIDE keeps the compare and selects for pairs
// whose ids reach FAST_IDS.
__device__ __forceinline__ int match_far(uint32_t a, uint32_t b)
{
    const float d = __uint_as_float(a) - __uint_as_float(b);
    return __float_as_int(__saturatef(__fmaf_rn(d, -d, 1.0f)));
}
__device__ __forceinline__ void pass(int far, int &h, int &v)
{
    const int nh = __viaddmin_s32(h, far, v);
    v = __viaddmax_s32(v, -far, h);
    h = nh;
}
template <bool WIDE>
__device__ __forceinline__ void cell(uint32_t a, uint32_t b, int &h, int &v)
{
    if constexpr (WIDE) {
        const bool swap = (a == b) | (h > v);
        const int nh = swap ? v : h;
        v = swap ? h : v;
        h = nh;
    } else {
        pass(match_far(a, b), h, v);
    }
}

// Two pairs (A, B) per register: every symbol, h and v register holds pair A
// in its low 16 bits and pair B in its high 16 bits, so one instruction works
// on two cells.  Strand ids are stored plus one (1..32767); a masked row holds
// h = 0 and symbol 0x1FF, a masked column v = 0x7FFF and symbol 0x100, so
// neither ever swaps.  The cell rule per half:
//   x = a ^ b                    0 on a match (both below 0x200)
//   far = fma.relu(x, -inf, 0)   on two 16-bit floats: 0 * -inf is NaN, which
//                                relu turns into 0x7FFF; a positive x gives
//                                -inf, which relu turns into 0
//   h' = min(h + far, v)         unsigned halves, one VIADDMNMX
//   v' = h + v - h'              as one 32-bit sum: the carries between the
//                                halves cancel
// On a match h + far is at least any v, so h' = v.  Seven integer instructions
// (a carry-safe difference, a byte permute expanding its sign to a mask, two
// bitwise selects) measured 5.50 cycles per warp and cell, these four 2.39
// (one sub-partition, 4 warps of 16 rows per lane).
constexpr uint32_t MASKED_ROW16 = 0x01FF01FFu, MASKED_COLUMN16 = 0x01000100u, MASKED_V16 = 0x7FFF7FFFu;
__device__ __forceinline__ uint32_t match16(uint32_t a, uint32_t b)
{
    uint32_t far;
    asm("{\n\t.reg .b32 ninf, zero;\n\tmov.b32 ninf, 0xFF80FF80;\n\tmov.b32 zero, 0;\n\t"
        "fma.rn.relu.bf16x2 %0, %1, ninf, zero;\n\t}"
        : "=r"(far)
        : "r"(a ^ b));
    return far;
}
__device__ __forceinline__ void pass16(uint32_t far, uint32_t &h, uint32_t &v)
{
    const uint32_t nh = __viaddmin_u16x2(h, far, v);
    v = h + v - nh;
    h = nh;
}
__device__ __forceinline__ void cell16(uint32_t a, uint32_t b, uint32_t &h, uint32_t &v)
{
    pass16(match16(a, b), h, v);
}

} // namespace slcs
