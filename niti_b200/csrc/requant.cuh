// NITI's int32 -> int8 requantisation and the counter-based random bits behind its
// stochastic rounding, as device functions shared by every kernel that narrows.
//
// Follows the reference's ti_torch.py: RangeEstimate :366-377 (bit-width from max|x|),
// act_calc/err_calc/grad_calc :103-147 (shift = bit-width - target), RoundShift :23-31,
// StoShift :33-46, PstoShift :48-69, int8_clip :71-72, with `//` truncating toward zero
// as in the torch release the reference was written for.
#pragma once
#include <cstdint>

namespace niti {

enum RoundMode : int { ROUND_NEAREST = 0, ROUND_STOCHASTIC = 1, ROUND_PSEUDO_STOCHASTIC = 2 };
enum CalcKind : int { CALC_ACT = 0, CALC_ERR = 1, CALC_GRAD = 2 };

// ---- Philox4x32-10 (Salmon et al., SC'11), keyed by (seed, stream), counter = element block.
__device__ __forceinline__ void philox4x32_10(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3,
                                              uint32_t k0, uint32_t k1, uint32_t (&out)[4]) {
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        uint32_t hi0 = __umulhi(0xD2511F53u, c0), lo0 = 0xD2511F53u * c0;
        uint32_t hi1 = __umulhi(0xCD9E8D57u, c2), lo1 = 0xCD9E8D57u * c2;
        uint32_t n0 = hi1 ^ c1 ^ k0, n2 = hi0 ^ c3 ^ k1;
        c0 = n0; c1 = lo1; c2 = n2; c3 = lo0;
        k0 += 0x9E3779B9u; k1 += 0xBB67AE85u;
    }
    out[0] = c0; out[1] = c1; out[2] = c2; out[3] = c3;
}
// Four words for elements 4*block .. 4*block+3 of `stream`.
__device__ __forceinline__ void random_block(uint64_t seed, uint32_t stream, uint64_t block, uint32_t (&out)[4]) {
    philox4x32_10(static_cast<uint32_t>(block), static_cast<uint32_t>(block >> 32), stream, 0u,
                  static_cast<uint32_t>(seed), static_cast<uint32_t>(seed >> 32), out);
}
__device__ __forceinline__ uint32_t random_word(uint64_t seed, uint32_t stream, uint64_t idx) {
    uint32_t w[4];
    random_block(seed, stream, idx >> 2, w);
    return w[idx & 3];
}

// ---- bit-width and shift selection
__host__ __device__ __forceinline__ int bitwidth_of_max(uint32_t m) {
    if (m == 0) return 0;
#ifdef __CUDA_ARCH__
    return 32 - __clz(static_cast<int>(m - 1));
#else
    int b = 0; uint32_t v = m - 1; while (v) { ++b; v >>= 1; } return b;
#endif
}
// shift (>= 0) applied to a tensor whose max|x| is `m`; `zero_out` is grad_calc's all-zero case.
__host__ __device__ __forceinline__ int shift_for(uint32_t m, int kind, int target_bits, bool* zero_out) {
    int b = bitwidth_of_max(m);
    *zero_out = (kind == CALC_GRAD) && (b == 0);
    int s = b - target_bits;
    return s > 0 ? s : 0;
}

__device__ __forceinline__ unsigned iabs_u(int x) { return static_cast<unsigned>(x < 0 ? -x : x); }
__device__ __forceinline__ unsigned absmax4(const int4 v) {
    return max(max(iabs_u(v.x), iabs_u(v.y)), max(iabs_u(v.z), iabs_u(v.w)));
}

__device__ __forceinline__ int clamp127(int v) { return max(-127, min(127, v)); }

// One element: shift == 0 wraps like `.type(torch.int8)`; shift > 0 rounds then clamps to +-127.
__device__ __forceinline__ int8_t narrow(int x, int shift, int mode, uint32_t rnd) {
    if (shift == 0) return static_cast<int8_t>(x);
    uint32_t a = static_cast<uint32_t>(x < 0 ? -x : x);
    uint32_t q = a >> shift;
    uint32_t lo = a & ((1u << shift) - 1u);
    uint32_t up;
    if (mode == ROUND_NEAREST) {
        up = lo >> (shift - 1);
    } else if (mode == ROUND_STOCHASTIC) {
        up = lo > (rnd & ((1u << shift) - 1u));
    } else {
        int h = shift >> 1;
        uint32_t qp = lo >> h;
        uint32_t pr = lo & ((1u << h) - 1u);
        if (shift & 1) pr <<= 1;
        up = qp > pr;
    }
    int v = static_cast<int>(q + up);
    return static_cast<int8_t>(clamp127(x < 0 ? -v : v));
}

// ---- four values at a time (shift > 0)
// Two int32 -> two saturated bytes in the low half of the result, `upper` moved into the high half
// (cvt.pack: d = upper << 16 | sat(hi) << 8 | sat(lo)).
__device__ __forceinline__ uint32_t pack2_sat_s8(int hi, int lo, uint32_t upper) {
    uint32_t d;
    asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(hi), "r"(lo), "r"(upper));
    return d;
}
__device__ __forceinline__ uint32_t pack2_sat_u8(int hi, int lo, uint32_t upper) {
    uint32_t d;
    asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(hi), "r"(lo), "r"(upper));
    return d;
}
// Round half away from zero is (x + half + (x >> 31)) >> shift with an arithmetic shift (for x < 0 that is
// -((|x| + half) >> shift)); the saturating pack clamps to a byte and one packed min / max finishes the clamp to
// +-127 (ReLU: the unsigned pack turns negatives into 0).  About 3 instructions per value.
template <bool RELU>
__device__ __forceinline__ uint32_t narrow4_nearest(const uint32_t* v, int shift, int half) {
    int y[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int x = static_cast<int>(v[j]);
        y[j] = RELU ? (x + half) >> shift : (x + half + (x >> 31)) >> shift;
    }
    if (RELU) return __vminu4(pack2_sat_u8(y[1], y[0], pack2_sat_u8(y[3], y[2], 0u)), 0x7F7F7F7Fu);
    return __vmaxs4(pack2_sat_s8(y[1], y[0], pack2_sat_s8(y[3], y[2], 0u)), 0x81818181u);
}
// Stochastic rounding: with lo the dropped bits of |x| and r the random word's, |x| is rounded up exactly
// when lo > r, i.e. when lo + (mask - r) carries into bit `shift`: y = (|x| + (~r & mask)) >> shift.  For x < 0 the
// negated quotient is the arithmetic shift (x + (r & mask)) >> shift (-floor(a / d) = floor((d - 1 - a) / d)), so both
// signs are one add and one shift behind a three-input logic operation.  For shifts below 24 and x <= 2^31 - 2^shift, as
// for the nearest form: negative sums only move towards zero, positive ones must not pass 2^31.  Under a ReLU the sign is left
// out: a negative value with any of these bits added stays below 2^shift and comes out as zero or less either way.
template <bool RELU>
__device__ __forceinline__ uint32_t narrow4_stochastic(const uint32_t* v, int shift, uint32_t mask, const uint32_t (&rnd)[4]) {
    int y[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int x = static_cast<int>(v[j]);
        y[j] = (x + static_cast<int>((RELU ? ~rnd[j] : rnd[j] ^ ~static_cast<uint32_t>(x >> 31)) & mask)) >> shift;
    }
    if (RELU) return __vminu4(pack2_sat_u8(y[1], y[0], pack2_sat_u8(y[3], y[2], 0u)), 0x7F7F7F7Fu);
    return __vmaxs4(pack2_sat_s8(y[1], y[0], pack2_sat_s8(y[3], y[2], 0u)), 0x81818181u);
}
// Pseudo-stochastic rounding (the upper half of the dropped bits against their lower half), clamped to 127 in magnitude.
__device__ __forceinline__ int narrow_pseudo(int x, int shift) {
    const uint32_t a = static_cast<uint32_t>(x < 0 ? -x : x);
    const int h = shift >> 1;
    const uint32_t lo = a & ((1u << shift) - 1u);
    const uint32_t up = (lo >> h) > ((lo & ((1u << h) - 1u)) << (shift & 1)) ? 1u : 0u;
    const int v = static_cast<int>(min((a >> shift) + up, 127u));
    return x < 0 ? -v : v;
}

// Four weights less their narrowed gradients.  Pseudo-stochastic rounding, the gradients' own mode, has a short form.
__device__ __forceinline__ uint32_t update_word(const int4 gv, const uint32_t wv, const uint32_t (&rnd)[4], int shift, int mode,
                                                bool zero_out) {
    const int gx[4] = {gv.x, gv.y, gv.z, gv.w};
    int y[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int g8 = zero_out ? 0 : mode == ROUND_PSEUDO_STOCHASTIC && shift > 0 ? narrow_pseudo(gx[j], shift) : narrow(gx[j], shift, mode, rnd[j]);
        y[j] = static_cast<int8_t>(wv >> (8 * j)) - g8;
    }
    return __vmaxs4(pack2_sat_s8(y[1], y[0], pack2_sat_s8(y[3], y[2], 0u)), 0x81818181u);
}

}  // namespace niti
