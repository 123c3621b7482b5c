// Expansion of W6A8 codes to int8, shared by the decode kernel (weight_pack.cu) and the fused GEMM (gemm_w6.inl).
// Storage (the reference's, csrc/h3.cu:8-37, csrc/vendor/w6a8_requant.cu:128-151): per weight row K/2 bytes of low nibbles
// (element e in byte e/2, even e in the low nibble), then K/4 bytes holding the top two bits of four consecutive
// elements; one fp8-e4m3 scale per 32 columns; the int8 value is clamp(rint((code - 32) * scale), +-127).
#pragma once

#include <cuda_fp8.h>

#include "common.cuh"

// One scale group: 32 codes (16 bytes of nibbles l, top bits ha for elements 0-15 and hb for 16-31, scale byte sb) ->
// 32 int8 in element order (o[0..7]).
// A word of nibbles holds 8 elements, the even ones in the low nibbles; its 16 top bits hold one 2-bit field per
// element. Masked with 0x3333 they are, as they stand, a byte-permute selector (one index 0..3 per nibble) for the
// even elements, and shifted right by two for the odd ones, so one permute of a 4-byte table turns four fields into
// the four high nibbles. With a scale of exactly 1 the table holds the high nibble of code - 32 as a signed byte
// (E, F, 0, 1) and the result is final; otherwise it holds code bits 5:4 and the bytes go through half-precision
// arithmetic two at a time: 1024 + code by setting exponent bits, one fused multiply-add with -1056 * s (exact while
// that constant is finite), clamp where 32 * |s| can pass 127, rint by adding 1536, low bytes gathered by a permute.
// The forms are chosen per warp, not per lane: lanes hold different rows with different scales, and a branch that splits the
// warp costs the sum of its sides. What a packer emits lies in (0, 4]: its largest group has 31 steps for 127, so a scale of
// 4.0 is common and only the unused code 0 can leave the range there, downwards, by one. That form clamps once, after the rint
// (12 operations for four pairs where the general form has 20), and a caller with several groups votes once for all of them.
// With scales of at least 1/4 besides (W6_MID), 32 s is a whole number and so is 1536 - 96 s, exact in half: (64 + code) s + that is the
// rounded code in one fused multiply-add. 64 + code is two bytes side by side, the nibble shifted up and 0x54 + the top bits, so nothing is
// merged before the permute that pairs them.
enum { W6_UNIT = 0, W6_SMALL = 1, W6_ANY = 2, W6_MID = 3 };
// The form for the four scale bytes of a lane and those of its warp's other lanes (absent ones filled with 0x38, a scale of 1)
// MID: whether the caller has the W6_MID form. The pair kernel has not: what bounds it is not its arithmetic, and a fourth form of eight groups
// beside the others took 234 us where three take 195 (2048 x 5120 -> 15360; 600 rows 132 and 116).
template <bool MID = true>
__device__ __forceinline__ int w6_mode(uint32_t sb4) {
    // bytes up to 0x48 (4.0), sign clear: adding 0x37 carries into bit 7 from 0x49 on
    const bool small = (((sb4 & 0x7f7f7f7fu) + 0x37373737u) & 0x80808080u) == 0u && (sb4 & 0x80808080u) == 0u;
    if (!__all_sync(0xffffffffu, small)) return W6_ANY;
    if (__all_sync(0xffffffffu, sb4 == 0x38383838u)) return W6_UNIT;
    return MID && __all_sync(0xffffffffu, (((sb4 | 0x80808080u) - 0x28282828u) & 0x80808080u) == 0x80808080u) ? W6_MID : W6_SMALL;      // from 0x28 (1/4) on
}
template <int MODE>
__device__ __forceinline__ void w6_group(const uint4 l, uint32_t ha, uint32_t hb, uint32_t sb, uint32_t (&o)[8]) {
    const uint32_t lw[4] = {l.x, l.y, l.z, l.w};
    const uint32_t hv[2] = {ha, hb};
    if constexpr (MODE == W6_UNIT) {
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            const uint32_t h = hv[w >> 1] >> (16 * (w & 1));
            const uint32_t te = __byte_perm(0x1000F0E0u, 0u, h & 0x3333u), to = __byte_perm(0x1000F0E0u, 0u, (h >> 2) & 0x3333u);
            const uint32_t de = (lw[w] & 0x0F0F0F0Fu) | te, dd = ((lw[w] >> 4) & 0x0F0F0F0Fu) | to;
            o[2 * w] = __byte_perm(de, dd, 0x5140);        // e0 o0 e1 o1
            o[2 * w + 1] = __byte_perm(de, dd, 0x7362);    // e2 o2 e3 o3
        }
        return;
    }
    if constexpr (MODE == W6_MID) {
        const __half2 s2 = __half2half2(__half(__nv_cvt_fp8_to_halfraw((__nv_fp8_storage_t)sb, __NV_E4M3)));
        const __half2 c2 = __hfma2(__float2half2_rn(-96.f), s2, __float2half2_rn(1536.f));
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            const uint32_t h = hv[w >> 1] >> (16 * (w & 1));
            const uint32_t te = __byte_perm(0x57565554u, 0u, h & 0x3333u), to = __byte_perm(0x57565554u, 0u, (h >> 2) & 0x3333u);
            const uint32_t ne = (lw[w] << 4) & 0xF0F0F0F0u, no = lw[w] & 0xF0F0F0F0u;
            uint32_t p[4] = {__byte_perm(ne, te, 0x5140), __byte_perm(no, to, 0x5140),       // (e0,e2) (e1,e3)
                             __byte_perm(ne, te, 0x7362), __byte_perm(no, to, 0x7362)};      // (e4,e6) (e5,e7)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const __half2 g = __hmax2(__hfma2(*reinterpret_cast<__half2*>(&p[i]), s2, c2), __float2half2_rn(1409.f));
                p[i] = *reinterpret_cast<const uint32_t*>(&g);
            }
            o[2 * w] = __byte_perm(p[0], p[1], 0x6240);
            o[2 * w + 1] = __byte_perm(p[2], p[3], 0x6240);
        }
        return;
    }
    const __half2 s2 = __half2half2(__half(__nv_cvt_fp8_to_halfraw((__nv_fp8_storage_t)sb, __NV_E4M3)));
    const __half2 magic = __float2half2_rn(1536.f);
    const __half2 c2 = __hmul2(__float2half2_rn(-1056.f), s2);
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        const uint32_t h = hv[w >> 1] >> (16 * (w & 1));
        const uint32_t te = __byte_perm(0x30201000u, 0u, h & 0x3333u), to = __byte_perm(0x30201000u, 0u, (h >> 2) & 0x3333u);
        const uint32_t ce = (lw[w] & 0x0F0F0F0Fu) | te, co = ((lw[w] >> 4) & 0x0F0F0F0Fu) | to;
        uint32_t p[4] = {__byte_perm(ce, 0x64646464u, 0x4140), __byte_perm(co, 0x64646464u, 0x4140),     // (e0,e2) (e1,e3)
                         __byte_perm(ce, 0x64646464u, 0x4342), __byte_perm(co, 0x64646464u, 0x4342)};    // (e4,e6) (e5,e7)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            __half2 g = *reinterpret_cast<__half2*>(&p[i]);
            if constexpr (MODE == W6_SMALL) {
                // (code - 32) * s is in [-128, 124]; the sum with 1536 stays where the spacing is 1
                g = __hmax2(__hadd2(__hfma2(g, s2, c2), magic), __float2half2_rn(1409.f));
            } else {
                g = __hmul2(__hsub2(g, __float2half2_rn(1056.f)), s2);
                g = __hmin2(__hmax2(g, __float2half2_rn(-127.f)), __float2half2_rn(127.f));
                g = __hadd2(g, magic);
            }
            p[i] = *reinterpret_cast<uint32_t*>(&g);
        }
        o[2 * w] = __byte_perm(p[0], p[1], 0x6240);
        o[2 * w + 1] = __byte_perm(p[2], p[3], 0x6240);
    }
}
// with the mode in a variable (the same in the whole warp)
template <bool MID = true>
__device__ __forceinline__ void w6_group_of(int mode, const uint4 l, uint32_t ha, uint32_t hb, uint32_t sb, uint32_t (&o)[8]) {
    if (MID && mode == W6_MID) w6_group<W6_MID>(l, ha, hb, sb, o);
    else if (mode == W6_SMALL) w6_group<W6_SMALL>(l, ha, hb, sb, o);
    else if (mode == W6_UNIT) w6_group<W6_UNIT>(l, ha, hb, sb, o);
    else w6_group<W6_ANY>(l, ha, hb, sb, o);
}
