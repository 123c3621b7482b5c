// The R256 rotation (the reference's csrc/common.cuh:99-126) in registers: buffer layout and butterflies for the quantizers
// (quant_rows.cu, which have the transposition inline, in forms with and without the rotation) and, whole, rotate256_regs for the
// weight packers (weight_pack.cu). A 256-wide group belongs to 8 consecutive lanes (a team), 32 consecutive values each;
// stages 0 and 1 run on those, a transposition through the team's padded piece of shared memory hands every lane the pairs
// (2t, 2t + 1) + 16 r, and stages 2 and 3 run on them.
#pragma once

#include "common.cuh"

// Transposition buffers: per 8-lane team 256 elements + 4 words of padding per 32 (288 words), laid out so that every
// shared-memory access of the transposition is free of bank conflicts across the four teams of a warp:
//   - a lane writes element 32 t8 + i as one 32-bit store per i; over a team's lanes these hit banks 4 t8 + i, i.e. one
//     residue class modulo 4. The four teams must cover the four classes: teams 1 and 3 store each element pair swapped
//     (column i ^ 1), teams 2 and 3 start two words later
//   - a lane reads element pairs (2 t8, 2 t8 + 1) + 16 r as 64-bit loads, 16 consecutive banks per team; a half-warp holds
//     two teams, which start 16 banks apart
// Teams 1 and 3 therefore hold their pairs as (odd element, even element) from the transposition on; the codes are
// swapped back when they are written out.
constexpr int kGroupWords = 304;          // team pitch inside a warp: 16 banks (mod 32) apart
constexpr int kWarpWords = 4 * 304 + 32;  // warp pitch: a multiple of 32 words with room for the two-word shift

__device__ __forceinline__ int tpad(int e) { return e + ((e >> 5) << 2); }

// Radix-4 butterfly of the regular Hadamard block on packed pairs; outputs in the reference's association:
//   r0 = .5*(((x0+x1)+x2)-x3)  r1 = .5*(((x0+x1)-x2)+x3)  r2 = .5*(((x0-x1)+x2)+x3)  r3 = .5*(((-x0+x1)+x2)+x3)
// HALVE = false leaves the factors 0.5 out.
template <bool HALVE = true>
__device__ __forceinline__ void h4x2(float2& x0, float2& x1, float2& x2, float2& x3) {
    const float2 m1 = make_float2(-1.f, -1.f), hf = make_float2(0.5f, 0.5f);
    const float2 s = __fadd2_rn(x0, x1);
    const float2 d = __ffma2_rn(x1, m1, x0);                         // x0 - x1
    const float2 r0 = __ffma2_rn(x3, m1, __fadd2_rn(s, x2));
    const float2 r1 = __fadd2_rn(__ffma2_rn(x2, m1, s), x3);
    const float2 r2 = __fadd2_rn(__fadd2_rn(d, x2), x3);
    const float2 r3 = __fadd2_rn(__ffma2_rn(d, m1, x2), x3);         // (-d + x2) + x3
    if (HALVE) x0 = __fmul2_rn(hf, r0), x1 = __fmul2_rn(hf, r1), x2 = __fmul2_rn(hf, r2), x3 = __fmul2_rn(hf, r3);
    else x0 = r0, x1 = r1, x2 = r2, x3 = r3;
}
// two radix-4 stages over 16 packed values: index bits (0,1) then (2,3) of the position in P
template <bool HALVE = true>
__device__ __forceinline__ void two_stages(float2 (&P)[16]) {
#pragma unroll
    for (int i = 0; i < 16; i += 4) h4x2<HALVE>(P[i], P[i + 1], P[i + 2], P[i + 3]);
#pragma unroll
    for (int i = 0; i < 4; ++i) h4x2<HALVE>(P[i], P[i + 4], P[i + 8], P[i + 12]);
}

// max(|a|, |b|, |c|) that is NaN as soon as one input is
__device__ __forceinline__ float max3_abs_nan(float a, float b, float c) {
    float m;
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(fabsf(a)), "f"(fabsf(b)), "f"(fabsf(c)));
    return m;
}


// This lane's place in its warp's transposition buffer
struct RotLane {
    int lane, team, tsw, t8;      // teams 1 and 3 (tsw) hold their pairs swapped after the transposition
    float* tbuf;                  // the team's buffer
    float* tbuf_w;                // where its transposition writes and reads start (two words later for teams 2 and 3)
};
__device__ __forceinline__ RotLane rot_lane(float* smem) {
    RotLane l;
    l.lane = threadIdx.x & 31, l.team = l.lane >> 3, l.tsw = l.team & 1, l.t8 = l.lane & 7;
    l.tbuf = smem + (threadIdx.x >> 5) * kWarpWords + l.team * kGroupWords + 4 * (l.team >> 1);
    l.tbuf_w = l.tbuf - 2 * (l.team >> 1);
    return l;
}
// v = elements 32 t8 .. 32 t8 + 31 of the group -> P[r] = rotated elements (2 t8, 2 t8 + 1) + 16 r (swapped pairs when tsw).
__device__ __forceinline__ void rotate256_regs(const float (&v)[32], float2 (&P)[16], const RotLane& l, unsigned wmask) {
#pragma unroll
    for (int i = 0; i < 16; ++i) P[i] = make_float2(v[i], v[i + 16]);
    two_stages(P);
    float* we = l.tbuf_w + tpad(l.t8 << 5) + l.tsw;     // even columns go one word up in a swapping team,
    float* wo = l.tbuf_w + tpad(l.t8 << 5) - l.tsw;     // odd columns one word down: column i ^ 1
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        float* w = (i & 1) ? wo : we;
        w[i] = P[i].x;
        w[16 + i] = P[i].y;   // element 32 t8 + 16 + i: same 32-run, no pad in between
    }
    __syncwarp(wmask);
#pragma unroll
    for (int r = 0; r < 16; ++r) P[r] = *reinterpret_cast<const float2*>(l.tbuf_w + tpad(2 * l.t8 + 16 * r));
    two_stages(P);   // index bits 4-7 = r
    __syncwarp(wmask);
}
// The way back: P as rotate256_regs leaves it -> v = rotated elements 32 t8 .. 32 t8 + 31 of the group.
__device__ __forceinline__ void untranspose256(const float2 (&P)[16], float (&v)[32], const RotLane& l, unsigned wmask) {
#pragma unroll
    for (int r = 0; r < 16; ++r) *reinterpret_cast<float2*>(l.tbuf_w + tpad(2 * l.t8 + 16 * r)) = P[r];
    __syncwarp(wmask);
    const float* re = l.tbuf_w + tpad(l.t8 << 5) + l.tsw;
    const float* ro = l.tbuf_w + tpad(l.t8 << 5) - l.tsw;
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = ((i & 1) ? ro : re)[i];
    __syncwarp(wmask);
}
