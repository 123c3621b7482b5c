// Dynamic per-token absmax int8 activation quantizer with the optional ConvRot rotation fused in.
//
// Entry points gpu_quant_rows / gpu_rotate_rows_f32 of the reference (csrc/kernels.cu:271-298, :316-327):
//   v = prologue(x[m, :])                      elementwise prologues; rounding to the activation dtype as there
//   v = R256(v) per 256-wide group             when rotate != 0 (csrc/common.cuh:99-126: four radix-4 stages of
//                                              the regular Hadamard block, each output 0.5*(((+-a+-b)+-c)+-d))
//   scale = max(min(amax, finite_max) * (1/127), 1e-30)      stored fp32
//   q = clamp(rint(T(T(v) / T(scale))), -128, 127)            T = activation dtype (csrc/kernels.cu:241-255)
//
// The kernel is bound by instruction issue before HBM, so it is organised around instruction count and around keeping
// the issue slots busy:
//   - without the rotation the kernel is short enough to wait for HBM: persistent CTAs walk row blocks and, while one
//     block is computed, one bulk asynchronous copy per row (cp.async.bulk, completion on an mbarrier) brings the next
//     block's rows into shared memory; with the rotation (arithmetic-bound) each CTA takes one block with direct loads
//   - a 256-wide group belongs to 8 consecutive lanes; a lane takes 32 consecutive elements (16-byte loads)
//   - stages 0 and 1 (index bits 0-3) run in registers on packed f32x2 pairs (element i with element i+16)
//   - the group is transposed through a padded per-warp shared-memory buffer; a lane then holds element pairs
//     (2t, 2t+1) + 16 r, r = 0..15, and runs stages 2 and 3 (index bits 4-7) in registers, again on packed pairs
//   - every butterfly adds in the reference's left-to-right order (a - b is fma(b, -1, a): one rounding, the same),
//     so results are bit-identical whichever thread computes them
//   - bf16 prologues of one variable (SiLU, GELU, GELU-tanh, the sigmoid of GATE) are a 65536-entry table built on
//     the device from the very expressions of the reference and read through L1 (keeping the hot part, 2^-14 <= |x| < 128,
//     in shared memory measured slower: 129 against 101 us at M = 4352, K = 12288, the index arithmetic and the bank
//     conflicts of 32 scattered 2-byte reads cost more than the L1 gather)
//   - the division by the scale is a multiplication by its reciprocal (exact for this purpose, see quant2), the
//     codes are rounded by cvt.rni straight from bf16 and packed with saturation, and go back through shared memory
//     so that each lane stores 32 contiguous bytes
#include <atomic>
#include <cstdlib>
#include <mutex>

#include "common.cuh"
#include "epilogue.cuh"
#include "rotate.cuh"

namespace {

enum { PRO_PLAIN = 0, PRO_RMS = 1, PRO_GATE = 2, PRO_SWIGLU = 3, PRO_LAYERNORM = 4, PRO_SILU = 5, PRO_GELU = 6,
       PRO_ADALN = 7, PRO_SITU = 8, PRO_LN_MOD = 9, PRO_LN_AFFINE = 10, PRO_GELU_TANH = 11, PRO_LN_AFFINE_SILU = 12,
       PRO_SITU_FAST = 13 };  // the reference's src/ffi.rs:15-29

enum { LUT_SILU = 0, LUT_GELU = 1, LUT_GELU_TANH = 2, LUT_SIGMOID = 3, LUT_COUNT = 4 };

// bf16 -> bf16 tables of the one-variable prologues: entry b = bf16(act(float(bf16 with bits b)))
__device__ uint16_t g_act_lut[LUT_COUNT][65536];

__global__ void build_lut_kernel(int which) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= 65536) return;
    const float x = __uint_as_float((uint32_t)b << 16);
    float y;
    switch (which) {
        case LUT_SILU: y = silu_f(x); break;
        case LUT_GELU: y = gelu_f(x); break;
        case LUT_GELU_TANH: y = gelu_tanh_f(x); break;
        default: y = sigmoid_f(x); break;
    }
    g_act_lut[which][b] = __bfloat16_as_ushort(__float2bfloat16_rn(y));
}

struct QuantArgs {
    const void* x;
    int64_t x_stride;   // elements between rows
    const void* g;      // PRO_GATE: gate logits
    int64_t g_stride;
    int64_t up_offset;  // PRO_SWIGLU, PRO_SITU*: column of the second half inside the x row
    int8_t* q;          // [M, K]
    float* scales;      // [M]
    float* out_f;       // when set: write the rotated fp32 rows here instead of quantizing
    int M, K;
    int rotate;
    int tpr;            // threads per row = K / 32 (quant_norm_kernel: warps per row)
    int rows_per_cta;
    int nblocks;        // row blocks; CTAs stride over them
    int lut;            // table index of the prologue, or -1
    const float* amax_in;   // when set: row maxima to quantize with (rows whose columns are split across devices)
    float* amax_out;        // when set: write each row's maximum here and stop (first pass of the same)
    // normalising prologues
    const float* norm_w;    // RMS / LAYERNORM weight [K] (nullable), LN_AFFINE weight
    const float* norm_b;    // LN_AFFINE bias [K]
    float eps;
    const void* mod_scale;  // [K] in the activation dtype (nullable except ADALN)
    const void* mod_shift;
    // shared-memory plan (byte offsets from the dynamic shared memory base), filled in by launch_quant
    int staged;             // rows arrive through the staging buffer (bulk copies) instead of direct loads
    uint32_t off_amax, off_norm, off_stage, off_bar;
    // when set (f32 rows, with q and out_f unset): the rotated rows leave as fixed-point numbers in three signed 8-bit digits, planes
    // [3][M, K], the row's factor in `scales`, the groups' shifts [K / 256][M] of spread rows in `shifts` (see store_digits); the first
    // CTA zeroes nzero words at `zero` for the kernel that follows
    int8_t* digits;
    uint8_t* shifts;
    int* zero;
    int nzero;
    int early;              // the stream's next kernel may start as soon as the rows are in (see early_trigger)
};

template <int PRO> __host__ __device__ constexpr bool is_ln() { return PRO == PRO_LAYERNORM || PRO == PRO_LN_MOD || PRO == PRO_LN_AFFINE; }
template <int PRO> __host__ __device__ constexpr bool is_norm() { return PRO == PRO_RMS || PRO == PRO_ADALN || is_ln<PRO>(); }
// prologues that read a second stream per row: the gate logits (GATE) or the other half of the row (SWIGLU, SITU)
template <int PRO> __host__ __device__ constexpr bool has_aux() {
    return PRO == PRO_GATE || PRO == PRO_SWIGLU || PRO == PRO_SITU || PRO == PRO_SITU_FAST;
}
// floats of shared memory a row needs for the sums of a normalising prologue: one partial per thread of the
// reference's block (ceil(K / 1024) warps), 32 warp sums, the total
__host__ __device__ inline int norm_words(int K) { return (((K >> 8) + 3) >> 2) * 32 + 33; }

template <typename T> __device__ __forceinline__ float finite_max();
template <> __device__ __forceinline__ float finite_max<float>() { return FLT_MAX; }
template <> __device__ __forceinline__ float finite_max<bf16>() { return 3.38953139e38f; }

__device__ __forceinline__ void unpack_bf16x8(const uint4 u, float* v) {
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        v[2 * i] = __uint_as_float(w[i] << 16);
        v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
}
__device__ __forceinline__ float2 bf16x2_f(const __nv_bfloat162 h) {
    const uint32_t w = *reinterpret_cast<const uint32_t*>(&h);
    return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}
// 32 consecutive elements -> floats, from global memory or from the staging buffer
template <typename T, bool SMEM> __device__ __forceinline__ void load32(const T* p, float (&v)[32]) {
    if constexpr (sizeof(T) == 2) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const uint4 u = SMEM ? reinterpret_cast<const uint4*>(p)[c] : gload(reinterpret_cast<const uint4*>(p) + c);
            unpack_bf16x8(u, v + 8 * c);
        }
    } else {
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const float4 a = SMEM ? reinterpret_cast<const float4*>(p)[c] : gload(reinterpret_cast<const float4*>(p) + c);
            v[4 * c] = a.x, v[4 * c + 1] = a.y, v[4 * c + 2] = a.z, v[4 * c + 3] = a.w;
        }
    }
}

__device__ __forceinline__ float lut_f(const uint16_t* lut, float x) {   // x holds a bf16 value; whole table, global
    return __uint_as_float((uint32_t)gload(lut + (__float_as_uint(x) >> 16)) << 16);
}
// Codes of two values: q = sat8(rint(T(T(v) / T(scale)))).
// bf16 fast path. Both operands of the division carry 8 significant bits: a = A 2^i, st = S 2^j with integers
// A, S < 256. A bf16 rounding boundary is M 2^k with M odd and 256 < M < 512; a quotient equal to one would need
// A 2^n = S M, impossible because the odd part of the left side is below 256 and that of the right side is at least 257.
// So the exact quotient differs from every boundary by at least 1 / (S M) > 2^-17 relative, while a (correctly rounded)
// reciprocal times a is within 2^-23 of it: both round to the same bf16, and no correction step is needed
// (tests/test_quant_division.py enumerates every pair of significands).
// The magic-number rint + saturating pack equal clamp(rint(.)) for finite values; the caller keeps rows that hold a NaN
// or an infinity off this path.
// (the fast path on two values already rounded to bf16, packed in one word)
__device__ __forceinline__ uint32_t quant2_bf16_bits(uint32_t au, float rcp) {
    const float2 a = make_float2(__uint_as_float(au << 16), __uint_as_float(au & 0xffff0000u));
    const float2 t = __fmul2_rn(a, make_float2(rcp, rcp));
    const __nv_bfloat162 tb = __floats2bfloat162_rn(t.x, t.y);
    const uint32_t tu = *reinterpret_cast<const uint32_t*>(&tb);
    // rint by adding 1.5 * 2^23 (round to nearest even at unit spacing, |t| <= 128): the integer sits in the low bits.
    // The float -> integer conversion instructions share a narrow pipe with the bf16 conversions above, and that
    // pipe, not HBM, bounded this kernel; the addition runs on the FP32 pipe instead.
    const float2 u = __fadd2_rn(make_float2(__uint_as_float(tu << 16), __uint_as_float(tu & 0xffff0000u)),
                                make_float2(12582912.f, 12582912.f));
    const int n0 = (int)__float_as_uint(u.x) - 0x4B400000, n1 = (int)__float_as_uint(u.y) - 0x4B400000;
    uint32_t packed;
    asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, 0;" : "=r"(packed) : "r"(n1), "r"(n0));
    return packed;   // byte 0 = code of the low half, byte 1 = code of the high half
}
template <typename T>
__device__ __forceinline__ uint32_t quant2(float2 v, float st, float rcp, bool fast) {
    if (sizeof(T) == 2 && fast) {
        const __nv_bfloat162 ab = __floats2bfloat162_rn(v.x, v.y);
        return quant2_bf16_bits(*reinterpret_cast<const uint32_t*>(&ab), rcp);
    }
    const int qx = clamp_rint_i8(rnd<T>(__fdiv_rn(rnd<T>(v.x), st)), -128.f);
    const int qy = clamp_rint_i8(rnd<T>(__fdiv_rn(rnd<T>(v.y), st)), -128.f);
    return (uint32_t)(qx & 0xff) | ((uint32_t)(qy & 0xff) << 8);
}

// 8 consecutive per-column values as floats
__device__ __forceinline__ void load8v(const float* p, float (&v)[8]) {
    const float4 a = gload(reinterpret_cast<const float4*>(p)), b = gload(reinterpret_cast<const float4*>(p) + 1);
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
}
__device__ __forceinline__ void load8v(const bf16* p, float (&v)[8]) {
    unpack_bf16x8(gload(reinterpret_cast<const uint4*>(p)), v);
}

// The reference's soft-capped gated activation (csrc/common.cuh:73-91), operation for operation.
__device__ __forceinline__ float stable_tanh_f(float x) {
    const float t = expm1f(__fmul_rn(-2.f, fabsf(x)));
    return copysignf(__fdiv_rn(-t, __fadd_rn(t, 2.f)), x);
}
__device__ __forceinline__ float situ_f(float hidden, float gate) {
    const float a = __fdiv_rn(__fmul_rn(4.f, stable_tanh_f(__fdiv_rn(gate, 4.f))), __fadd_rn(1.f, expf(-gate)));
    return __fmul_rn(a, __fmul_rn(25.f, stable_tanh_f(__fdiv_rn(hidden, 25.f))));
}
__device__ __forceinline__ float tanh_approx_f(float x) {
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float situ_fast_f(float hidden, float gate) {
    return __fmul_rn(__fdividef(__fmul_rn(4.f, tanh_approx_f(__fmul_rn(gate, 0.25f))), __fadd_rn(1.f, __expf(-gate))),
                     __fmul_rn(25.f, tanh_approx_f(__fmul_rn(hidden, 0.04f))));
}

// One bulk asynchronous copy, global -> this CTA's shared memory, completion credited to an mbarrier. Both addresses
// 16-byte aligned, size a multiple of 16 bytes.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

// The rotated values of a lane ((2 t8, 2 t8 + 1) + 16 r, pairs swapped when tsw) as the weight-only linear takes them:
// x = (d0 2^16 + d1 2^8 + d2) f with signed 8-bit digits and a power of two f, chosen so that a maximum lies in [2^21, 2^22): what rounds
// away is at most 2^-22 of that maximum. The product with the power of two is exact and rint comes with the addition of 1.5 * 2^23.
// The maximum is the row's as long as every group of 256 that is not all zero reaches 2^19 with it, so that no value loses more than 2^-20 of its
// group's maximum, about what the rotation's own f32 sums leave (two bf16 terms kept 2^-18 of each value). A row spread
// wider (a massive activation beside ordinary ones) has a power of two per group instead: the row's factor is stored negative, and
// f_group = f_row 2^-shift. A row holding an infinity or a NaN gets the factor NaN.
// P and the maxima come in units of `unit` (1/16 without the rotation's halvings).
constexpr int kDigitSpread = 3;           // binary orders of magnitude between the row's and a group's maximum that make a spread row
// floor(log2 v) of a positive v; a subnormal one's is found too, through a product
__device__ __forceinline__ int exponent_of(float v) {
    const bool low = v < 0x1p-90f;
    return (int)(__float_as_uint(low ? v * 0x1p64f : v) >> 23) - (low ? 127 + 64 : 127);
}
struct DigitMax { float row, least, group; };      // maxima: the row's, the smallest of its groups' that are not zero, this lane's group's
__device__ __forceinline__ void store_digits(float2 (&P)[16], DigitMax mx, float unit, const QuantArgs& p, bool live, int64_t m, int col, bool first,
                                             int tsw, int t8, float* tbuf, unsigned wmask) {
    float inv = 0.f, f = 0.f;
    if (!(mx.row <= FLT_MAX)) f = __int_as_float(0x7fc00000);
    else if (mx.row > 0.f) {
        const int kr = max(exponent_of(mx.row), -124);      // f ends at 2^-149
        int k = kr;
        if (kr - exponent_of(mx.least) >= kDigitSpread) {
            unit = -unit;
            if (mx.group > 0.f) k = max(exponent_of(mx.group), max(kr - kWo8MaxShift, -124));
            if (live && t8 == 0) p.shifts[(int64_t)(col >> 8) * p.M + m] = (uint8_t)(kr - k);
        }
        // f as a product of two, it may be subnormal; k + 64 where 2^(21 - k) would leave f32's range
        f = __uint_as_float((uint32_t)(127 - 21 + kr + (kr < -90 ? 64 : 0)) << 23) * (kr < -90 ? unit * 0x1p-64f : unit);
        if (k < -90) {
            k += 64;
#pragma unroll
            for (int r = 0; r < 16; ++r) P[r] = __fmul2_rn(P[r], make_float2(0x1p64f, 0x1p64f));
        }
        inv = __uint_as_float((uint32_t)(127 + 21 - k) << 23);
    }
    if (live && first) p.scales[m] = f;
    uint32_t w[32];
    const float2 inv2 = make_float2(inv, inv), magic = make_float2(12582912.f, 12582912.f);
#pragma unroll
    for (int r = 0; r < 16; ++r) {
        const float2 t = __ffma2_rn(P[r], inv2, magic);
        // 0x4B400000 + n; with 128 (2^16 + 2^8 + 1) added, the bytes are the digits plus 128
        w[2 * r] = __float_as_uint(t.x) + (0x808080u - 0x4B400000u), w[2 * r + 1] = __float_as_uint(t.y) + (0x808080u - 0x4B400000u);
    }
    uint16_t* cb = reinterpret_cast<uint16_t*>(tbuf);
    int8_t* q = p.digits + m * (int64_t)p.K + col;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const uint32_t pick = tsw ? (uint32_t)((6 - d) | (2 - d) << 4) : (uint32_t)((2 - d) | (6 - d) << 4);
#pragma unroll
        for (int r = 0; r < 16; ++r) cb[t8 + 8 * r] = (uint16_t)__byte_perm(w[2 * r], w[2 * r + 1], pick);
        __syncwarp(wmask);
        uint4 lo = reinterpret_cast<const uint4*>(tbuf)[2 * t8], hi = reinterpret_cast<const uint4*>(tbuf)[2 * t8 + 1];
        __syncwarp(wmask);
        lo.x ^= 0x80808080u, lo.y ^= 0x80808080u, lo.z ^= 0x80808080u, lo.w ^= 0x80808080u;
        hi.x ^= 0x80808080u, hi.y ^= 0x80808080u, hi.z ^= 0x80808080u, hi.w ^= 0x80808080u;
        if (live) {
            reinterpret_cast<uint4*>(q + d * (int64_t)p.M * p.K)[0] = lo;
            reinterpret_cast<uint4*>(q + d * (int64_t)p.M * p.K)[1] = hi;
        }
    }
}

__device__ int g_quant_status = 0;   // a staging wait that ran out records ST_TIMEOUT_FULL here

// v = T(act(a)) [* b] of the prologues without row statistics: a is the gate logit u (GATE), the row itself otherwise; u the second
// stream of the others. `lut`: the activation's table, or null.
template <typename T, int PRO, int N = 32>
__device__ __forceinline__ void elementwise_prologue(float* v, float* u, const uint16_t* lut) {
    if (PRO == PRO_GATE || PRO == PRO_SWIGLU || PRO == PRO_SILU || PRO == PRO_GELU || PRO == PRO_GELU_TANH) {
        float* a = PRO == PRO_GATE ? u : v;
        if (lut) {
#pragma unroll
            for (int i = 0; i < N; ++i) a[i] = lut_f(lut, a[i]);
        } else {
#pragma unroll
            for (int i = 0; i < N; ++i)
                a[i] = rnd<T>(PRO == PRO_GATE ? sigmoid_f(a[i]) : (PRO == PRO_SILU || PRO == PRO_SWIGLU) ? silu_f(a[i])
                              : PRO == PRO_GELU ? gelu_f(a[i]) : gelu_tanh_f(a[i]));
        }
        if (PRO == PRO_GATE || PRO == PRO_SWIGLU) {
#pragma unroll
            for (int i = 0; i < N; ++i) v[i] = rnd<T>(__fmul_rn(v[i], u[i]));
        }
    } else if (PRO == PRO_SITU || PRO == PRO_SITU_FAST) {
        // u = the gate half of the row; the product is not rounded here (csrc/kernels.cu:107-112)
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] = PRO == PRO_SITU ? situ_f(v[i], u[i]) : situ_fast_f(v[i], u[i]);
    }
}

// ---- rotated rows to codes and scales: the form of a block's linears and of the packers ---------------------------------------
// Kernels of their own beside the general one below: one row block per CTA, no staging, none of the other outputs, which leaves 56 to 64
// registers and 32 to 36 warps per SM (the general kernel: 80 and 24). What bounds them is instruction issue, so the rotation comes
// without its sixteen halvings: sums of unhalved values are the reference's times a power of two, whose rounding is the same as long as
// nothing overflows and nothing that matters is subnormal (values that small become code 0 beside any scale: scales end at
// 1e-30). An overflow, like an infinity or a NaN in the row, leaves something that is not finite among the rotated values; a CTA that
// meets one, or a value of 2^127, goes through its rows a second time with the halvings, the IEEE division and the exact clamp.

// The rotation of a lane's 32 consecutive values: P[r] = elements (2 t8, 2 t8 + 1) + 16 r of the group, swapped in a swapping team;
// 16 times the reference's values without HALVE.
template <bool HALVE>
__device__ __forceinline__ void rotate_lane(float2 (&P)[16], const float (&v)[32], float* tbuf_w, int t8, int tsw, unsigned wmask) {
#pragma unroll
    for (int i = 0; i < 16; ++i) P[i] = make_float2(v[i], v[i + 16]);
    two_stages<HALVE>(P);
    float* we = tbuf_w + tpad(t8 << 5) + tsw;
    float* wo = tbuf_w + tpad(t8 << 5) - tsw;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        float* w = (i & 1) ? wo : we;
        w[i] = P[i].x;
        w[16 + i] = P[i].y;
    }
    __syncwarp(wmask);
#pragma unroll
    for (int r = 0; r < 16; ++r) P[r] = *reinterpret_cast<const float2*>(tbuf_w + tpad(2 * t8 + 16 * r));
    two_stages<HALVE>(P);
    __syncwarp(wmask);
}
__device__ __forceinline__ float max32_abs_nan(const float2 (&P)[16]) {
    float m = 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) m = max3_abs_nan(m, P[i].x, P[i].y);
    return m;
}
// Code pairs (low 16 bits of c16[r], in element order) -> 32 contiguous bytes per lane of the group's 256
__device__ __forceinline__ void store_codes(const uint32_t (&c16)[16], int8_t* q, bool live, float* tbuf, int t8, unsigned wmask) {
    uint16_t* cb = reinterpret_cast<uint16_t*>(tbuf);
#pragma unroll
    for (int r = 0; r < 16; ++r) cb[t8 + 8 * r] = (uint16_t)c16[r];
    __syncwarp(wmask);
    const uint4 lo = reinterpret_cast<const uint4*>(tbuf)[2 * t8], hi = reinterpret_cast<const uint4*>(tbuf)[2 * t8 + 1];
    if (live) {
        reinterpret_cast<uint4*>(q)[0] = lo;
        reinterpret_cast<uint4*>(q)[1] = hi;
    }
}
// P = 16 x the rotated values, all finite; amax = the row's maximum
template <typename T>
__device__ __forceinline__ void codes_fast(float2 (&P)[16], uint32_t (&c16)[16], float amax, float scale, int tsw, unsigned wmask) {
    const float2 magic = make_float2(12582912.f, 12582912.f);       // rint: the integer's low byte is the sum's
    const uint32_t pick = tsw ? 0x0004u : 0x0040u;                   // the two low bytes in element order
    const float st = rnd<T>(scale);
    const float rcp = __frcp_rn(st);
    const float2 rcp2 = make_float2(rcp * 0.0625f, rcp * 0.0625f);
    if constexpr (sizeof(T) == 2) {
        auto quotient = [&](float2 v) {      // T(T(v) / T(scale)), see quant2
            const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y);
            const float2 t = __fmul2_rn(bf16x2_f(a), rcp2);
            return bf16x2_f(__floats2bfloat162_rn(t.x, t.y));
        };
        // 128 needs the clamp. Quotients grow with their dividends, so the maximum's tells for the row (about one row in eight). One form for the warp:
        // with rows of 256 its teams have four, and each would wait for the others' form (16896 x 256 6.7 us, 6.2 with one).
        if (!__any_sync(wmask, !(rnd<T>(rnd<T>(amax) * rcp) < 127.5f))) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const float2 u = __fadd2_rn(quotient(P[i]), magic);
                c16[i] = __byte_perm(__float_as_uint(u.x), __float_as_uint(u.y), pick);
            }
        } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const float2 u = __fadd2_rn(quotient(P[i]), magic);
                const int n0 = (int)__float_as_uint(u.x) - 0x4B400000, n1 = (int)__float_as_uint(u.y) - 0x4B400000;
                c16[i] = __byte_perm((uint32_t)min(n0, 127), (uint32_t)min(n1, 127), pick);
            }
        }
    } else {
        // The correctly rounded quotient: with the correctly rounded reciprocal y of b, q' = q + (a - b q) y is a / b rounded once q is
        // one of its two neighbours (Markstein 1990), which a first such step makes of a y. 16 a / (16 b) is the same quotient;
        // where something underflows on the way the code is 0. The maximum is 127 scales and 2^-22: nothing needs the clamp.
        const float2 nst2 = make_float2(st * -16.f, st * -16.f);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            float2 t = __fmul2_rn(P[i], rcp2);
            t = __ffma2_rn(__ffma2_rn(t, nst2, P[i]), rcp2, t);
            t = __ffma2_rn(__ffma2_rn(t, nst2, P[i]), rcp2, t);
            const float2 u = __fadd2_rn(t, magic);
            c16[i] = __byte_perm(__float_as_uint(u.x), __float_as_uint(u.y), pick);
        }
    }
}
template <typename T> __device__ __forceinline__ float row_scale(float amax) {
    return fmaxf(fminf(amax, finite_max<T>()) * (1.f / 127.f), 1.0e-30f);
}
// A lane's place in both kernels. `bits` in shared memory, zero before: [rows] maxima of the first pass, [rows] of the second, one word that
// is set when something is not finite or nearly so; for the digits then [rows] and [rows] complements of the groups' least maxima.
__host__ __device__ constexpr int direct_words(int rows, bool digits) { return (digits ? 4 : 2) * rows + 1; }
struct DirectLane {
    float *tbuf, *tbuf_w;     // the team's transposition buffer, and where the transposition starts in it
    unsigned* bits;
    int64_t m;                // the row it works on
    int rloc, col, t8, tsw;
    bool live, first;         // whether it stores; whether it stores the row's scale
    unsigned wmask;
};
// From a lane's values to stored codes; false when something in the CTA's rows is not finite.
template <typename T, bool DIGITS>
__device__ __forceinline__ bool direct_first(const QuantArgs& p, const DirectLane& l, const float (&v)[32]) {
    if (p.early) pdl_trigger();      // the row is in
    float2 P[16];
    rotate_lane<false>(P, v, l.tbuf_w, l.t8, l.tsw, l.wmask);
    unsigned b = __float_as_uint(max32_abs_nan(P));      // non-negative floats order as integers, infinities and NaNs above
    b = max(b, __shfl_xor_sync(l.wmask, b, 1));
    b = max(b, __shfl_xor_sync(l.wmask, b, 2));
    b = max(b, __shfl_xor_sync(l.wmask, b, 4));
    if (l.t8 == 0) {
        atomicMax(l.bits + l.rloc, b);
        if (DIGITS && b) atomicMax(l.bits + 2 * p.rows_per_cta + 1 + l.rloc, ~b);
        if (b >= 0x7f000000u) l.bits[2 * p.rows_per_cta] = 1u;     // 2^127: short of what rounds to an infinity of bf16
    }
    __syncthreads();
    if (l.bits[2 * p.rows_per_cta] != 0u) return false;
    pdl_trigger();
    if constexpr (DIGITS) {
        const DigitMax mx = {__uint_as_float(l.bits[l.rloc]), __uint_as_float(~l.bits[2 * p.rows_per_cta + 1 + l.rloc]), __uint_as_float(b)};
        store_digits(P, mx, 0.0625f, p, l.live, l.m, l.col, l.first, l.tsw, l.t8, l.tbuf, l.wmask);
    } else {
        const float amax = __uint_as_float(l.bits[l.rloc]) * 0.0625f, scale = row_scale<T>(amax);
        if (l.live && l.first) p.scales[l.m] = scale;
        uint32_t c16[16];
        codes_fast<T>(P, c16, amax, scale, l.tsw, l.wmask);
        store_codes(c16, p.q + l.m * (int64_t)p.K + l.col, l.live, l.tbuf, l.t8, l.wmask);
    }
    return true;
}
template <typename T, bool DIGITS>
__device__ __forceinline__ void direct_second(const QuantArgs& p, const DirectLane& l, const float (&v)[32]) {
    float2 P[16];
    rotate_lane<true>(P, v, l.tbuf_w, l.t8, l.tsw, l.wmask);
    float amax = 0.f;                                    // without NaNs, which the reference's fmaxf drops
#pragma unroll
    for (int i = 0; i < 16; ++i) amax = fmaxf(amax, fmaxf(fabsf(P[i].x), fabsf(P[i].y)));
    if constexpr (DIGITS) {
        amax = max32_abs_nan(P);                         // with them: the row's factor becomes one
        unsigned b = __float_as_uint(amax);
        b = max(b, __shfl_xor_sync(l.wmask, b, 1));
        b = max(b, __shfl_xor_sync(l.wmask, b, 2));
        b = max(b, __shfl_xor_sync(l.wmask, b, 4));
        amax = __uint_as_float(b);
        if (b) atomicMax(l.bits + 3 * p.rows_per_cta + 1 + l.rloc, ~b);
    }
    atomicMax(l.bits + p.rows_per_cta + l.rloc, __float_as_uint(amax));
    __syncthreads();
    const float group = amax;
    amax = __uint_as_float(l.bits[p.rows_per_cta + l.rloc]);
    if constexpr (DIGITS) {
        const DigitMax mx = {amax, __uint_as_float(~l.bits[3 * p.rows_per_cta + 1 + l.rloc]), group};
        store_digits(P, mx, 1.f, p, l.live, l.m, l.col, l.first, l.tsw, l.t8, l.tbuf, l.wmask);
    } else {
        const float scale = row_scale<T>(amax), st = rnd<T>(scale);
        if (l.live && l.first) p.scales[l.m] = scale;
        const uint32_t order = l.tsw ? 0x3201u : 0x3210u;
        uint32_t c16[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) c16[i] = __byte_perm(quant2<T>(P[i], st, 0.f, false), 0u, order);
        store_codes(c16, p.q + l.m * (int64_t)p.K + l.col, l.live, l.tbuf, l.t8, l.wmask);
    }
}
template <bool DIGITS> __device__ __forceinline__ void direct_clear(const QuantArgs& p, unsigned* bits) {
    for (int i = threadIdx.x; i < direct_words(p.rows_per_cta, DIGITS); i += blockDim.x) bits[i] = 0u;
}
// for the kernel that follows the digits
__device__ __forceinline__ void clear_counters(const QuantArgs& p) {
    if (blockIdx.x == 0)
        for (int i = threadIdx.x; i < p.nzero; i += blockDim.x) p.zero[i] = 0;
}

// Rows as they lie and the prologues without row statistics. f32 rows other than the packers' and SITU would spill and keep the general
// kernel. In a chain of launches, us, before | now (the halvings kept, the exact form in the same kernel): PLAIN 4352 x 3072 15.9 | 15.7, GATE 1111 x 3072
// 10.1 | 9.4.
template <typename T, int PRO> __host__ __device__ constexpr int direct_threads() {
    if (sizeof(T) == 4) return PRO == PRO_PLAIN ? 288 : 0;
    return is_norm<PRO>() || PRO == PRO_SITU ? 0 : PRO == PRO_SWIGLU ? 256 : 288;
}
// f32 rows are read in whole lines (lane t8 of a team the 16-byte pieces t8 + 8 j of its group) and pass through the team's buffer, piece c
// at c ^ (c >> 3), into 32 consecutive values per lane: read as those, a load touched 32 lines for 16 bytes each. 5120 x 5120
// f32 packed: 46 -> 31 us; the digits of 512 x 9728 with SWIGLU 25 -> 21.
template <typename T, int PRO>
__device__ __forceinline__ void direct_values(const QuantArgs& p, const DirectLane& l, float (&v)[32]) {
    if constexpr (sizeof(T) == 4) {
        const float4* x = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p.x) + l.m * p.x_stride + (l.col & ~255)) + l.t8;
        const float4* up = PRO == PRO_SWIGLU ? reinterpret_cast<const float4*>(reinterpret_cast<const float*>(x) + p.up_offset) : x;
        float4* stage = reinterpret_cast<float4*>(l.tbuf);
        constexpr int kAhead = PRO == PRO_SWIGLU ? 4 : 8;      // pieces requested together
#pragma unroll
        for (int j0 = 0; j0 < 8; j0 += kAhead) {
            float4 a[kAhead], b[kAhead];
#pragma unroll
            for (int j = 0; j < kAhead; ++j) {
                a[j] = gload(x + 8 * (j0 + j));
                if (PRO == PRO_SWIGLU) b[j] = gload(up + 8 * (j0 + j));
            }
#pragma unroll
            for (int j = 0; j < kAhead; ++j) {
                if constexpr (PRO == PRO_SWIGLU) {
                    a[j].x = __fmul_rn(silu_f(a[j].x), b[j].x), a[j].y = __fmul_rn(silu_f(a[j].y), b[j].y);
                    a[j].z = __fmul_rn(silu_f(a[j].z), b[j].z), a[j].w = __fmul_rn(silu_f(a[j].w), b[j].w);
                }
                stage[8 * (j0 + j) + (l.t8 ^ (j0 + j))] = a[j];
            }
        }
        __syncwarp(l.wmask);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float4 a = stage[8 * l.t8 + (j ^ l.t8)];
            v[4 * j] = a.x, v[4 * j + 1] = a.y, v[4 * j + 2] = a.z, v[4 * j + 3] = a.w;
        }
        __syncwarp(l.wmask);
    } else if constexpr (PRO == PRO_GATE || PRO == PRO_SWIGLU) {
        // two streams: read in whole lines too, multiplied there (eight values of a lane at a time) and passed on as the bf16 they are rounded to.
        // 64 bytes a lane from each left every sector to be fetched in turn: 1111 x 8192 SwiGLU 20.9 us, now 18.0; 1111 x 3072 gated 10.4, now 8.9.
        const int64_t g0 = l.m * p.x_stride + (l.col & ~255);
        const uint4* x = reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(p.x) + g0) + l.t8;
        const uint4* aux = PRO == PRO_GATE ? reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(p.g) + l.m * p.g_stride + (l.col & ~255)) + l.t8
                                           : reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(p.x) + g0 + p.up_offset) + l.t8;
        const uint16_t* lut = p.lut >= 0 ? g_act_lut[p.lut] : nullptr;
        uint4* stage = reinterpret_cast<uint4*>(l.tbuf);
        uint4 xw[4], uw[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) xw[j] = gload(x + 8 * j), uw[j] = gload(aux + 8 * j);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float a[8], u[8];
            unpack_bf16x8(xw[j], a), unpack_bf16x8(uw[j], u);
            elementwise_prologue<T, PRO, 8>(a, u, lut);
            uint32_t o[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) o[i] = __byte_perm(__float_as_uint(a[2 * i]), __float_as_uint(a[2 * i + 1]), 0x7632);      // rounded: the upper halves
            const int c = l.t8 + 8 * j;
            stage[c ^ ((c >> 2) & 7)] = make_uint4(o[0], o[1], o[2], o[3]);
        }
        __syncwarp(l.wmask);
#pragma unroll
        for (int k = 0; k < 4; ++k) unpack_bf16x8(stage[(4 * l.t8 + k) ^ l.t8], v + 8 * k);
        __syncwarp(l.wmask);
    } else {
        float u[32];
        const T* x = reinterpret_cast<const T*>(p.x) + l.m * p.x_stride + l.col;
        load32<T, false>(x, v);
        if (has_aux<PRO>()) load32<T, false>(x + p.up_offset, u);
        if (p.early) pdl_trigger();
        elementwise_prologue<T, PRO>(v, u, PRO != PRO_GELU && p.lut >= 0 ? g_act_lut[p.lut] : nullptr);      // GELU's table: see launch_quant
    }
}
__device__ __forceinline__ DirectLane direct_lane(const QuantArgs& p, uint8_t* smem, unsigned tid, unsigned wmask) {
    const int warp = tid >> 5, lane = tid & 31, team = lane >> 3;
    const int rloc = tid / (unsigned)p.tpr, tin = tid - rloc * p.tpr;
    const int64_t m = (int64_t)blockIdx.x * p.rows_per_cta + rloc;
    float* tbuf = reinterpret_cast<float*>(smem) + warp * kWarpWords + team * kGroupWords + 4 * (team >> 1);
    // idle rows compute on the last row and store nothing; the last warp of a CTA may be partial (threads = rows * K / 32)
    return {tbuf, tbuf - 2 * (team >> 1), reinterpret_cast<unsigned*>(smem + p.off_amax), m < p.M ? m : p.M - 1, rloc, tin << 5, tin & 7, team & 1,
            m < p.M, tin == 0, wmask};
}
// The thread's index, read anew: what is worked out from it need not stay in registers while a row's 32 values and their look-ups fill them
__device__ __forceinline__ unsigned tid_anew() {
    unsigned t;
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
    return t;
}
// The second pass, out of line: what it holds would take registers from the first. The warp's mask is the kernel's: it says which lanes there are,
// and is read where all of them are together.
template <typename T, int PRO, bool DIGITS>
__device__ __noinline__ void direct_again(const QuantArgs& p, unsigned wmask) {
    extern __shared__ __align__(128) uint8_t smem[];
    const DirectLane l = direct_lane(p, smem, threadIdx.x, wmask);
    float v[32];
    direct_values<T, PRO>(p, l, v);
    direct_second<T, DIGITS>(p, l, v);
}
template <typename T, int PRO, int MAXT, bool DIGITS>
__global__ void __launch_bounds__(MAXT, MAXT <= 288 ? 4 : 1) quant_direct_kernel(const __grid_constant__ QuantArgs p) {
    extern __shared__ __align__(128) uint8_t smem[];
    constexpr bool kAnew = sizeof(T) == 2 && (PRO == PRO_SILU || PRO == PRO_GELU || PRO == PRO_GELU_TANH || PRO == PRO_SWIGLU);
    const DirectLane l = direct_lane(p, smem, threadIdx.x, __activemask());
    direct_clear<DIGITS>(p, l.bits);
    pdl_wait();
    if (DIGITS) clear_counters(p);
    __syncthreads();
    bool done;
    {
        float v[32];
        direct_values<T, PRO>(p, l, v);
        if constexpr (kAnew) done = direct_first<T, DIGITS>(p, direct_lane(p, smem, tid_anew(), l.wmask), v);
        else done = direct_first<T, DIGITS>(p, l, v);
    }
    if (!done) direct_again<T, PRO, DIGITS>(p, l.wmask);
}

// Normalising prologues on bf16 rows. The row sums are added in the reference's order (csrc/kernels.cu:113-147, csrc/common.cuh:30-55), so
// that they, and everything after them, come out bit for bit: there a block of nwr = ceil(K / 1024) warps holds the row, warp w the
// groups w, w + nwr, ..., lane l elements 8 l .. 8 l + 7 of each; a thread adds its elements in that order, then a xor-shuffle tree
// runs over the lanes and another over the warps. Here the same warps hold the same elements until the row is normalised: the sums are a
// thread's own, loads (rows, weights, modulation) are whole lines, and a row takes one barrier per sum. The normalised values pass
// through shared memory as bf16, which they are, into the rotation's layout: warp w' takes the groups 4 w' .. 4 w' + 3 there, from a
// slice that lies in its own transposition buffer. With the sums in the rotation's layout, running from group to group through
// shared memory in up to four rounds with a quarter of the lanes at work each, LN_MOD was 50 instructions a value where PLAIN was 22.
// In a chain of launches: LN_MOD 4352 x 3072 33.3 -> 25.3 us, RMS 1111 x 3072 11.1 -> 8.2.
__device__ __forceinline__ void row_barrier(int rloc, int warps) {
    if (warps == 1) __syncwarp();
    else named_bar_sync(1 + rloc, 32 * warps);
}
// f32 rows (RMS without modulation, the weight-only linear's): the same with 1 KB a group.
// ROWS: rows a warp holds, more than one for rows of 256 (four) and 512 (two) values: a group each in the same four places. With a row a warp three of its four
// teams had nothing to rotate: 16896 x 256 RMS 19.9 us, 8.3 with four rows; 16896 x 512 21.6 and 13.6 with two.
template <typename T, int PRO, int ROWS>
__device__ __forceinline__ void norm_values(const QuantArgs& p, const DirectLane& l, uint8_t* smem, float (&v)[32]) {
    static_assert((sizeof(T) == 2 || PRO == PRO_RMS) && (sizeof(T) == 2 || ROWS == 1), "f32 rows: RMS only, a row a warp or more");
    constexpr int kPer = 4 / ROWS;              // places of a row
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwr = ROWS > 1 ? 1 : p.tpr, row0 = ROWS > 1 ? warp * ROWS : l.rloc;
    const int w = ROWS > 1 ? 0 : warp - l.rloc * nwr, ngroups = ROWS > 1 ? kPer : p.K >> 8, grp = l.col >> 8;
    float* slice0 = reinterpret_cast<float*>(smem) + (ROWS > 1 ? warp : l.rloc * nwr) * kWarpWords;       // the row's first warp's buffer
    float* sums = reinterpret_cast<float*>(smem + p.off_norm) + l.rloc * 64;          // [2][32]
    auto group_of = [&](int i) { return ROWS > 1 ? i % kPer : w + nwr * i; };         // in place i
    const T* x = reinterpret_cast<const T*>(p.x) + (ROWS > 1 ? 0 : l.m * p.x_stride) + 8 * lane;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int g = group_of(i);
        if constexpr (ROWS > 1) {
            const int64_t m = min((int64_t)blockIdx.x * p.rows_per_cta + row0 + i / kPer, (int64_t)p.M - 1);
            unpack_bf16x8(gload(reinterpret_cast<const uint4*>(x + m * p.x_stride + (g << 8))), v + 8 * i);
        } else if constexpr (sizeof(T) == 2) {
            unpack_bf16x8(g < ngroups ? gload(reinterpret_cast<const uint4*>(x + (g << 8))) : make_uint4(0, 0, 0, 0), v + 8 * i);
        } else {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float4 a = g < ngroups ? gload(reinterpret_cast<const float4*>(x + (g << 8)) + h) : make_float4(0.f, 0.f, 0.f, 0.f);
                v[8 * i + 4 * h] = a.x, v[8 * i + 4 * h + 1] = a.y, v[8 * i + 4 * h + 2] = a.z, v[8 * i + 4 * h + 3] = a.w;
            }
        }
    }
    auto row_sum = [&](int r, bool squares, float* slot) -> float {      // r: the warp's row
        float s = 0.f;                             // the zeros of missing groups come last and change nothing
#pragma unroll
        for (int i = 0; i < 8 * kPer; ++i) s = squares ? __fmaf_rn(v[8 * kPer * r + i], v[8 * kPer * r + i], s) : __fadd_rn(s, v[8 * kPer * r + i]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s = __fadd_rn(s, __shfl_xor_sync(0xffffffffu, s, o));
        if constexpr (ROWS > 1) return __fadd_rn(s, 0.f);      // the tree over one warp adds zeros
        if (lane == 0) slot[w] = s;
        row_barrier(l.rloc, nwr);
        s = lane < nwr ? slot[lane] : 0.f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s = __fadd_rn(s, __shfl_xor_sync(0xffffffffu, s, o));
        return s;
    };
    if constexpr (is_ln<PRO>()) {
        float mean[ROWS];
#pragma unroll
        for (int r = 0; r < ROWS; ++r) mean[r] = __fdiv_rn(row_sum(r, false, sums), (float)p.K);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float sub = group_of(i) < ngroups ? mean[i / kPer] : 0.f;
#pragma unroll
            for (int j = 0; j < 8; j += 2) {
                const float2 d = __fadd2_rn(make_float2(v[8 * i + j], v[8 * i + j + 1]), make_float2(-sub, -sub));
                v[8 * i + j] = d.x, v[8 * i + j + 1] = d.y;
            }
        }
    }
    float rstd[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) rstd[r] = rsqrtf(__fadd_rn(__fdiv_rn(row_sum(r, true, sums + 32), (float)p.K), p.eps));
    const bf16* ms_p = reinterpret_cast<const bf16*>(p.mod_scale);
    const bf16* sh_p = reinterpret_cast<const bf16*>(p.mod_shift);
    if constexpr (sizeof(T) == 4) {
        const float2 rstd2 = make_float2(rstd[0], rstd[0]);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int g = group_of(i);
            if (g >= ngroups) break;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float* e = v + 8 * i + 4 * h;
                float2 a = __fmul2_rn(make_float2(e[0], e[1]), rstd2), b = __fmul2_rn(make_float2(e[2], e[3]), rstd2);
                if (p.norm_w) {
                    const float4 nw = gload(reinterpret_cast<const float4*>(p.norm_w + (g << 8) + 8 * lane) + h);
                    a = __fmul2_rn(a, make_float2(nw.x, nw.y)), b = __fmul2_rn(b, make_float2(nw.z, nw.w));
                }
                const int c = ((g & 3) << 6) + 2 * lane + h;
                reinterpret_cast<float4*>(slice0 + (g >> 2) * kWarpWords)[c ^ ((c >> 3) & 7)] = make_float4(a.x, a.y, b.x, b.y);
            }
        }
        row_barrier(l.rloc, nwr);
        const float4* mine = reinterpret_cast<const float4*>(slice0 + w * kWarpWords) + ((grp - 4 * w) << 6);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const float4 a = mine[(8 * l.t8 + k) ^ l.t8];
            v[4 * k] = a.x, v[4 * k + 1] = a.y, v[4 * k + 2] = a.z, v[4 * k + 3] = a.w;
        }
        __syncwarp();
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int g = group_of(i);
            if (g >= ngroups) break;
            const float2 rstd2 = make_float2(rstd[i / kPer], rstd[i / kPer]);
            const int c0 = (g << 8) + 8 * lane;
            uint4 mw = make_uint4(0, 0, 0, 0), sw = mw;
            float nw[8], nb[8];
            if (ms_p) mw = gload(reinterpret_cast<const uint4*>(ms_p + c0)), sw = gload(reinterpret_cast<const uint4*>(sh_p + c0));
            const bool has_w = (PRO == PRO_RMS || PRO == PRO_LAYERNORM || PRO == PRO_LN_AFFINE) && p.norm_w;
            if (has_w) load8v(p.norm_w + c0, nw);
            if (PRO == PRO_LN_AFFINE) load8v(p.norm_b + c0, nb);
            const uint32_t m4[4] = {mw.x, mw.y, mw.z, mw.w}, s4[4] = {sw.x, sw.y, sw.z, sw.w};
            uint32_t o[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                // two values at a time, one packed conversion per rounding (a scalar conversion runs on a narrow pipe)
                float2 n = __fmul2_rn(make_float2(v[8 * i + 2 * j], v[8 * i + 2 * j + 1]), rstd2);
                const float2 ms = make_float2(__uint_as_float(m4[j] << 16), __uint_as_float(m4[j] & 0xffff0000u));
                const float2 sh = make_float2(__uint_as_float(s4[j] << 16), __uint_as_float(s4[j] & 0xffff0000u));
                auto round2 = [](float2 f) { return bf16x2_f(__floats2bfloat162_rn(f.x, f.y)); };
                // 1 + scale as a bf16 addition rounds once where the reference rounds to f32 first, which makes no difference (the f32
                // sum is inexact only beside a scale below 2^-16 or above 2^16, and neither comes near a tie of bf16)
                auto one_plus = [&]() { return bf16x2_f(__hadd2(__floats2bfloat162_rn(1.f, 1.f), *reinterpret_cast<const __nv_bfloat162*>(&m4[j]))); };
                if (PRO == PRO_ADALN) {                // one rounding
                    n = __ffma2_rn(n, __fadd2_rn(make_float2(1.f, 1.f), ms), sh);
                } else if (PRO == PRO_LN_AFFINE) {
                    n = __ffma2_rn(n, make_float2(nw[2 * j], nw[2 * j + 1]), make_float2(nb[2 * j], nb[2 * j + 1]));
                } else {
                    if (has_w) n = __fmul2_rn(n, make_float2(nw[2 * j], nw[2 * j + 1]));
                    if (PRO == PRO_LN_MOD) {           // one rounding after the norm, one after the multiply-add
                        n = ms_p ? __ffma2_rn(round2(n), one_plus(), sh) : __ffma2_rn(round2(n), make_float2(1.f, 1.f), make_float2(0.f, 0.f));
                    } else if (ms_p) {                 // RMS, LAYERNORM: every step rounded
                        n = __fadd2_rn(round2(__fmul2_rn(one_plus(), round2(n))), sh);
                    }
                }
                const __nv_bfloat162 h = __floats2bfloat162_rn(n.x, n.y);
                o[j] = *reinterpret_cast<const uint32_t*>(&h);
            }
            // piece (g & 3) * 32 + lane of the slice, its low bits mixed with the next ones: free of bank conflicts both ways
            const int c = ((ROWS > 1 ? i : g & 3) << 5) + lane;
            reinterpret_cast<uint4*>(slice0 + (ROWS > 1 ? 0 : g >> 2) * kWarpWords)[c ^ ((c >> 2) & 7)] = make_uint4(o[0], o[1], o[2], o[3]);
        }
        row_barrier(l.rloc, nwr);
        const uint4* mine = reinterpret_cast<const uint4*>(slice0 + w * kWarpWords);
        const int place = ROWS > 1 ? lane >> 3 : grp - 4 * w;
#pragma unroll
        for (int k = 0; k < 4; ++k) unpack_bf16x8(mine[(place * 32 + 4 * l.t8 + k) ^ l.t8], v + 8 * k);
        __syncwarp();                                  // the slice is the transposition buffer from here on
    }
}
template <int ROWS>
__device__ __forceinline__ DirectLane norm_lane(const QuantArgs& p, uint8_t* smem) {
    if constexpr (ROWS > 1) {
        constexpr int kPer = 4 / ROWS;
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, team = lane >> 3, rloc = warp * ROWS + team / kPer;
        const int64_t m = (int64_t)blockIdx.x * p.rows_per_cta + rloc;
        float* tbuf = reinterpret_cast<float*>(smem) + warp * kWarpWords + team * kGroupWords + 4 * (team >> 1);
        return {tbuf, tbuf - 2 * (team >> 1), reinterpret_cast<unsigned*>(smem + p.off_amax), m < p.M ? m : p.M - 1, rloc,
                (team % kPer << 8) + ((lane & 7) << 5), lane & 7, team & 1, m < p.M, team % kPer == 0 && (lane & 7) == 0, 0xffffffffu};
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, team = lane >> 3, nwr = p.tpr;      // nwr: warps per row
    const int rloc = warp / nwr, w = warp - rloc * nwr, ngroups = p.K >> 8, grp = min(4 * w + team, ngroups - 1);
    const int64_t m = (int64_t)blockIdx.x * p.rows_per_cta + rloc;
    float* tbuf = reinterpret_cast<float*>(smem) + warp * kWarpWords + team * kGroupWords + 4 * (team >> 1);
    // teams past the row's last group redo it and store nothing, like rows past the last
    return {tbuf, tbuf - 2 * (team >> 1), reinterpret_cast<unsigned*>(smem + p.off_amax), m < p.M ? m : p.M - 1, rloc,
            (grp << 8) + ((lane & 7) << 5), lane & 7, team & 1, m < p.M && 4 * w + team < ngroups, w == 0 && lane == 0, 0xffffffffu};
}
template <typename T, int PRO, bool DIGITS, int ROWS>
__device__ __noinline__ void norm_again(const QuantArgs& p) {
    extern __shared__ __align__(128) uint8_t smem[];
    const DirectLane l = norm_lane<ROWS>(p, smem);
    float v[32];
    norm_values<T, PRO, ROWS>(p, l, smem, v);
    direct_second<T, DIGITS>(p, l, v);
}
template <typename T, int PRO, int MAXT, bool DIGITS, int ROWS>
__global__ void __launch_bounds__(MAXT, MAXT <= 256 ? 4 : 1) quant_norm_kernel(const __grid_constant__ QuantArgs p) {
    extern __shared__ __align__(128) uint8_t smem[];
    const DirectLane l = norm_lane<ROWS>(p, smem);
    direct_clear<DIGITS>(p, l.bits);
    pdl_wait();
    if (DIGITS) clear_counters(p);
    __syncthreads();
    bool done;
    {
        float v[32];
        norm_values<T, PRO, ROWS>(p, l, smem, v);
        done = direct_first<T, DIGITS>(p, l, v);
    }
    if (!done) norm_again<T, PRO, DIGITS, ROWS>(p);
}

// MAXT = 384 asks for two CTAs per SM (at most 80 registers: 768 threads with the next block's rows in flight);
// longer rows take one larger CTA.
template <typename T, int PRO, int MAXT>
__global__ void __launch_bounds__(MAXT, MAXT <= 384 ? 2 : 1) quant_rows_kernel(const QuantArgs p) {
    const bool staged = p.staged, rotate = p.rotate;
    extern __shared__ __align__(128) uint8_t smem[];
    const uint16_t* lut = g_act_lut[p.lut >= 0 ? p.lut : 0];
    const unsigned wmask = __activemask();            // the last warp of a CTA may be partial (threads = rows * K / 32)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;   // nwarps: whole warps
    const int team = lane >> 3, tsw = team & 1;        // team of the warp; teams 1 and 3 keep their pairs swapped
    float* tbuf = reinterpret_cast<float*>(smem) + warp * kWarpWords + team * kGroupWords + 4 * (team >> 1);   // this team's buffer
    float* tbuf_w = tbuf - 2 * (team >> 1);            // where its transposition writes and reads start (two words later for teams 2, 3)
    unsigned* amax_s = reinterpret_cast<unsigned*>(smem + p.off_amax);   // [3][rows]
    float* norm_s = reinterpret_cast<float*>(smem + p.off_norm);         // [rows][norm_words(K)], normalising prologues only
    const bool use_lut = sizeof(T) == 2 && p.lut >= 0;
    const uint32_t bar = smem_u32(smem + p.off_bar);
    uint8_t* stage = smem + p.off_stage;              // [x rows | aux rows], one block of rows
    const uint32_t row_bytes = (uint32_t)p.K * sizeof(T);

    for (int i = threadIdx.x; i < 3 * p.rows_per_cta; i += blockDim.x) amax_s[i] = 0u;
    if (staged && threadIdx.x == 0) {
        mbar_init(bar, 1);
        fence_mbar_init();
    }
    pdl_wait();
    __syncthreads();

    // Staging: the rows of block `blk` (and their second stream) -> the staging buffer, one bulk copy each, issued by
    // the first warp; the barrier's phase completes when all their bytes have landed.
    auto issue_block = [&](int blk) {
        if (warp != 0) return;
        const int64_t m0 = (int64_t)blk * p.rows_per_cta;
        const int live = (int)min((int64_t)p.rows_per_cta, (int64_t)p.M - m0);
        if (lane == 0) mbar_arrive_expect_tx(bar, (uint32_t)live * row_bytes * (has_aux<PRO>() ? 2u : 1u));
        __syncwarp();
        for (int r = lane; r < live; r += 32) {
            const T* src = reinterpret_cast<const T*>(p.x) + (m0 + r) * p.x_stride;
            bulk_load(smem_u32(stage + (size_t)r * row_bytes), src, row_bytes, bar);
            if (has_aux<PRO>()) {
                const T* aux = PRO == PRO_GATE ? reinterpret_cast<const T*>(p.g) + (m0 + r) * p.g_stride : src + p.up_offset;
                bulk_load(smem_u32(stage + (size_t)(p.rows_per_cta + r) * row_bytes), aux, row_bytes, bar);
            }
        }
    };
    if (staged && (int)blockIdx.x < p.nblocks) issue_block(blockIdx.x);

    const int tpr = p.tpr;
    const int rloc = threadIdx.x / tpr;               // row inside the CTA
    const int tin = threadIdx.x - rloc * tpr;         // thread inside the row
    const int grp = tin >> 3, t8 = tin & 7;
    const int col = (grp << 8) + (t8 << 5);
    int it = 0;
    for (int blk = blockIdx.x; blk < p.nblocks; blk += gridDim.x, ++it) {
        const int64_t m_raw = (int64_t)blk * p.rows_per_cta + rloc;
        const bool live = m_raw < p.M;
        const int64_t m = live ? m_raw : p.M - 1;      // idle rows compute on the last row (or on stale staging) and store nothing

        float v[32], u[32];
        if (staged) {
            // bounded wait for this block's bytes; on expiry the CTA records the fact and leaves
            bool ok = mbar_try_wait(bar, it & 1);
            if (!ok) {
                const uint64_t t0 = globaltimer_ns();
                for (uint32_t n = 1; !(ok = mbar_try_wait(bar, it & 1)); ++n)
                    if ((n & 255u) == 0u && globaltimer_ns() - t0 > kWaitLimitNs) break;
            }
            if (!ok) {
                atomicCAS(&g_quant_status, 0, ST_TIMEOUT_FULL);
                return;
            }
            const T* xs = reinterpret_cast<const T*>(stage + (size_t)rloc * row_bytes) + col;
            load32<T, true>(xs, v);
            if (has_aux<PRO>()) load32<T, true>(reinterpret_cast<const T*>(stage + (size_t)(p.rows_per_cta + rloc) * row_bytes) + col, u);
            // every thread holds its elements, so the buffer can take the next block; the copy engine writes through the
            // asynchronous proxy, hence the proxy fence between these reads and the barrier that releases the buffer
            fence_proxy_async_smem();
            __syncthreads();
            if (blk + (int)gridDim.x < p.nblocks) issue_block(blk + gridDim.x);
        } else {
            const T* x = reinterpret_cast<const T*>(p.x) + m * p.x_stride + col;
            load32<T, false>(x, v);
            if (PRO == PRO_GATE) load32<T, false>(reinterpret_cast<const T*>(p.g) + m * p.g_stride + col, u);
            else if (has_aux<PRO>()) load32<T, false>(x + p.up_offset, u);
        }

        elementwise_prologue<T, PRO>(v, u, use_lut ? lut : nullptr);

        if constexpr (is_norm<PRO>()) {
            // Row statistics in the reference's order of additions (csrc/kernels.cu:113-147, csrc/common.cuh:30-55), so
            // that the sums, and everything after them, come out bit for bit: there a block of nwr = ceil(K / 1024)
            // warps holds the row, warp w the groups w, w + nwr, ..., lane l elements 8 l .. 8 l + 7 of each; a thread
            // adds its elements in that order, then a xor-shuffle tree runs over the lanes and another over the warps.
            // Here a thread holds four such 8-runs of one group, so the running sums pass from group to group through
            // shared memory, one round per group of a reference warp.
            const int ngroups = p.K >> 8, nwr = (ngroups + 3) >> 2, words = nwr * 32 + 33;
            const int nrounds = (ngroups + nwr - 1) / nwr;
            float* part = norm_s + rloc * words;
            const int rgi = grp / nwr, rw = grp - rgi * nwr;
            auto row_sum = [&](bool squares) -> float {
                for (int round = 0; round < nrounds; ++round) {
                    if (rgi == round) {
#pragma unroll
                        for (int sub = 0; sub < 4; ++sub) {
                            float* slot = part + rw * 32 + 4 * t8 + sub;
                            float ss = round ? *slot : 0.f;
#pragma unroll
                            for (int j = 0; j < 8; ++j) {
                                const float e = v[8 * sub + j];
                                ss = squares ? __fmaf_rn(e, e, ss) : __fadd_rn(ss, e);
                            }
                            *slot = ss;
                        }
                    }
                    __syncthreads();
                }
                // the two shuffle trees run in whole warps only
                for (int pi = warp; pi < p.rows_per_cta * nwr && warp < nwarps; pi += nwarps) {
                    const int row = pi / nwr, ww = pi - row * nwr;
                    float* pr = norm_s + row * words;
                    float t = pr[ww * 32 + lane];
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) t = __fadd_rn(t, __shfl_xor_sync(0xffffffffu, t, o));
                    if (lane == 0) pr[nwr * 32 + ww] = t;
                }
                __syncthreads();
                for (int row = warp; row < p.rows_per_cta && warp < nwarps; row += nwarps) {
                    float* pr = norm_s + row * words;
                    float t = lane < nwr ? pr[nwr * 32 + lane] : 0.f;
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) t = __fadd_rn(t, __shfl_xor_sync(0xffffffffu, t, o));
                    if (lane == 0) pr[nwr * 32 + 32] = t;
                }
                __syncthreads();
                return part[nwr * 32 + 32];
            };
            if constexpr (is_ln<PRO>()) {
                const float mean = __fdiv_rn(row_sum(false), (float)p.K);
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                    if (PRO == PRO_LAYERNORM) v[i] = __fsub_rn(v[i], mean), v[i + 1] = __fsub_rn(v[i + 1], mean);     // pairs: spills
                    else {
                        const float2 d = __fadd2_rn(make_float2(v[i], v[i + 1]), make_float2(-mean, -mean));
                        v[i] = d.x, v[i + 1] = d.y;
                    }
                }
            }
            const float rstd = rsqrtf(__fadd_rn(__fdiv_rn(row_sum(true), (float)p.K), p.eps));
            const T* ms_p = reinterpret_cast<const T*>(p.mod_scale);
            const T* sh_p = reinterpret_cast<const T*>(p.mod_shift);
            // The common bf16 forms two values at a time, one packed conversion per rounding. 1 + scale is a bf16 addition: it
            // rounds once where the other forms round to f32 first, which makes no difference (the f32 sum is inexact only
            // beside a scale below 2^-16 or above 2^16, and neither comes near a tie of bf16). A scalar conversion runs on the
            // narrow conversion pipe; LN_MOD 4352 x 3072 37.2 us with scalar ones and 80 registers, 30.0 now.
            // (Not RMS rows beyond 16384 values: 1024 threads leave 64 registers, and both forms in one kernel spilled 268 bytes.)
            constexpr bool kPacked = sizeof(T) == 2 && (PRO == PRO_LN_MOD || (PRO == PRO_RMS && MAXT < 1024));
            if (kPacked && (PRO == PRO_LN_MOD ? ms_p != nullptr : ms_p == nullptr)) {
                const float2 rstd2 = make_float2(rstd, rstd);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    uint4 mw = make_uint4(0, 0, 0, 0), sw = mw;
                    float nw[8];
                    if (PRO == PRO_LN_MOD) mw = gload(reinterpret_cast<const uint4*>(ms_p + col + 8 * c)), sw = gload(reinterpret_cast<const uint4*>(sh_p + col + 8 * c));
                    else if (p.norm_w) load8v(p.norm_w + col + 8 * c, nw);
                    const uint32_t m4[4] = {mw.x, mw.y, mw.z, mw.w}, s4[4] = {sw.x, sw.y, sw.z, sw.w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        float* e = v + 8 * c + 2 * i;
                        float2 n = __fmul2_rn(make_float2(e[0], e[1]), rstd2);
                        if (PRO == PRO_LN_MOD) {
                            const __nv_bfloat162 a = __hadd2(__floats2bfloat162_rn(1.f, 1.f), *reinterpret_cast<const __nv_bfloat162*>(&m4[i]));
                            n = __ffma2_rn(bf16x2_f(__floats2bfloat162_rn(n.x, n.y)), bf16x2_f(a),
                                           make_float2(__uint_as_float(s4[i] << 16), __uint_as_float(s4[i] & 0xffff0000u)));
                        } else if (p.norm_w) {
                            n = __fmul2_rn(n, make_float2(nw[2 * i], nw[2 * i + 1]));
                        }
                        n = bf16x2_f(__floats2bfloat162_rn(n.x, n.y));
                        e[0] = n.x, e[1] = n.y;
                    }
                }
            } else
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                float ms[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, sh[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, nw[8], nb[8];
                if (ms_p) load8v(ms_p + col + 8 * c, ms), load8v(sh_p + col + 8 * c, sh);
                const bool has_w = p.norm_w != nullptr;
                if (has_w) load8v(p.norm_w + col + 8 * c, nw);
                if (PRO == PRO_LN_AFFINE) load8v(p.norm_b + col + 8 * c, nb);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    float n = __fmul_rn(v[8 * c + j], rstd);
                    if (PRO == PRO_ADALN) {          // one rounding
                        n = rnd<T>(__fmaf_rn(n, __fadd_rn(1.f, ms[j]), sh[j]));
                    } else if (PRO == PRO_LN_MOD) {  // one rounding after the norm, one after the multiply-add
                        n = rnd<T>(__fmaf_rn(rnd<T>(n), rnd<T>(__fadd_rn(1.f, ms[j])), sh[j]));
                    } else if (PRO == PRO_LN_AFFINE) {
                        n = rnd<T>(__fmaf_rn(n, nw[j], nb[j]));
                    } else {                          // RMS, LAYERNORM: every step rounded
                        if (has_w) n = __fmul_rn(n, nw[j]);
                        n = rnd<T>(n);
                        if (ms_p) {
                            const float a = rnd<T>(__fadd_rn(1.f, ms[j]));
                            // f32 rows: nothing rounds between the product and the sum, and whether they fuse into one
                            // multiply-add is the compiler's choice. In the reference as nvcc 12.9 builds it, LAYERNORM
                            // fuses everywhere and RMS only in the last of its four unrolled group iterations (found by
                            // comparing outputs); that build is what these results are pinned to.
                            if (sizeof(T) == 4 && (PRO == PRO_LAYERNORM || rgi == 3)) n = __fmaf_rn(a, n, sh[j]);
                            else n = rnd<T>(__fadd_rn(rnd<T>(__fmul_rn(a, n)), sh[j]));
                        }
                    }
                    v[8 * c + j] = n;
                }
            }
        }

        float2 P[16];
        if (rotate) {
            // stages 0, 1 on the lane's two runs of 16, packed as (element i, element i + 16)
#pragma unroll
            for (int i = 0; i < 16; ++i) P[i] = make_float2(v[i], v[i + 16]);
            two_stages(P);
            // transpose inside the group: lane t8 wrote elements 32 t8 + i, now takes (2 t8, 2 t8 + 1) + 16 r
            float* we = tbuf_w + tpad(t8 << 5) + tsw;     // even columns go one word up in a swapping team,
            float* wo = tbuf_w + tpad(t8 << 5) - tsw;     // odd columns one word down: column i ^ 1
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                float* w = (i & 1) ? wo : we;
                w[i] = P[i].x;
                w[16 + i] = P[i].y;   // element 32 t8 + 16 + i: same 32-run, no pad in between
            }
            __syncwarp(wmask);
#pragma unroll
            for (int r = 0; r < 16; ++r) P[r] = *reinterpret_cast<const float2*>(tbuf_w + tpad(2 * t8 + 16 * r));
            two_stages(P);   // index bits 4-7 = r; in a swapping team .x is the odd element of the pair
            __syncwarp(wmask);
        } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) P[i] = make_float2(v[2 * i], v[2 * i + 1]);   // natural order
        }

        if (p.out_f) {   // gpu_rotate_rows_f32: always rotated, so P holds (2 t8, 2 t8 + 1) + 16 r
            if (live) {
                float* o = p.out_f + m * (int64_t)p.K + (grp << 8) + 2 * t8;
#pragma unroll
                for (int r = 0; r < 16; ++r) *reinterpret_cast<float2*>(o + 16 * r) = tsw ? make_float2(P[r].y, P[r].x) : P[r];
            }
            continue;
        }

        // This thread's maximum. The three-input form propagates a NaN, which the reference's fmaxf drops: a thread that
        // meets one recomputes its maximum without it and takes the exact division below.
        float amax = 0.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) amax = max3_abs_nan(amax, P[i].x, P[i].y);
        const bool has_nan = amax != amax;
        if (has_nan) {
            amax = 0.f;
#pragma unroll
            for (int i = 0; i < 16; ++i) amax = fmaxf(amax, fmaxf(fabsf(P[i].x), fabsf(P[i].y)));
        }
        // the group's 8 lanes first, then one shared-memory atomic per group (non-negative floats order as integers)
        amax = fmaxf(amax, __shfl_xor_sync(wmask, amax, 1));
        amax = fmaxf(amax, __shfl_xor_sync(wmask, amax, 2));
        amax = fmaxf(amax, __shfl_xor_sync(wmask, amax, 4));
        unsigned* slot = amax_s + (it % 3) * p.rows_per_cta + rloc;
        if (t8 == 0) atomicMax(slot, __float_as_uint(amax));
        __syncthreads();
        amax = __uint_as_float(*slot);
        amax_s[((it + 2) % 3) * p.rows_per_cta + rloc] = 0u;   // next use is two barriers away, last use one barrier back
        if (p.amax_out) {
            if (live && tin == 0) p.amax_out[m] = amax;
            continue;
        }
        if (p.amax_in) amax = p.amax_in[m];

        const float scale = fmaxf(fminf(amax, finite_max<T>()) * (1.f / 127.f), 1.0e-30f);
        if (live && tin == 0) p.scales[m] = scale;
        const float st = rnd<T>(scale);
        // rows holding an infinity, and threads holding a NaN, keep the IEEE division and the exact clamp
        const bool fast = sizeof(T) == 2 && amax <= FLT_MAX && !has_nan;
        const float rcp = fast ? __frcp_rn(st) : 0.f;
        uint32_t c16[16];
        if (fast) {      // one branch for the row, not one per pair
#pragma unroll
            for (int i = 0; i < 16; ++i) c16[i] = quant2<T>(P[i], st, rcp, true);
        } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) c16[i] = quant2<T>(P[i], st, rcp, false);
        }
        int8_t* q = p.q + m * (int64_t)p.K + col;
        if (rotate) {
            // codes of (2 t8, 2 t8 + 1) + 16 r back through the group's buffer, so each lane stores 32 contiguous bytes
            uint16_t* cb = reinterpret_cast<uint16_t*>(tbuf);
            const uint32_t order = tsw ? 0x3201u : 0x3210u;   // a swapping team puts its two codes back in element order
#pragma unroll
            for (int r = 0; r < 16; ++r) cb[t8 + 8 * r] = (uint16_t)__byte_perm(c16[r], 0u, order);
            __syncwarp(wmask);
            const uint4 lo = reinterpret_cast<const uint4*>(tbuf)[2 * t8], hi = reinterpret_cast<const uint4*>(tbuf)[2 * t8 + 1];
            __syncwarp(wmask);
            if (live) {
                reinterpret_cast<uint4*>(q)[0] = lo;
                reinterpret_cast<uint4*>(q)[1] = hi;
            }
        } else if (live) {
            uint32_t w[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) w[i] = (c16[2 * i] & 0xffffu) | (c16[2 * i + 1] << 16);
            reinterpret_cast<uint4*>(q)[0] = make_uint4(w[0], w[1], w[2], w[3]);
            reinterpret_cast<uint4*>(q)[1] = make_uint4(w[4], w[5], w[6], w[7]);
        }
    }
}

// ---- fp16 (SD / SDXL) flavour ------------------------------------------------------------------------------------------
// The reference's fp16 row quantizer (csrc/sd.cu:578-597) differs from the one above in its rounding points: values are
// rounded to half after the rotation, the row maximum is taken over the rounded values, scale = max(mx, 1e-30) / 127 is
// a division, the divisor is half(scale) unless that underflows, and q = clamp(rint(half(half(v) / st))). Rotation groups
// are 256 (four stages) or 64 (three). Same thread layout as above (32 consecutive elements per lane): 256-groups go
// through the same conflict-free transposition; a 64-group is two neighbouring lanes, whose third stage is one exchange
// of registers. The division is a reciprocal multiply with one Newton step: the exact quotient of two 11-bit significands
// is never on a half rounding boundary and at least 2^-23 (relative) away from one, and the refined product is within
// 2^-24 of it, so both round to the same half (tests/test_quant_division.py enumerates the significand pairs).
//
// SRC: where a row comes from. SDQ_ROWS reads it as it lies; the other sources compute it as the reference kernel that would
// have written it in half does (csrc/sd.cu:611-724: LayerNorm, GEGLU, head un-padding, GroupNorm without SiLU). They run as a
// first phase in which consecutive lanes hold consecutive 16-byte pieces (eight values), so that rows, gates and per-column
// vectors are read coalesced and each once, and leave the rows in shared memory as half, from where the lanes pick up their
// 32 values. A row at a time in shared memory as floats, one value per thread and step, was bound by its instruction count:
// 8192 x 640 LayerNorm 46.8 us, GroupNorm 60.9 with its statistics, GEGLU 8192 x 2560 114; this form takes 12.2, 24.7 and 47.7.
// LayerNorm statistics in the reference's order of additions: there 256 threads hold the row, thread t the elements t, t + 256,
// ... one after the other, then a xor-shuffle tree over the lanes of each warp and another over the eight warps. Here one
// warp holds a row, lane l the values 8 l .. 8 l + 7 of each run of 256, so the chains over the runs are the lane's own eight
// accumulators, and the trees run over lane bits 1, 0 and index bits 2, 1, 0 (the lanes of a warp there), then over lane bits
// 4, 3, 2 (the warps).
__device__ __forceinline__ float sd_tree256(float (&a)[8]) {
#pragma unroll
    for (int o = 2; o >= 1; o >>= 1) {
#pragma unroll
        for (int i = 0; i < 8; ++i) a[i] = __fadd_rn(a[i], __shfl_xor_sync(0xffffffffu, a[i], o));
    }
    float t = __fadd_rn(__fadd_rn(__fadd_rn(a[0], a[4]), __fadd_rn(a[2], a[6])), __fadd_rn(__fadd_rn(a[1], a[5]), __fadd_rn(a[3], a[7])));
#pragma unroll
    for (int o = 16; o >= 4; o >>= 1) t = __fadd_rn(t, __shfl_xor_sync(0xffffffffu, t, o));
    return t;
}
// 16-byte piece c of a row in shared memory sits at piece c ^ ((c >> 2) & 7): pieces in order (phase one) and pieces
// 4 t + k over lanes t (phase two) are both free of bank conflicts. Rows are padded to whole blocks of eight pieces.
__device__ __forceinline__ int sd_piece(int c) { return c ^ ((c >> 2) & 7); }
__device__ __forceinline__ void unpack_half8(const uint4 u, float (&v)[8]) {
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
        v[2 * i] = f.x, v[2 * i + 1] = f.y;
    }
}
__device__ __forceinline__ uint4 pack_half8(const float (&v)[8]) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const __half2 h = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
        w[i] = *reinterpret_cast<const uint32_t*>(&h);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// Piece i = threadIdx.x, threadIdx.x + blockDim.x, ... of the CTA's rows as (row, piece of the row): one division at the start
// instead of one per piece.
struct SdPieces {
    int r, c, dr, dc, pieces;
    __device__ __forceinline__ explicit SdPieces(int n) : pieces(n) {
        r = (int)threadIdx.x / n, c = (int)threadIdx.x - r * n;
        dr = (int)blockDim.x / n, dc = (int)blockDim.x - dr * n;
    }
    __device__ __forceinline__ void next() {
        r += dr, c += dc;
        if (c >= pieces) c -= pieces, ++r;
    }
};
template <int SRC>
__device__ __forceinline__ void sd_source_rows(const SdSrc& s, uint4* row_s, int pitch, float2* stat, int64_t m0, int live_rows, int K) {
    const int pieces = K >> 3, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    if constexpr (SRC == SDQ_LN) {
        // Up to 1280 values a warp holds its row's pieces in registers from the load to the normalised half (through shared memory, as longer rows
        // go, each of the three passes reads them again behind a barrier: 8192 x 640 14.0 us, now 12.1; 2048 x 1280 9.5, now 8.8).
        constexpr int kRegPieces = 5;
        if (pieces <= 32 * kRegPieces) {
            if (warp >= nwarps) return;      // whole warps only
            for (int r = warp; r < live_rows; r += nwarps) {
                const uint4* in = reinterpret_cast<const uint4*>(s.x + (m0 + r) * s.x_stride) + lane;
                uint4 u[kRegPieces];
                float a[8], e[8];
#pragma unroll
                for (int i = 0; i < kRegPieces; ++i)
                    if (lane + 32 * i < pieces) u[i] = gload(in + 32 * i);
#pragma unroll
                for (int j = 0; j < 8; ++j) a[j] = 0.f;
#pragma unroll
                for (int i = 0; i < kRegPieces; ++i) {
                    if (lane + 32 * i >= pieces) break;
                    unpack_half8(u[i], e);
#pragma unroll
                    for (int j = 0; j < 8; ++j) a[j] = __fadd_rn(a[j], e[j]);
                }
                const float mean = __fdiv_rn(sd_tree256(a), (float)K);
#pragma unroll
                for (int j = 0; j < 8; ++j) a[j] = 0.f;
#pragma unroll
                for (int i = 0; i < kRegPieces; ++i) {
                    if (lane + 32 * i >= pieces) break;
                    unpack_half8(u[i], e);
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const float d = __fsub_rn(e[j], mean);
                        a[j] = __fmaf_rn(d, d, a[j]);
                    }
                }
                const float rstd = rsqrtf(__fadd_rn(__fdiv_rn(sd_tree256(a), (float)K), s.eps));
#pragma unroll
                for (int i = 0; i < kRegPieces; ++i) {
                    const int c = lane + 32 * i;
                    if (c >= pieces) break;
                    float w[8], b[8];
                    load8v(s.w + 8 * c, w), load8v(s.b + 8 * c, b);
                    unpack_half8(u[i], e);
#pragma unroll
                    for (int j = 0; j < 8; j += 2) {
                        const float2 d = __fmul2_rn(__fadd2_rn(make_float2(e[j], e[j + 1]), make_float2(-mean, -mean)), make_float2(rstd, rstd));
                        const float2 n = __ffma2_rn(d, make_float2(w[j], w[j + 1]), make_float2(b[j], b[j + 1]));
                        e[j] = n.x, e[j + 1] = n.y;
                    }
                    row_s[r * pitch + sd_piece(c)] = pack_half8(e);
                }
            }
            return;
        }
        // the rows as they lie first, all of them in flight together
        for (SdPieces i(pieces); i.r < live_rows; i.next()) {
            const int r = i.r, c = i.c;
            row_s[r * pitch + sd_piece(c)] = gload(reinterpret_cast<const uint4*>(s.x + (m0 + r) * s.x_stride) + c);
        }
        __syncthreads();
        if (warp < nwarps)       // whole warps only
            for (int r = warp; r < live_rows; r += nwarps) {
                uint4* row = row_s + r * pitch;
                float a[8], e[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) a[i] = 0.f;
                for (int c = lane; c < pieces; c += 32) {
                    unpack_half8(row[sd_piece(c)], e);
#pragma unroll
                    for (int i = 0; i < 8; ++i) a[i] = __fadd_rn(a[i], e[i]);
                }
                const float mean = __fdiv_rn(sd_tree256(a), (float)K);
#pragma unroll
                for (int i = 0; i < 8; ++i) a[i] = 0.f;
                for (int c = lane; c < pieces; c += 32) {
                    unpack_half8(row[sd_piece(c)], e);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float d = __fsub_rn(e[i], mean);
                        a[i] = __fmaf_rn(d, d, a[i]);
                    }
                }
                const float rstd = rsqrtf(__fadd_rn(__fdiv_rn(sd_tree256(a), (float)K), s.eps));
                for (int c = lane; c < pieces; c += 32) {
                    float w[8], b[8];
                    load8v(s.w + 8 * c, w), load8v(s.b + 8 * c, b);
                    unpack_half8(row[sd_piece(c)], e);
#pragma unroll
                    for (int i = 0; i < 8; ++i) e[i] = __fmaf_rn(__fmul_rn(__fsub_rn(e[i], mean), rstd), w[i], b[i]);
                    row[sd_piece(c)] = pack_half8(e);
                }
            }
    } else if constexpr (SRC == SDQ_GN) {
        // mean and reciprocal deviation of this image's groups (csrc/sd.cu:198-205), once per CTA
        const int n = (int)(m0 / s.P);
        for (int g = threadIdx.x; g < s.groups; g += blockDim.x) {
            const double su = s.sums[(n * s.groups + g) * 2], sq = s.sums[(n * s.groups + g) * 2 + 1];
            const double mean = su / s.cnt;
            const double var = fmax(fma(-mean, mean, sq / s.cnt), 0.0);
            stat[g] = make_float2((float)mean, (float)(1.0 / sqrt(var + (double)s.eps)));
        }
        __syncthreads();
        const int per = K / s.groups;
        for (SdPieces i(pieces); i.r < live_rows; i.next()) {
            const int r = i.r, c = i.c;
            float e[8], w[8], b[8];
            unpack_half8(gload(reinterpret_cast<const uint4*>(s.x + (m0 + r) * (int64_t)K) + c), e);
            load8v(s.w + 8 * c, w), load8v(s.b + 8 * c, b);
            int g = (8 * c) / per, left = per - (8 * c - g * per);      // values of the group from here on
            float2 st = stat[g];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (left == 0) st = stat[++g], left = per;
                --left;
                e[j] = __fmaf_rn(__fmul_rn(__fsub_rn(e[j], st.x), st.y), w[j], b[j]);
            }
            row_s[r * pitch + sd_piece(c)] = pack_half8(e);
        }
    } else if constexpr (SRC == SDQ_GEGLU) {
        for (SdPieces i(pieces); i.r < live_rows; i.next()) {
            const int r = i.r, c = i.c;
            const uint4* in = reinterpret_cast<const uint4*>(s.x + (m0 + r) * 2 * (int64_t)K);
            float e[8], g[8];
            unpack_half8(gload(in + c), e), unpack_half8(gload(in + pieces + c), g);
#pragma unroll
            for (int j = 0; j < 8; ++j) e[j] = __fmul_rn(e[j], rnd<half>(gelu_f(g[j])));
            row_s[r * pitch + sd_piece(c)] = pack_half8(e);
        }
    } else if constexpr (SRC == SDQ_UNPAD) {
        for (SdPieces i(pieces); i.r < live_rows; i.next()) {
            const int r = i.r, c = i.c, h = (8 * c) / s.d;      // d % 8 == 0: a piece lies inside one head
            row_s[r * pitch + sd_piece(c)] =
                gload(reinterpret_cast<const uint4*>(s.x + (m0 + r) * (int64_t)s.heads * s.dp + (int64_t)h * s.dp + (8 * c - h * s.d)));
        }
    }
}

// Up to 288 threads (rows up to 9216 values) the kernel is held to 56 registers, seven CTAs of 160 threads per SM instead of
// six: 8192 rows of 640 values are 1024 such CTAs, which six per SM take in two rounds, the second an eighth full.
// In a chain of launches 8192 x 640: rows as they lie 7.6 -> 6.0 us.
constexpr int kSdThreads = 288;
template <int ROT, int SRC, int MAXT, bool EARLY>
__global__ void __launch_bounds__(MAXT, MAXT <= kSdThreads ? 4 : 1) sd_quant_fast_kernel(const SdSrc s, int8_t* q, float* scales, int M,
                                                            int K, int tpr, int rows, uint32_t off_amax, uint32_t off_rows, int early) {
    extern __shared__ __align__(128) uint8_t smem[];
    const unsigned wmask = __activemask();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int team = lane >> 3, tsw = team & 1, t8 = lane & 7;
    float* tbuf = reinterpret_cast<float*>(smem) + warp * kWarpWords + team * kGroupWords + 4 * (team >> 1);
    float* tbuf_w = tbuf - 2 * (team >> 1);
    unsigned* amax_s = reinterpret_cast<unsigned*>(smem + off_amax);
    for (int i = threadIdx.x; i < rows; i += blockDim.x) amax_s[i] = 0u;
    pdl_wait();
    // rows of this CTA; GroupNorm's belong to one image (blockIdx.y), so that one set of statistics serves the CTA
    const int64_t limit = SRC == SDQ_GN ? (int64_t)(blockIdx.y + 1) * s.P : M;
    const int64_t m0 = (SRC == SDQ_GN ? (int64_t)blockIdx.y * s.P : 0) + (int64_t)blockIdx.x * rows;
    // threads beyond the rows' (they help with the source only) and those of rows past the end recompute the last row and store nothing
    const int piece = threadIdx.x / tpr, tin = threadIdx.x - piece * tpr, rloc = SRC == SDQ_ROWS ? piece : min(piece, rows - 1);
    const int64_t m_raw = m0 + rloc;
    const bool live = (SRC == SDQ_ROWS || piece < rows) && m_raw < limit;
    const int64_t m = SRC == SDQ_ROWS ? (live ? m_raw : limit - 1) : 0;
    const int rl = (int)min((int64_t)rloc, limit - 1 - m0);      // the row it works on; its own where it has one
    float v[32];
    if constexpr (SRC == SDQ_ROWS) {
        __syncthreads();
        const uint4* r = reinterpret_cast<const uint4*>(s.x + m * s.x_stride) + 4 * tin;
#pragma unroll
        for (int c = 0; c < 4; ++c) unpack_half8(gload(r + c), *reinterpret_cast<float(*)[8]>(v + 8 * c));
    } else {
        uint4* row_s = reinterpret_cast<uint4*>(smem + off_rows);
        const int pitch = ((K >> 3) + 7) & ~7;
        sd_source_rows<SRC>(s, row_s, pitch, reinterpret_cast<float2*>(amax_s + ((rows + 1) & ~1)), m0, (int)min((int64_t)rows, limit - m0), K);
        __syncthreads();
        const uint4* r = row_s + rl * pitch;
#pragma unroll
        for (int c = 0; c < 4; ++c) unpack_half8(r[sd_piece(4 * tin + c)], *reinterpret_cast<float(*)[8]>(v + 8 * c));
    }
    if (EARLY && early) pdl_trigger();      // a kernel of its own where the rows are values at once: the branch there cost the others 3 %
    float2 P[16];
    if (ROT) {
#pragma unroll
        for (int i = 0; i < 16; ++i) P[i] = make_float2(v[i], v[i + 16]);
        two_stages<false>(P);                           // index bits 0-3
    } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) P[i] = make_float2(v[2 * i], v[2 * i + 1]);
    }
    if (ROT == 256) {
        float* we = tbuf_w + tpad(t8 << 5) + tsw;
        float* wo = tbuf_w + tpad(t8 << 5) - tsw;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            float* w = (i & 1) ? wo : we;
            w[i] = P[i].x;
            w[16 + i] = P[i].y;
        }
        __syncwarp(wmask);
#pragma unroll
        for (int rr = 0; rr < 16; ++rr) P[rr] = *reinterpret_cast<const float2*>(tbuf_w + tpad(2 * t8 + 16 * rr));
        two_stages<false>(P);                           // index bits 4-7
        __syncwarp(wmask);
    } else if (ROT == 64) {
        // third stage, index bits 4 and 5: bit 4 is the pair's half, bit 5 the lane's parity. The even lane holds x0, x1
        // and computes outputs 0 and 1 of the block, the odd lane holds x2, x3 and computes outputs 2 and 3.
        const bool even = (lane & 1) == 0;
        const float sg = even ? 1.f : -1.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const float ox = __shfl_xor_sync(wmask, P[i].x, 1), oy = __shfl_xor_sync(wmask, P[i].y, 1);
            const float x0 = even ? P[i].x : ox, x1 = even ? P[i].y : oy, x2 = even ? ox : P[i].x, x3 = even ? oy : P[i].y;
            const float sd = __fmaf_rn(x1, sg, x0);                                   // x0 + x1 (even) or x0 - x1 (odd)
            const float rx = __fmaf_rn(x3, -sg, __fadd_rn(sd, x2));                   // (sd + x2) - x3   or (sd + x2) + x3
            const float ry = __fadd_rn(__fmaf_rn(even ? x2 : sd, -1.f, even ? sd : x2), x3);   // (sd - x2) + x3 or (-sd + x2) + x3
            P[i] = make_float2(rx, ry);
        }
    }
    // The stages' halvings come as one multiplication here. For halves that is exact and the same: the sums stay below 2^16 * 256,
    // nothing is small enough to underflow, and scaling by a power of two moves no rounding.
    constexpr float kScale = ROT == 256 ? 0.0625f : 0.125f;
    // round to half; the row maximum is over the rounded values (the NaN-propagating form flags threads that hold one)
    float amax = 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        if (ROT) P[i] = __fmul2_rn(P[i], make_float2(kScale, kScale));
        P[i] = __half22float2(__floats2half2_rn(P[i].x, P[i].y));
        amax = max3_abs_nan(amax, P[i].x, P[i].y);
    }
    const bool has_nan = amax != amax;
    if (has_nan) {
        amax = 0.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) amax = fmaxf(amax, fmaxf(fabsf(P[i].x), fabsf(P[i].y)));
    }
    if ((tpr & 7) == 0) {
        amax = fmaxf(amax, __shfl_xor_sync(wmask, amax, 1));
        amax = fmaxf(amax, __shfl_xor_sync(wmask, amax, 2));
        amax = fmaxf(amax, __shfl_xor_sync(wmask, amax, 4));
        if (t8 == 0) atomicMax(amax_s + rloc, __float_as_uint(amax));
    } else {
        atomicMax(amax_s + rloc, __float_as_uint(amax));
    }
    __syncthreads();
    pdl_trigger();
    const float mx = __uint_as_float(amax_s[rloc]);
    const float scale = __fdiv_rn(fmaxf(mx, 1e-30f), 127.f);
    if (live && tin == 0) scales[m_raw] = scale;
    const float sh16 = rnd<half>(scale);
    const float st = sh16 > 0.f ? sh16 : scale;          // a scale below half's range divides in float
    const bool fast = sh16 > 0.f && mx <= 65504.f && !has_nan;
    uint32_t c16[16];
    if (fast) {
        const float rcp = __frcp_rn(st);
        const float2 rcp2 = make_float2(rcp, rcp), nst2 = make_float2(-st, -st), magic = make_float2(12582912.f, 12582912.f);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const float2 q0 = __fmul2_rn(P[i], rcp2);
            const float2 t = __ffma2_rn(__ffma2_rn(q0, nst2, P[i]), rcp2, q0);
            const float2 th = __half22float2(__floats2half2_rn(t.x, t.y));
            const float2 u = __fadd2_rn(th, magic);
            const int n0 = (int)__float_as_uint(u.x) - 0x4B400000, n1 = (int)__float_as_uint(u.y) - 0x4B400000;
            asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, 0;" : "=r"(c16[i]) : "r"(n1), "r"(n0));
        }
    } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int qx = clamp_rint_i8(rnd<half>(__fdiv_rn(P[i].x, st)), -128.f), qy = clamp_rint_i8(rnd<half>(__fdiv_rn(P[i].y, st)), -128.f);
            c16[i] = (uint32_t)(qx & 0xff) | ((uint32_t)(qy & 0xff) << 8);
        }
    }
    int8_t* qr = q + m_raw * K + tin * 32;              // of live rows only
    if (ROT == 256) {
        uint16_t* cb = reinterpret_cast<uint16_t*>(tbuf);
        const uint32_t order = tsw ? 0x3201u : 0x3210u;
#pragma unroll
        for (int rr = 0; rr < 16; ++rr) cb[t8 + 8 * rr] = (uint16_t)__byte_perm(c16[rr], 0u, order);
        __syncwarp(wmask);
        const uint4 lo = reinterpret_cast<const uint4*>(tbuf)[2 * t8], hi = reinterpret_cast<const uint4*>(tbuf)[2 * t8 + 1];
        if (live) {
            reinterpret_cast<uint4*>(qr)[0] = lo;
            reinterpret_cast<uint4*>(qr)[1] = hi;
        }
    } else if (live) {
        uint32_t w[8];
        if (ROT == 64) {      // c16[i] = codes of elements (i, i + 16)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t a = __byte_perm(c16[4 * j], c16[4 * j + 1], 0x5140), b = __byte_perm(c16[4 * j + 2], c16[4 * j + 3], 0x5140);
                w[j] = __byte_perm(a, b, 0x5410);          // bytes: codes of elements 4j .. 4j+3
                w[4 + j] = __byte_perm(a, b, 0x7632);      // and of elements 16+4j .. 16+4j+3
            }
        } else {              // c16[i] = codes of elements (2i, 2i + 1)
#pragma unroll
            for (int i = 0; i < 8; ++i) w[i] = (c16[2 * i] & 0xffffu) | (c16[2 * i + 1] << 16);
        }
        reinterpret_cast<uint4*>(qr)[0] = make_uint4(w[0], w[1], w[2], w[3]);
        reinterpret_cast<uint4*>(qr)[1] = make_uint4(w[4], w[5], w[6], w[7]);
    }
}

// ---- host side ------------------------------------------------------------------------------------------------
struct LutState {
    std::mutex mu;
    bool launched[LUT_COUNT] = {};
    bool done[LUT_COUNT] = {};
    cudaEvent_t ev[LUT_COUNT] = {};
};
LutState g_lut_state[64];

// Makes table `which` of the current device usable by work enqueued on `st` afterwards. The first call per device
// and table launches the builder on `st` (so it should come before any stream capture); later calls on other
// streams are ordered behind it until it is known complete.
int ensure_lut(int which, cudaStream_t st) {
    int dev = 0;
    cudaGetDevice(&dev);
    LutState& s = g_lut_state[dev & 63];
    std::lock_guard<std::mutex> lk(s.mu);
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cap) != cudaSuccess) (void)cudaGetLastError();
    if (cap != cudaStreamCaptureStatusNone) {
        // While a graph is being captured neither event queries nor waits on outside events are allowed. A table
        // requested first inside a capture is built by the captured graph itself, every replay (idempotent); one
        // launched before is taken as complete: the warm-up call that launched it precedes the capture.
        if (!s.launched[which]) {
            build_lut_kernel<<<256, 256, 0, st>>>(which);
            KCHECK();
        }
        return 0;
    }
    if (!s.launched[which]) {
        build_lut_kernel<<<256, 256, 0, st>>>(which);
        KCHECK();
        cudaError_t e = cudaEventCreateWithFlags(&s.ev[which], cudaEventDisableTiming);
        if (e != cudaSuccess) return (int)e;
        e = cudaEventRecord(s.ev[which], st);
        if (e != cudaSuccess) return (int)e;
        s.launched[which] = true;
        return 0;
    }
    if (!s.done[which]) {
        if (cudaEventQuery(s.ev[which]) == cudaSuccess) s.done[which] = true;
        else {
            const cudaError_t e = cudaStreamWaitEvent(st, s.ev[which], 0);
            if (e != cudaSuccess) return (int)e;
        }
    }
    return 0;
}

}  // namespace

namespace {
int sm_count_of(int dev) {
    static int count[64];
    static std::mutex mu;
    std::lock_guard<std::mutex> lk(mu);
    int& c = count[dev & 63];
    if (c == 0) cudaDeviceGetAttribute(&c, cudaDevAttrMultiProcessorCount, dev);
    return c;
}

// A quantizer of few CTAs, each on an SM of its own, lets its successor in as soon as its rows are in (elementwise prologues: requested), before
// their rotation: the other SMs are idle, the successor's setup and whatever it may do ahead (the few-rows GEMM brings its weights to
// L2) run beside the rest, and no CTA of the quantizer is left that could land badly. The adaLN linear 1 x 3072 -> 18432 with its
// quantizer: 17.2 us, now 16.4. Right behind the wait the successor's CTAs and their prefetches compete with the quantizer's own loads: the
// W6A8 block of 64 rows (four quantizers of 64 CTAs) takes 121.5 us that way, 116.4 this. Up to seven SMs in eight: 125 CTAs and a GEMM (250 x 3072 -> 3072)
// 12.8 us, 12.9 without; 139 (1111 x 1024 -> 3072) 12.5 and 12.1, 140 (140 x 8192 -> 3072) 19.9 and 19.5, for what starts early finds no SM idle.
int early_trigger(int64_t ctas) {
    int dev = 0;
    cudaGetDevice(&dev);
    return ctas * 8 <= (int64_t)sm_count_of(dev) * 7;
}
template <int ROT, int SRC, int MAXT, bool EARLY = true>
int launch_sd_cfg(const SdSrc& s, int8_t* q, float* scales, int M, int K, dim3 grid, int threads, int rows, uint32_t smem, uint32_t off_amax,
                  uint32_t off_rows, cudaStream_t st) {
    const int early = early_trigger((int64_t)grid.x * grid.y);
    if constexpr (SRC == SDQ_ROWS && EARLY)
        if (!early) return launch_sd_cfg<ROT, SRC, MAXT, false>(s, q, scales, M, K, grid, threads, rows, smem, off_amax, off_rows, st);
    auto kern = sd_quant_fast_kernel<ROT, SRC, MAXT, EARLY>;
    if (smem > 48 * 1024) {
        static std::atomic<uint64_t> configured{0};
        int dev = 0;
        cudaGetDevice(&dev);
        const uint64_t bit = 1ull << (dev & 63);
        if (!(configured.load(std::memory_order_acquire) & bit)) {
            const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024);
            if (e != cudaSuccess) return (int)e;
            configured.fetch_or(bit, std::memory_order_release);
        }
    }
    return launch_pdl(kern, grid, threads, smem, st, s, q, scales, M, K, K / 32, rows, off_amax, off_rows, early);
}
template <int ROT, int SRC>
int launch_sd_fast(const SdSrc& s, int8_t* q, float* scales, int M, int K, cudaStream_t st) {
    const int tpr = K / 32;
    // whole rows and about 256 threads; a whole number of warps where that takes no more than 512
    int rows = 256 / tpr;
    if (rows < 1) rows = 1;
    if (rows * tpr < 32) rows = (32 + tpr - 1) / tpr;
    int even = 32;                                      // rows that make a whole number of warps
    while (even > 1 && (even / 2 * tpr) % 32 == 0) even /= 2;
    if (even * tpr <= kSdThreads || (SRC != SDQ_ROWS && even * tpr <= 512)) rows = rows / even > 0 ? rows / even * even : even;
    int threads = rows * tpr;
    if (SRC != SDQ_ROWS) {
        // Few rows: a row or as few as give every SM a CTA, and up to 256 threads for the source, which has a 16-byte piece of the
        // row for each (a warp per row for LayerNorm's sums). With the row counts above, 16 rows of 320 values kept one CTA
        // busy for 6.6 us (LayerNorm; GEGLU 3.8) where a CTA per row had taken 3.4 (2.6).
        int dev = 0;
        cudaGetDevice(&dev);
        const int sms = sm_count_of(dev), share = (M + sms - 1) / sms;
        if (share < rows) {
            rows = share;
            const int work = rows * (SRC == SDQ_LN && 4 * tpr < 32 ? 32 : 4 * tpr);
            threads = rows * tpr;
            if (threads < 256) threads = work < 256 ? (work > threads ? work : threads) : 256;
            threads = (threads + 31) & ~31;
        }
    }
    uint32_t off = ROT == 256 ? (uint32_t)((threads + 31) / 32) * kWarpWords * 4 : 0;
    const uint32_t off_amax = off;
    off += (uint32_t)((rows + 1) & ~1) * 4 + (SRC == SDQ_GN ? (uint32_t)s.groups * 8 : 0);
    off = (off + 127) & ~127u;
    const uint32_t off_rows = off;
    if (SRC != SDQ_ROWS) off += (uint32_t)rows * (((K >> 3) + 7) & ~7) * 16;
    const dim3 grid = SRC == SDQ_GN ? dim3((unsigned)((s.P + rows - 1) / rows), (unsigned)(M / s.P)) : dim3((unsigned)((M + rows - 1) / rows));
    if (threads <= kSdThreads) return launch_sd_cfg<ROT, SRC, kSdThreads>(s, q, scales, M, K, grid, threads, rows, off, off_amax, off_rows, st);
    return launch_sd_cfg<ROT, SRC, 512>(s, q, scales, M, K, grid, threads, rows, off, off_amax, off_rows, st);
}
template <int SRC>
int launch_sd_fast_rot(const SdSrc& s, int8_t* q, float* scales, int M, int K, int rotate, cudaStream_t st) {
    return rotate == 256 ? launch_sd_fast<256, SRC>(s, q, scales, M, K, st)
           : rotate == 64 ? launch_sd_fast<64, SRC>(s, q, scales, M, K, st) : launch_sd_fast<0, SRC>(s, q, scales, M, K, st);
}
}  // namespace

// The fp16 quantizers (gpu_sd_*quant_rows) through the register kernel above; false when the shape is not one it takes (the
// caller falls back): rows of whole 32-value pieces and rotation groups up to 16384 values, 16-byte aligned.
bool b200q::sd_quant_fast(int src, const SdSrc& s, int8_t* q, float* scales, int M, int K, int rotate, cudaStream_t st, int* rc) {
    if (K % 32 || K > 16384 || (rotate == 64 && K % 64) || (rotate == 256 && K % 256) || (rotate != 0 && rotate != 64 && rotate != 256))
        return false;
    if (((uintptr_t)s.x | (uintptr_t)q) & 15) return false;
    switch (src) {
        case SDQ_ROWS:
            if (s.x_stride & 7) return false;
            *rc = launch_sd_fast_rot<SDQ_ROWS>(s, q, scales, M, K, rotate, st);
            return true;
        case SDQ_LN:
            if ((s.x_stride & 7) || (((uintptr_t)s.w | (uintptr_t)s.b) & 15)) return false;
            *rc = launch_sd_fast_rot<SDQ_LN>(s, q, scales, M, K, rotate, st);
            return true;
        case SDQ_GEGLU:
            *rc = launch_sd_fast_rot<SDQ_GEGLU>(s, q, scales, M, K, rotate, st);
            return true;
        case SDQ_UNPAD:
            if ((s.d & 7) || (s.dp & 7)) return false;
            *rc = launch_sd_fast_rot<SDQ_UNPAD>(s, q, scales, M, K, rotate, st);
            return true;
        case SDQ_GN:
            if ((((uintptr_t)s.w | (uintptr_t)s.b) & 15) || M / s.P > 65535) return false;
            *rc = launch_sd_fast_rot<SDQ_GN>(s, q, scales, M, K, rotate, st);
            return true;
        default: return false;
    }
}

// Reads and clears the quantizer's status word (a staging wait that ran out); used by gpu_kernels_status.
int b200q::quant_status_read_clear(int* out) {
    int v = 0;
    cudaError_t e = cudaMemcpyFromSymbol(&v, g_quant_status, sizeof(int));
    if (e != cudaSuccess) return (int)e;
    if (v != 0) {
        const int zero = 0;
        e = cudaMemcpyToSymbol(g_quant_status, &zero, sizeof(int));
        if (e != cudaSuccess) return (int)e;
    }
    *out = v;
    return 0;
}

// Device address of the bf16 -> bf16 table of a GEMM-epilogue activation (epilogue.cuh's Act codes), built on first use
// like the quantizer's own: the epilogue's out(act(out(v))) on bf16 outputs is a function of 16 bits.
int b200q::act_lut_ptr(int act, cudaStream_t st, const uint16_t** out) {
    const int which = act == 1 ? LUT_GELU_TANH : act == 2 ? LUT_SILU : act == 3 ? LUT_GELU : -1;
    if (which < 0) return -204;
    if (int rc = ensure_lut(which, st)) return rc;
    static const uint16_t* base[64];
    static std::mutex mu;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(mu);
    const uint16_t*& b = base[dev & 63];
    if (!b) {
        void* addr = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&addr, g_act_lut);
        if (e != cudaSuccess) return (int)e;
        b = reinterpret_cast<const uint16_t*>(addr);
    }
    *out = b + (size_t)which * 65536;
    return 0;
}

namespace {

// CTAs of one kernel instantiation that fit an SM at a given size: asked of the runtime once per (threads, smem).
struct OccCache {
    std::mutex mu;
    int threads[8] = {}, blocks[8] = {}, n = 0;
    size_t smem[8] = {};
};

// A kernel's limit of dynamic shared memory, raised once per device
template <typename Kern> int raise_smem(Kern kern, std::atomic<uint64_t>& configured, size_t smem) {
    if (smem <= 48 * 1024) return 0;
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = 1ull << (dev & 63);
    if (configured.load(std::memory_order_acquire) & bit) return 0;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e == cudaSuccess) configured.fetch_or(bit, std::memory_order_release);
    return (int)e;
}
template <typename T, int PRO, int MAXT, bool DIGITS = false>
int launch_direct(QuantArgs& p, int threads, size_t smem, cudaStream_t st) {
    static std::atomic<uint64_t> configured{0};
    auto kern = quant_direct_kernel<T, PRO, MAXT, DIGITS>;
    p.early = early_trigger(p.nblocks);
    if (int rc = raise_smem(kern, configured, smem)) return rc;
    return launch_pdl(kern, dim3(p.nblocks), threads, smem, st, p);
}
template <typename T, int PRO, int MAXT, bool DIGITS, int ROWS = 1>
int launch_norm_cfg(const QuantArgs& p, int threads, size_t smem, cudaStream_t st) {
    static std::atomic<uint64_t> configured{0};
    auto kern = quant_norm_kernel<T, PRO, MAXT, DIGITS, ROWS>;
    if (int rc = raise_smem(kern, configured, smem)) return rc;
    return launch_pdl(kern, dim3(p.nblocks), threads, smem, st, p);
}
// Rows of ceil(K / 1024) warps, about eight warps per CTA. Warps of four rows of 256 values or two of 512 from two CTAs an SM on: 2368 x 256 RMS takes
// 5.6 us with a row a warp, 2369 4.5 with four, 4736 6.6 and 5.3. On fewer rows more warps hide one another's latencies (1111 x 256: 4.0).
template <typename T, int PRO, bool DIGITS = false> int launch_norm(QuantArgs p, cudaStream_t st) {
    int dev = 0;
    cudaGetDevice(&dev);
    const int nwr = ((p.K >> 8) + 3) >> 2, per_warp = sizeof(T) == 2 && p.K <= 512 && p.M > 8 * 2 * sm_count_of(dev) ? 1024 / p.K : 1;
    const int rows = per_warp * (nwr >= 8 ? 1 : 8 / nwr), warps = rows / per_warp * nwr;
    p.tpr = nwr, p.rows_per_cta = rows, p.nblocks = (p.M + rows - 1) / rows;
    p.off_norm = (uint32_t)(warps * kWarpWords * 4);
    p.off_amax = p.off_norm + (per_warp > 1 ? 0 : rows * 64 * 4);
    p.early = early_trigger(p.nblocks);
    const size_t smem = p.off_amax + direct_words(rows, DIGITS) * 4;
    if constexpr (sizeof(T) == 2) {
        if (per_warp == 4) return launch_norm_cfg<T, PRO, 256, DIGITS, 4>(p, 32 * warps, smem, st);
        if (per_warp == 2) return launch_norm_cfg<T, PRO, 256, DIGITS, 2>(p, 32 * warps, smem, st);
    }
    return warps <= 8 ? launch_norm_cfg<T, PRO, 256, DIGITS>(p, 32 * warps, smem, st) : launch_norm_cfg<T, PRO, 1024, DIGITS>(p, 32 * warps, smem, st);
}

template <typename T, int PRO, int MAXT>
int launch_cfg(QuantArgs& p, int threads, size_t smem, bool persistent, cudaStream_t st) {
    auto kern = quant_rows_kernel<T, PRO, MAXT>;
    static std::atomic<uint64_t> configured{0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (smem > 48 * 1024) {
        const uint64_t bit = 1ull << (dev & 63);
        if (!(configured.load(std::memory_order_acquire) & bit)) {
            const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
            if (e != cudaSuccess) return (int)e;
            configured.fetch_or(bit, std::memory_order_release);
        }
    }
    int grid = p.nblocks;
    if (persistent) {
        static OccCache occ;
        int per_sm = 0;
        {
            std::lock_guard<std::mutex> lk(occ.mu);
            for (int i = 0; i < occ.n; ++i)
                if (occ.threads[i] == threads && occ.smem[i] == smem) per_sm = occ.blocks[i];
            if (!per_sm) {
                if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem) != cudaSuccess || per_sm < 1) {
                    (void)cudaGetLastError();
                    per_sm = 1;
                }
                const int slot = occ.n < 8 ? occ.n++ : 7;
                occ.threads[slot] = threads, occ.smem[slot] = smem, occ.blocks[slot] = per_sm;
            }
        }
        const int resident = per_sm * sm_count_of(dev);
        if (grid > resident) grid = resident;
    }
    return launch_pdl(kern, dim3(grid), threads, smem, st, p);
}

constexpr size_t kMaxSmem = 227 * 1024;


template <typename T, int PRO>
int launch_quant(QuantArgs& p, cudaStream_t st) {
    p.tpr = p.K / 32;
    if (p.tpr > 1024) return -2;  // the reference's limit: K <= 32768 (csrc/kernels.cu:264)
    if (p.M <= 0) return 0;
    // 16-byte loads and bulk copies: rows must start 16-byte aligned, as the reference's load8 requires too
    const uintptr_t mis = (uintptr_t)p.x | (uintptr_t)(p.x_stride * sizeof(T)) |
                          (PRO == PRO_GATE ? (uintptr_t)p.g | (uintptr_t)(p.g_stride * sizeof(T)) : 0) |
                          (has_aux<PRO>() && PRO != PRO_GATE ? (uintptr_t)(p.up_offset * sizeof(T)) : 0) | (uintptr_t)p.q |
                          (uintptr_t)p.out_f | (uintptr_t)p.digits;
    if (mis & 15) return -5;
    int lut = -1;
    if (sizeof(T) == 2 && (int64_t)p.M * p.K >= (1 << 20)) {
        lut = PRO == PRO_SILU || PRO == PRO_SWIGLU ? LUT_SILU : PRO == PRO_GELU ? LUT_GELU : PRO == PRO_GELU_TANH ? LUT_GELU_TANH
              : PRO == PRO_GATE ? LUT_SIGMOID : -1;
    }
    if (lut >= 0) {
        if (int rc = ensure_lut(lut, st)) return rc;
    }
    p.lut = lut;
    // CTA shape: whole rows, about 256 threads, at least one warp; any multiple of 8 threads up to 1024 works (the
    // last warp may be partial), so every K the reference accepts is served
    int rows = 256 / p.tpr;
    if (rows < 1) rows = 1;
    if (rows * p.tpr < 32) rows = (32 + p.tpr - 1) / p.tpr;
    p.rows_per_cta = rows;
    p.nblocks = (p.M + rows - 1) / rows;
    const int threads = rows * p.tpr;
    auto up = [](size_t v, size_t a) { return (v + a - 1) / a * a; };
    size_t off = (size_t)((threads + 31) / 32) * kWarpWords * 4;
    p.off_amax = (uint32_t)off, off += (size_t)(p.digits ? direct_words(rows, true) : 3 * rows) * 4;
    p.off_norm = (uint32_t)off, off += is_norm<PRO>() ? (size_t)rows * norm_words(p.K) * 4 : 0;
    off = up(off, 16);
    off = up(off, 8);
    p.off_bar = (uint32_t)off, off += 8;
    off = up(off, 128);
    p.off_stage = (uint32_t)off;
    const size_t stage_bytes = (size_t)rows * p.K * sizeof(T) * (has_aux<PRO>() ? 2 : 1);
    // Measured on B200 (M = 4352, K = 12288, bf16): without the rotation, persistent CTAs with the next block's rows in
    // flight through the staging buffer win (49 against 54 us); with it the kernel is bound by its arithmetic and the
    // transposition, not by waiting for HBM, and one block per CTA with direct loads is as fast or faster (74 against 78).
    p.staged = !p.rotate && !is_norm<PRO>() && off + stage_bytes <= kMaxSmem;
    const size_t smem = p.staged ? off + stage_bytes : off;
    if (smem > kMaxSmem) return -2;
    if constexpr (sizeof(T) == 4 && (PRO == PRO_PLAIN || PRO == PRO_SWIGLU)) {
        if (p.digits) return threads <= 256 ? launch_direct<T, PRO, 256, true>(p, threads, smem, st) : launch_direct<T, PRO, 1024, true>(p, threads, smem, st);
    }
    if constexpr (sizeof(T) == 4 && PRO == PRO_RMS) {
        if (p.digits) return launch_norm<T, PRO, true>(p, st);
    }
    const bool codes = p.rotate && !p.out_f && !p.digits && !p.amax_in && !p.amax_out;
    if constexpr (direct_threads<T, PRO>() > 0) {
        // Tabulated, GELU is SILU's kernel on another table; its own computes it. Both forms in one, erff beside the look-ups, spilled.
        constexpr int kPro = sizeof(T) == 2 && PRO == PRO_GELU ? PRO_SILU : PRO;
        if (codes && threads <= direct_threads<T, PRO>())
            return p.lut >= 0 ? launch_direct<T, kPro, direct_threads<T, PRO>()>(p, threads, smem, st) : launch_direct<T, PRO, direct_threads<T, PRO>()>(p, threads, smem, st);
    }
    if constexpr (sizeof(T) == 2 && is_norm<PRO>()) {
        if (codes) return launch_norm<T, PRO>(p, st);
    }
    if (threads > 512) return launch_cfg<T, PRO, 1024>(p, threads, smem, p.staged != 0, st);
    if (threads > 384) return launch_cfg<T, PRO, 512>(p, threads, smem, p.staged != 0, st);
    return launch_cfg<T, PRO, 384>(p, threads, smem, p.staged != 0, st);
}

template <typename T>
int dispatch_prologue(int prologue, QuantArgs& p, cudaStream_t st) {
    switch (prologue) {
        case PRO_PLAIN: return launch_quant<T, PRO_PLAIN>(p, st);
        case PRO_GATE: return launch_quant<T, PRO_GATE>(p, st);
        case PRO_SWIGLU: return launch_quant<T, PRO_SWIGLU>(p, st);
        case PRO_SILU: return launch_quant<T, PRO_SILU>(p, st);
        case PRO_GELU: return launch_quant<T, PRO_GELU>(p, st);
        case PRO_GELU_TANH: return launch_quant<T, PRO_GELU_TANH>(p, st);
        case PRO_SITU: return launch_quant<T, PRO_SITU>(p, st);
        case PRO_SITU_FAST: return launch_quant<T, PRO_SITU_FAST>(p, st);
        case PRO_RMS: return launch_quant<T, PRO_RMS>(p, st);
        case PRO_LAYERNORM: return launch_quant<T, PRO_LAYERNORM>(p, st);
        case PRO_LN_MOD: return launch_quant<T, PRO_LN_MOD>(p, st);
        case PRO_ADALN: return p.mod_scale && p.mod_shift ? launch_quant<T, PRO_ADALN>(p, st) : -3;
        // LN_AFFINE needs the bias that only gpu_quant_rows_b carries (the reference reads a null pointer there)
        case PRO_LN_AFFINE: return p.norm_w && p.norm_b ? launch_quant<T, PRO_LN_AFFINE>(p, st) : -3;
        default: return -3;
    }
}

}  // namespace

// Same contract as the reference's gpu_quant_rows (csrc/kernels.cu:271-298): K % 256 == 0 (-1), K <= 32768 (-2),
// known prologue (-3), dtype bf16 or f32 (-4); rows of x start 16-byte aligned.
GPU_API int gpu_quant_rows(int dtype, int prologue, const void* x, int64_t x_stride, const void* g, int64_t g_stride,
                           int64_t up_offset, const float* norm_w, float eps, const void* mod_scale, const void* mod_shift,
                           int8_t* q, float* scales, int M, int K, int rotate, void* stream) {
    if ((K % 256) != 0) return -1;
    QuantArgs p{x, x_stride, g, g_stride, up_offset, q, scales, nullptr, M, K, rotate, 0, 0, 0, -1, nullptr, nullptr,
                norm_w, nullptr, eps, mod_scale, mod_shift};
    if (dtype == DT_BF16) return dispatch_prologue<bf16>(prologue, p, (cudaStream_t)stream);
    if (dtype == DT_F32) return dispatch_prologue<float>(prologue, p, (cudaStream_t)stream);
    return -4;
}

// gpu_quant_rows with a LayerNorm bias (csrc/kernels.cu:301-314): bf16 only (-4), prologues LN_MOD and LN_AFFINE (-3).
GPU_API int gpu_quant_rows_b(int dtype, int prologue, const void* x, int64_t x_stride, const float* norm_w, const float* norm_b,
                             float eps, const void* mod_scale, const void* mod_shift, int8_t* q, float* scales, int M, int K,
                             int rotate, void* stream) {
    if ((K % 256) != 0) return -1;
    if (dtype != DT_BF16) return -4;
    if (prologue != PRO_LN_MOD && prologue != PRO_LN_AFFINE) return -3;
    QuantArgs p{x, x_stride, nullptr, 0, 0, q, scales, nullptr, M, K, rotate, 0, 0, 0, -1, nullptr, nullptr,
                norm_w, norm_b, eps, mod_scale, mod_shift};
    return dispatch_prologue<bf16>(prologue, p, (cudaStream_t)stream);
}

// Prologue + rotation, fp32 rows out (the weight-only int8 path's activation side; csrc/kernels.cu:316-327).
GPU_API int gpu_rotate_rows_f32(int prologue, const float* x, int64_t x_stride, int64_t up_offset, const float* norm_w,
                                float eps, float* out, int M, int K, void* stream) {
    if ((K % 256) != 0) return -1;
    QuantArgs p{x, x_stride, nullptr, 0, up_offset, nullptr, nullptr, out, M, K, 1, 0, 0, 0, -1, nullptr, nullptr,
                norm_w, nullptr, eps, nullptr, nullptr};
    switch (prologue) {
        case PRO_PLAIN: return launch_quant<float, PRO_PLAIN>(p, (cudaStream_t)stream);
        case PRO_RMS: return launch_quant<float, PRO_RMS>(p, (cudaStream_t)stream);
        case PRO_SWIGLU: return launch_quant<float, PRO_SWIGLU>(p, (cudaStream_t)stream);
        default: return -3;
    }
}

// The same with the rotated rows written as three 8-bit digits [3][M, K], a factor per row and, for spread rows, a shift per group
// [K / 256][M]: the activation side of the weight-only linear on the int8 tensor cores. The first CTA zeroes `nzero` words at `zero`.
int b200q::rotate_rows_digits(int prologue, const float* x, int64_t x_stride, int64_t up_offset, const float* norm_w, float eps,
                              int8_t* digits, float* factors, uint8_t* shifts, int* zero, int nzero, int M, int K, cudaStream_t st) {
    if ((K % 256) != 0) return -1;
    QuantArgs p{x, x_stride, nullptr, 0, up_offset, nullptr, factors, nullptr, M, K, 1, 0, 0, 0, -1, nullptr, nullptr,
                norm_w, nullptr, eps, nullptr, nullptr};
    p.digits = digits, p.shifts = shifts, p.zero = zero, p.nzero = nzero;
    switch (prologue) {
        case PRO_PLAIN: return launch_quant<float, PRO_PLAIN>(p, st);
        case PRO_RMS: return launch_quant<float, PRO_RMS>(p, st);
        case PRO_SWIGLU: return launch_quant<float, PRO_SWIGLU>(p, st);
        default: return -3;
    }
}

// New, for rows whose K columns are split across devices (row-parallel linears): the per-token scale must come from
// the maximum over the whole row, so quantization runs in two passes around a max-reduction between the devices.
//   pass 1  gpu_quant_rows_amax: prologue + rotation of the local columns, row maxima -> amax [M] (f32)
//   pass 2  gpu_quant_rows_scaled: the same, quantized with the given (reduced) maxima; `scales` receives the scale
// With the reduced maxima the codes equal the corresponding columns of the single-device result bit for bit.
GPU_API int gpu_quant_rows_amax(int dtype, int prologue, const void* x, int64_t x_stride, const void* g, int64_t g_stride,
                                int64_t up_offset, float* amax, int M, int K, int rotate, void* stream) {
    if ((K % 256) != 0) return -1;
    QuantArgs p{x, x_stride, g, g_stride, up_offset, nullptr, nullptr, nullptr, M, K, rotate, 0, 0, 0, -1, nullptr, amax};
    if (dtype == DT_BF16) return dispatch_prologue<bf16>(prologue, p, (cudaStream_t)stream);
    if (dtype == DT_F32) return dispatch_prologue<float>(prologue, p, (cudaStream_t)stream);
    return -4;
}
GPU_API int gpu_quant_rows_scaled(int dtype, int prologue, const void* x, int64_t x_stride, const void* g, int64_t g_stride,
                                  int64_t up_offset, const float* amax, int8_t* q, float* scales, int M, int K, int rotate,
                                  void* stream) {
    if ((K % 256) != 0) return -1;
    QuantArgs p{x, x_stride, g, g_stride, up_offset, q, scales, nullptr, M, K, rotate, 0, 0, 0, -1, amax, nullptr};
    if (dtype == DT_BF16) return dispatch_prologue<bf16>(prologue, p, (cudaStream_t)stream);
    if (dtype == DT_F32) return dispatch_prologue<float>(prologue, p, (cudaStream_t)stream);
    return -4;
}

// ---- second pass after a rotating GEMM epilogue -------------------------------------------------------------------------
// gpu_int8_gemm_act_rot leaves the rows rotated and rounded to bf16, and per row N / 64 partial maxima of the unrounded
// rotated values (sign bit: a NaN among them), stored part-major [N / 64, M]. What is left of the quantizer is the row
// maximum, the scale and one pass over the row: 2 bytes read and 1 written per element. A CTA takes 8 consecutive rows
// (whose partial maxima are 32 contiguous bytes per part), `wpr` warps per row; a lane converts 16 consecutive values per
// step.
namespace {
constexpr int kRotRows = 8;
__global__ void __launch_bounds__(512) quant_rotated_kernel(const bf16* xr, const float* parts,
                                                            int8_t* q, float* scales, int M, int K,
                                                            int P, int wpr) {
    __shared__ unsigned s_amax[kRotRows], s_flag[kRotRows];
    pdl_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int rloc = warp / wpr, seg = warp - rloc * wpr;
    const int64_t m0 = (int64_t)blockIdx.x * kRotRows, m = m0 + rloc;
    const bool live = m < M;
    const int per = K / wpr;
    const bf16* src = xr + m * (int64_t)K + (int64_t)seg * per;
    int8_t* dst = q + m * (int64_t)K + (int64_t)seg * per;
    if (threadIdx.x < kRotRows) s_amax[threadIdx.x] = 0u, s_flag[threadIdx.x] = 0u;
    // the first two steps' values are requested before the row's maximum is known: the partial maxima and the rows then
    // arrive together instead of one after the other
    uint4 a0, b0, a1, b1;
    a0 = b0 = a1 = b1 = make_uint4(0, 0, 0, 0);
    const int e0 = lane * 16;
    if (live && e0 < per) a0 = gload(reinterpret_cast<const uint4*>(src + e0)), b0 = gload(reinterpret_cast<const uint4*>(src + e0 + 8));
    if (live && e0 + 512 < per) a1 = gload(reinterpret_cast<const uint4*>(src + e0 + 512)), b1 = gload(reinterpret_cast<const uint4*>(src + e0 + 520));
    __syncthreads();
    // the 8 rows' partial maxima, 8 consecutive floats per part; non-negative floats order as integers
    for (int i = threadIdx.x; i < P * kRotRows; i += blockDim.x) {
        const int r = i & (kRotRows - 1);
        if (m0 + r < M) {
            const uint32_t u = __float_as_uint(gload(parts + (int64_t)(i >> 3) * M + m0 + r));
            atomicMax(&s_amax[r], u & 0x7fffffffu);
            if (u & 0x80000000u) s_flag[r] = 1u;
        }
    }
    __syncthreads();
    if (!live) return;
    const float amax = __uint_as_float(s_amax[rloc]);
    const uint32_t flag = s_flag[rloc];
    const float scale = fmaxf(fminf(amax, finite_max<bf16>()) * (1.f / 127.f), 1.0e-30f);
    if (seg == 0 && lane == 0) scales[m] = scale;
    const float st = rnd<bf16>(scale);
    // rows holding an infinity or a NaN keep the IEEE division and the exact clamp
    const bool fast = amax <= FLT_MAX && flag == 0;
    const float rcp = fast ? __frcp_rn(st) : 0.f;
    auto convert = [&](const uint4 a, const uint4 b, int e) {
        const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        uint32_t c[8];
        if (fast) {
#pragma unroll
            for (int i = 0; i < 8; ++i) c[i] = quant2_bf16_bits(w[i], rcp);
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i)
                c[i] = quant2<bf16>(make_float2(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xffff0000u)), st, 0.f, false);
        }
        *reinterpret_cast<uint4*>(dst + e) = make_uint4((c[0] & 0xffffu) | (c[1] << 16), (c[2] & 0xffffu) | (c[3] << 16),
                                                        (c[4] & 0xffffu) | (c[5] << 16), (c[6] & 0xffffu) | (c[7] << 16));
    };
    // two steps in flight: a step's values are replaced by those of the step after next before it is converted
#pragma unroll 1
    for (int e = e0; e < per; e += 1024) {
        uint4 a = a0, b = b0;
        if (e + 1024 < per) a0 = gload(reinterpret_cast<const uint4*>(src + e + 1024)), b0 = gload(reinterpret_cast<const uint4*>(src + e + 1032));
        convert(a, b, e);
        if (e + 512 < per) {
            a = a1, b = b1;
            if (e + 1536 < per) a1 = gload(reinterpret_cast<const uint4*>(src + e + 1536)), b1 = gload(reinterpret_cast<const uint4*>(src + e + 1544));
            convert(a, b, e + 512);
        }
    }
}
}  // namespace

// New: the quantizer's second pass on rows a rotating GEMM epilogue left (gpu_int8_gemm_act_rot): xr [M, K] bf16, rotated;
// amax_part [K / 64, M]; q [M, K] int8 and scales [M] as gpu_quant_rows(prologue = that activation, rotate = 1) gives them
// on the plain GEMM's output. K % 256 == 0 (-1); xr and q 16-byte aligned (-5).
GPU_API int gpu_quant_rows_rotated(const void* xr, const float* amax_part, int8_t* q, float* scales, int M, int K, void* stream) {
    if (K <= 0 || (K % 256) != 0) return -1;
    if (M <= 0) return 0;
    if ((((uintptr_t)xr | (uintptr_t)q) & 15) != 0) return -5;
    // enough warps for every SM to have many loads in flight: two warps share a long row
    const int wpr = K >= 4096 ? 2 : 1;
    const unsigned grid = (unsigned)((M + kRotRows - 1) / kRotRows);
    return launch_pdl(quant_rotated_kernel, dim3(grid), kRotRows * wpr * 32, 0, (cudaStream_t)stream, reinterpret_cast<const bf16*>(xr),
                      amax_part, q, scales, M, K, K / 64, wpr);
}
