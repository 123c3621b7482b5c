// The dequant epilogue's arithmetic, shared by the GEMM kernels (one element at a time here; the tensor-core kernel
// applies the same operations eight columns at a time).
//   t0 = float(acc) * xs;  y = out(fma(t0, ws, bias));  residual: fma(y, rscale, resid);  activation: act(y)
// The caller rounds the returned value to the output type when it stores it.
// Reference: csrc/vendor/cutlass_gemm_int8.cu:84-95 and :143-161 (nvcc fuses both multiply-adds there).
#pragma once

#include "common.cuh"

// EPI_ACT computes the activation; EPI_ACT_LUT (tensor-core kernel, bf16 outputs) reads bf16(act(x)) from a table instead;
// EPI_ACT_ROT does that and rotates each 256-column group of the row (R256) before the store
enum EpiMode { EPI_PLAIN = 0, EPI_RESID = 1, EPI_ACT = 2, EPI_ACC = 3, EPI_ACT_LUT = 4, EPI_ACT_ROT = 5 };
enum Act { ACT_NONE = 0, ACT_GELU_TANH = 1, ACT_SILU = 2, ACT_GELU_ERF = 3 };

template <typename OutT, int EPI>
__device__ __forceinline__ float epilogue1(int acc, float xs, float ws, float bias, float rscale, float resid, int act) {
    const float t0 = __fmul_rn(__int2float_rn(acc), xs);
    float v = rnd<OutT>(__fmaf_rn(t0, ws, bias));
    if (EPI == EPI_RESID) v = __fmaf_rn(v, rscale, resid);
    else if (EPI == EPI_ACT) v = act == ACT_GELU_TANH ? gelu_tanh_f(v) : act == ACT_SILU ? silu_f(v) : gelu_f(v);
    return v;
}

// Arguments of the few-rows kernel (gemm_skinny.cu); launched from the GEMM entry points in gemm_i8.cu.
struct SkinnyParams {
    const int8_t* A;     // [M, K]
    const int8_t* W;     // [N, K]
    const float* xs;
    const float* ws;
    const void* bias;
    const void* rscale;
    const void* resid;
    void* D;
    int M, N, K;
    int act;
};
// Rows of the fp16 quantizers: read as they lie, or computed as the kernel of the reference that would have written them in
// half does (csrc/sd.cu:611-724).
enum { SDQ_ROWS = 0, SDQ_LN = 1, SDQ_GEGLU = 2, SDQ_UNPAD = 3, SDQ_GN = 4 };
struct SdSrc {
    const half* x;
    int64_t x_stride;   // ROWS, LN: elements between rows
    const float* w;     // LN, GN: weight and bias
    const float* b;
    float eps;          // LN, GN
    int heads, d, dp;   // UNPAD: heads of d values stored dp wide
    const double* sums; // GN: per (image, group) sum and sum of squares
    int groups;         // GN
    int64_t P;          // GN: pixels per image
    double cnt;         // GN: values per group, P * C / groups
};
// Helpers shared between the translation units (a namespace of their own: the static archive exports them).
namespace b200q {
// quant_rows.cu: table of bf16(act(x)) over all bf16 x for Act code `act`, built on first use (on `st`)
int act_lut_ptr(int act, cudaStream_t st, const uint16_t** out);
// quant_rows.cu: the quantizer's status word (non-zero after a staging wait ran out), read and cleared
int quant_status_read_clear(int* out);
// quant_rows.cu: gpu_rotate_rows_f32's prologue + rotation with the rows written as three signed 8-bit digits [3][M, K] and a factor
// per row, negative for a spread row, whose groups of 256 have the factor |f| 2^-shift with shifts [K / 256][M] (written for spread
// rows only); zeroes nzero words at `zero`
int rotate_rows_digits(int prologue, const float* x, int64_t x_stride, int64_t up_offset, const float* norm_w, float eps, int8_t* digits,
                       float* factors, uint8_t* shifts, int* zero, int nzero, int M, int K, cudaStream_t st);
// The largest shift. A spread row's sums are kept in units of |f| 2^-40 where the row's maximum is at least 1 (and of |f| below: no group lies
// more than 149 under such a maximum), which lets 2^-shift end at f32's 2^-149 without a sum of 2^43 units ending beyond 2^127.
constexpr int kWo8MaxShift = 189, kWo8Lift = 40;
// quant_rows.cu: the fp16 row quantizers on the register kernel; false when the shape is outside what it takes
bool sd_quant_fast(int src, const SdSrc& s, int8_t* q, float* scales, int M, int K, int rotate, cudaStream_t st, int* rc);
bool skinny_gemm_applies(int64_t M, int64_t N, int64_t K);
int launch_skinny_gemm(int epi, const SkinnyParams& p, int out_dt, int sms, cudaStream_t st);
// gemm_skinny.cu: the CUDA-core kernel for operands TMA cannot address (K % 16 != 0, bases off a 16-byte boundary)
int launch_generic_gemm(int epi, const SkinnyParams& p, int out_dt, cudaStream_t st);
}  // namespace b200q
using namespace b200q;
