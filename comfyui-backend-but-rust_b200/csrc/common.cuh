// Shared device/host helpers of the sm_100a quantized-linear kernels.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>

#define GPU_API extern "C" __attribute__((visibility("default")))

// dtype codes of the C ABI (the reference's src/ffi.rs:11-13)
enum DType { DT_F32 = 0, DT_F16 = 1, DT_BF16 = 2 };

// Launch-error convention of the ABI: a positive cudaError_t (the reference's KCHECK, csrc/common.cuh:128).
#define KCHECK()                                    \
    do {                                            \
        cudaError_t e__ = cudaGetLastError();       \
        if (e__ != cudaSuccess) return (int)e__;    \
    } while (0)

typedef __nv_bfloat16 bf16;

// ---- programmatic dependent launch ------------------------------------------------------------------------------------
// The linears of a block are ten to fifteen short kernels one after the other, and between two of them a stream idles for
// the drain of the first, the launch of the second and its setup (barriers, tensor memory, tensor maps): 2 to 4 us. So every
// kernel of a forward pass is launched with `launch_pdl` and has
//   - pdl_wait(), before the first access to memory that another kernel reads or writes: everything launched before in the
//     stream has ended and its writes are visible. Every thread that touches such memory waits, so an order that held
//     between whole kernels (results, buffers used again, the zeros of the split scratch) holds as before;
//   - in the quantizers and the W6 decoder pdl_trigger(), when a CTA has its rows and little but the codes and their stores is
//     left, or as soon as its rows are in where the CTAs leave SMs idle (early_trigger() in quant_rows.cu): the stream's next kernel may be
//     brought onto the SMs once every CTA has got there or ended. The others, the GEMMs among them, leave it at the end of their CTAs. A trigger at a kernel's start loses more than it hides: the successor's
//     CTAs then go where there is room beside the running kernel, and a small quantizer after a GEMM on 64 of 74 cluster pairs
//     lands on the twenty idle SMs, all of it. As CUDA graphs, with the trigger at the start | here | ordinary launches: DiT block
//     512 x 1536 105 | 85 | 90 us, SwiGLU block 512 x 1536 90 | 70 | 75, linear 333 x 3072 x 3072 18.3 | 15.4 | 16.9, two
//     linears 154 x 2048 x 1280 18.0 | 18.4 | 19.8.
// Such memory may change while the kernel is resident, so it is not read-only for the kernel's duration: no __ldg and no
// __restrict__ on what a kernel with a wait reads or writes. Both allow loads through the read-only path, which PTX defines only for
// memory nothing writes meanwhile and which the compiler may move ahead of the wait; gload() is an ordinary load, which the wait's
// memory clobber holds back.
// A successor launched the ordinary way waits for the end of the grid as always. While a cluster limit keeps SMs free for another
// stream's kernels (gpu_int8_gemm_set_cluster_limit), every launch is the ordinary way: a successor waiting on the free SMs would
// take the very room the limit keeps.
namespace b200q { int gemm_cluster_limit(); }      // gemm_i8.cu
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
template <typename T> __device__ __forceinline__ T gload(const T* p) { return *p; }
template <typename... P, typename... A>
inline int launch_pdl_cluster(void (*kern)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st, int cluster, const A&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid, cfg.blockDim = dim3(threads), cfg.dynamicSmemBytes = smem, cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = (unsigned)cluster, at[1].val.clusterDim.y = 1, at[1].val.clusterDim.z = 1;
    const int first = b200q::gemm_cluster_limit() > 0 ? 1 : 0;      // 1: without the first attribute
    cfg.attrs = at + first, cfg.numAttrs = (cluster > 1 ? 2 : 1) - first;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
    if (e != cudaSuccess) (void)cudaGetLastError();
    return (int)e;
}
template <typename... P, typename... A>
inline int launch_pdl(void (*kern)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st, const A&... args) {
    return launch_pdl_cluster(kern, grid, threads, smem, st, 1, args...);
}

// ---- device status word ---------------------------------------------------------------------------
// A kernel whose bounded wait runs out records a code here and returns; gpu_kernels_status() reads it.
enum KernelStatus {
    ST_OK = 0,
    ST_TIMEOUT_EMPTY = 1,    // TMA producer waited for a free shared-memory stage
    ST_TIMEOUT_FULL = 2,     // MMA issuer waited for a filled stage
    ST_TIMEOUT_TMEM_FULL = 3,  // epilogue waited for an accumulator
    ST_TIMEOUT_TMEM_EMPTY = 4, // MMA issuer waited for a drained accumulator
    ST_TIMEOUT_UNPACK = 5,   // W6 unpack warps waited for a packed stage
};

// ---- rounding to a storage type and back (what materialising a tensor of that type does) ----------
template <typename T> __device__ __forceinline__ float rnd(float v);
template <> __device__ __forceinline__ float rnd<float>(float v) { return v; }
template <> __device__ __forceinline__ float rnd<bf16>(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
template <> __device__ __forceinline__ float rnd<half>(float v) { return __half2float(__float2half_rn(v)); }

template <typename T> __device__ __forceinline__ float to_f(T v);
template <> __device__ __forceinline__ float to_f<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f<bf16>(bf16 v) { return __bfloat162float(v); }
template <> __device__ __forceinline__ float to_f<half>(half v) { return __half2float(v); }

template <typename T> __device__ __forceinline__ T from_f(float v);
template <> __device__ __forceinline__ float from_f<float>(float v) { return v; }
template <> __device__ __forceinline__ bf16 from_f<bf16>(float v) { return __float2bfloat16_rn(v); }
template <> __device__ __forceinline__ half from_f<half>(float v) { return __float2half_rn(v); }

// ---- activations, the expressions of the reference's quantizer prologues (csrc/common.cuh:71-95) --
// Compiled without fast-math like the reference's units, so expf/tanhf/erff are the same CUDA routines.
__device__ __forceinline__ float silu_f(float x) { return x / (1.f + expf(-x)); }
__device__ __forceinline__ float sigmoid_f(float x) { return 1.f / (1.f + expf(-x)); }
__device__ __forceinline__ float gelu_f(float x) { return 0.5f * x * (1.f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_tanh_f(float x) {
    const float k0 = 0.7978845608028654f, k1 = 0.044715f;
    return 0.5f * x * (1.f + tanhf(k0 * (x + k1 * x * x * x)));
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// (int8) min(127, max(lo, rint(t))) with fmaxf/fminf NaN rules (NaN -> lo)
__device__ __forceinline__ int clamp_rint_i8(float t, float lo) {
    return (int)fminf(127.f, fmaxf(lo, nearbyintf(t)));
}

// ---- PTX wrappers: mbarrier, TMA, tcgen05 ------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// The same with a suspend-time hint: the thread may stay suspended in hardware for up to `ns` nanoseconds (it is
// woken when the phase completes), instead of returning after the short system default and spinning in software.
__device__ __forceinline__ bool mbar_try_wait_hint(uint32_t bar, uint32_t parity, uint32_t ns) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(ns)
        : "memory");
    return ok != 0;
}
// Bounded wait built on it, for roles that can afford a wake-up latency: a handful of instructions per poll and a
// poll only every few microseconds, so that many waiting warps do not take issue slots from the working ones.
__device__ __forceinline__ bool mbar_wait_suspended(uint32_t bar, uint32_t parity, volatile int* abort_flag, int code);
// Non-blocking test of an mbarrier phase.
__device__ __forceinline__ bool mbar_test_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ uint64_t globaltimer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// Bounded wait: gives up after about two seconds, or as soon as another role has raised `*abort_flag`
// (shared memory). On giving up it raises the flag with `code` itself. Returns false when it gave up.
constexpr uint64_t kWaitLimitNs = 2000000000ull;
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int code) {
    if (mbar_try_wait(bar, parity)) return true;
    uint64_t t0 = 0;
    for (uint32_t it = 1;; ++it) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((it & 63u) == 0u) {
            if (*abort_flag) return false;
            const uint64_t now = globaltimer_ns();
            if (t0 == 0) t0 = now;
            else if (now - t0 > kWaitLimitNs) {
                *abort_flag = code;
                return false;
            }
        }
    }
}

__device__ __forceinline__ bool mbar_wait_suspended(uint32_t bar, uint32_t parity, volatile int* abort_flag, int code) {
    uint64_t t0 = 0;
    for (;;) {
        if (mbar_try_wait_hint(bar, parity, 4000u)) return true;
        if (*abort_flag) return false;
        const uint64_t now = globaltimer_ns();
        if (t0 == 0) t0 = now;
        else if (now - t0 > kWaitLimitNs) {
            *abort_flag = code;
            return false;
        }
    }
}

// The same wait for a whole warp whose wake-up is not urgent: one lane polls, sleeping between polls, so that
// hundreds of idle threads do not hammer the barrier's shared-memory word while the tensor core reads operands.
__device__ __forceinline__ bool mbar_wait_warp_relaxed(uint32_t bar, uint32_t parity, volatile int* abort_flag, int code) {
    bool ok = true;
    if ((threadIdx.x & 31) == 0) {
        uint64_t t0 = 0;
        for (uint32_t it = 0;; ++it) {
            if (mbar_try_wait(bar, parity)) break;
            __nanosleep(128);
            if ((it & 15u) == 15u) {
                if (*abort_flag) { ok = false; break; }
                const uint64_t now = globaltimer_ns();
                if (t0 == 0) t0 = now;
                else if (now - t0 > kWaitLimitNs) { *abort_flag = code; ok = false; break; }
            }
        }
    }
    return __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
}

// 2-D tiled TMA load, global -> this CTA's shared memory, completion on an mbarrier (no multicast).
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const void* tmap, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(tmap), "r"(x), "r"(y), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void prefetch_tmap(const void* tmap) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(tmap) : "memory");
}
// Makes generic-proxy writes to shared memory visible to the async proxy (TMA, tcgen05.mma operand reads).
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t ncols) {  // whole warp
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {  // whole warp
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// One lane of a converged warp
__device__ __forceinline__ bool elect_one() {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(r));
    return r != 0;
}
// The mbarrier gets one arrival once every tcgen05.mma this thread issued before has completed.
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// 32 lanes x 32 consecutive 32-bit columns: thread t of the warp gets lane (base lane + t), columns c..c+31.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}

// 16 consecutive columns of the same shape
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
// The store of the same shape: thread t of the warp writes columns c..c+31 of lane (base lane + t).
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
          "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]),
          "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]),
          "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// Barrier `id` (1-15) among `threads` threads of the CTA (whole warps)
__device__ __forceinline__ void named_bar_sync(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Shared-memory matrix descriptor of a K-major operand tile stored as rows of 128 bytes with the 128-byte
// swizzle (what a TMA box of 128 bytes x rows with SWIZZLE_128B writes; tile base 1024-byte aligned):
// start address >> 4 in bits [0,14); leading byte offset (unused for this layout) 1 in [16,30);
// stride byte offset = 1024 B between 8-row groups, >> 4, in [32,46); descriptor version 1 in [46,48);
// layout type 2 (128-byte swizzle) in [61,64).
// As (low word, high word): all but the start address is the same for every tile.
constexpr uint32_t kDescHiSw128 = (uint32_t)(((uint64_t)(1024 >> 4) << 32 | (1ull << 46) | (2ull << 61)) >> 32);
__device__ __forceinline__ uint32_t umma_desc_lo(uint32_t smem_addr) { return ((smem_addr & 0x3FFFFu) >> 4) | (1u << 16); }
// Instruction descriptor for kind::i8: D s32 (bits 4-5 = 2), A and B signed 8-bit (bits 7-9, 10-12 = 1),
// both K-major (bits 15, 16 = 0), N >> 3 in bits 17-22, M >> 4 in bits 24-28, no saturation.
__host__ __device__ constexpr uint32_t umma_idesc_i8(int m, int n) {
    return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// ---- CTA-pair (cta_group::2) variants -----------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// shared::cluster address of `smem_addr` (a shared::cta address of this CTA's layout) in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t mapa_shared(uint32_t smem_addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// arrive on an mbarrier given by its shared::cluster address (this CTA's or the peer's)
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// The same arrival with the default (CTA-scope) release: for hand-offs whose data the consumer reads through the async
// proxy after the producer's own fence.proxy.async, where the cluster-scope release (measured at about a thousand
// cycles per arrival on B200) buys nothing.
__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// 2-D tiled TMA load issued by one CTA of a pair: data lands in this CTA's shared memory, the byte count is
// credited to an mbarrier that may live in the peer CTA (shared::cluster address). No multicast.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const void* tmap, int x, int y, uint32_t bar_cluster_addr) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(tmap), "r"(x), "r"(y), "r"(bar_cluster_addr)
        : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const void* tmap, int x, int y, int z, uint32_t bar_cluster_addr) {
    asm volatile(
        "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(dst), "l"(tmap), "r"(x), "r"(y), "r"(z), "r"(bar_cluster_addr)
        : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t smem_dst, uint32_t ncols) {  // one warp in each CTA of the pair
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// One arrival on the mbarrier at this shared-memory offset in BOTH CTAs of the pair, once every MMA this thread
// issued for the pair has completed. (A commit's arrival may be multicast; the TMA loads of this library never are.)
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"((uint16_t)3)
                 : "memory");
}

// D[tmem] (+)= A[smem desc] * B[smem desc], int8 x int8 -> int32, issued by one thread, which takes the descriptors as (low word, shared
// high word): its instruction count is what bounds the tensor pipe, so nothing 64-bit is computed per instruction.
__device__ __forceinline__ void umma_i8_lo(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "mov.b64 da, {%1, %5};\n\t"
        "mov.b64 db, {%2, %5};\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], da, db, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(kDescHiSw128)
        : "memory");
}
// The same over both SMs of a pair: D rows 0-127 accumulate in the leader's tensor memory, rows 128-255 in the peer's; A comes from
// each CTA's own tile, B's N columns are split between the two CTAs' tiles.
__device__ __forceinline__ void umma_pair_lo(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "mov.b64 da, {%1, %5};\n\t"
        "mov.b64 db, {%2, %5};\n\t"
        "tcgen05.mma.cta_group::2.kind::i8 [%0], da, db, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(kDescHiSw128)
        : "memory");
}
