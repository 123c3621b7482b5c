// The weight-only int8 linear's product (included by gemm_i8.cu): D[M,N] (f32) = [D +] x[M,K] . (Wq[N,K] * ws[n])^T on the int8
// tensor cores. The f32 rows arrive as fixed-point numbers of 22 bits and sign, a power of two per row, cut into three signed 8-bit
// digits: x = (d0 2^16 + d1 2^8 + d2) xs[m], planes [3][M, K] int8 (quant_rows.cu). W is int8 as it lies, so the three products are
// exact int32 sums, and what is lost is the row's rounding to 2^-22 of its maximum, at most 2^-20 of the maximum of the value's rotation
// group (two bf16 terms leave 2^-18 of each value), and a few f32 roundings at the end.
//
// Rows whose groups lie further apart (xs[m] negative) have a power of two per group of 256. A token tile with such a row is
// drained after every group, two K boxes, and the groups meet in f32: the price is the drain between each two boxes' MMAs, which is why ordinary
// tiles do not go this way. 512 tokens, gate-up 2560 -> 19456 + down 9728 -> 2560: ordinary rows 68.1 + 54.8 us, every row spread 122.5 + 77.9 (two bf16 terms
// 121.9 + 116.5), one row of the 512 spread 81.1 + 55.2; 20 tokens, all spread, 24.1 + 22.2.
//
// Three int8 products take three quarters of the time of the two bf16 ones they replace, W goes to the SMs in one byte
// instead of two, and the pass that widened W is gone: bound by the tensor core from a few hundred tokens up, by W's bytes below.
// Weight rows are the MMA's M (256 per CTA pair), tokens and digits its N: all 3 T columns in one MMA, or in two of about the same
// width (an MMA of 128 columns reads its operands from shared memory nearly as long as one of 256; a digit each took 81 us where two
// wide ones take 69, 512 x 2560 -> 19456), and a lane owns an output column, so that a warp's stores are whole lines. T <= 160 is what
// 512 columns of tensor memory hold.
//
// The K boxes of all tiles are dealt out in equal contiguous shares, one per cluster (a tile is 20 to 76 boxes long and there are
// seldom a whole number of rounds of them: 512 x 9728 -> 2560 is 40 tiles for 74 clusters). A tile that two or more clusters share
// meets in scratch: each leaves the f32 values of its boxes, and the one that arrives last adds them up in the order of the
// clusters, so the sum does not depend on who that is. Where the scratch is too small, or whole tiles fill the rounds, the shares
// are rounded to whole tiles.
constexpr int kWo8Threads = 320;          // warp 0 loads, warp 1 issues the MMAs, warps 2-9 drain
constexpr int kWo8MaxTokens = 160;
constexpr int kWo8Counters = 16;          // per shared tile: CTA of the pair x lane quarter x half of the tokens
struct Wo8Params {
    const float* xs;     // [M] row factors, negative: a spread row, with
    const uint8_t* shifts;      // [K / 256][M]: the factor of group g is |xs[m]| 2^-shifts[g][m]
    const float* ws;     // [N]
    float* D;            // [M, N]
    int M, N, add;
    int tiles_m;         // token tiles, fastest in the tile order: a tile of W is used by all of them before the next
    int k_iters;         // 128-byte K boxes
    int stages;
    // cluster c's share starts at (c * share + min(c, extra)) * unit boxes
    int64_t share;
    int extra, unit;     // unit: 1, or k_iters where shares are whole tiles
    int* counters;       // [clusters][kWo8Counters], zero before the launch
    float* parts;        // [2 clusters][2][4][2][T / 2][32]
};
__device__ __forceinline__ int64_t wo8_start(const Wo8Params& p, int c) { return (c * p.share + min(c, p.extra)) * p.unit; }

// Rows of a CTA's digits in the first MMA: all of them up to 256 columns, else about half (columns of an MMA come in 32s)
__host__ __device__ constexpr int wo8_rows0(int T) { return 3 * T <= 256 ? 3 * T / 2 : T == 96 ? 80 : T == 128 ? 96 : 128; }

// NCH: 16-token pieces a draining warp holds (T = 32 NCH)
template <int NCH>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kWo8Threads, 1)
gemm_wo8_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const Wo8Params p) {
    constexpr int T = 32 * NCH;
    constexpr uint32_t w_bytes = BM * BK, x_bytes = (3 * T / 2) * BK, stage_bytes = w_bytes + x_bytes;
    // A CTA's 3 T / 2 rows are digit-major; the first r0 of both CTAs go to the first MMA (columns 0 .. 2 r0 - 1, CTA 0's before
    // CTA 1's), the others to the second.
    constexpr int r0 = wo8_rows0(T), r1 = 3 * T / 2 - r0;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    const uint32_t base = (raw_addr + 1023u) & ~1023u;
    uint8_t* sm = smem_raw + (base - raw_addr);
    const int S = p.stages;
    uint8_t* tail = sm + S * stage_bytes;
    const uint32_t bar_full = smem_u32(tail), bar_empty = bar_full + 8 * kMaxStages, bar_tfull = bar_empty + 8 * kMaxStages, bar_tempty = bar_tfull + 8;
    uint32_t* tmem_ptr_s = reinterpret_cast<uint32_t*>(tail + 8 * (2 * kMaxStages + 2));
    volatile int* abort_s = reinterpret_cast<volatile int*>(tmem_ptr_s + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const bool leader = rank == 0;
    const int cluster_id = blockIdx.x >> 1;

    if (threadIdx.x == 0) {
        for (int i = 0; i < S; ++i) mbar_init(bar_full + 8 * i, 1), mbar_init(bar_empty + 8 * i, 1);
        mbar_init(bar_tfull, 1), mbar_init(bar_tempty, 16);
        *abort_s = 0;
        fence_mbar_init();
        prefetch_tmap(&tmap_w), prefetch_tmap(&tmap_x);
    }
    if (warp == 1) {
        tmem_alloc_pair(smem_u32(tmem_ptr_s), 512);
        tmem_relinquish_pair();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();
    tc_fence_after();
    pdl_wait();
    const uint32_t tmem_base = *tmem_ptr_s;
    const int64_t u0 = wo8_start(p, cluster_id), u1 = wo8_start(p, cluster_id + 1);
    // Whether a tile's tokens hold a spread row, in two steps: the loads, and the warp's answer
    struct Factors { float v[NCH]; };
    auto tile_factors = [&](int tile) {
        Factors f;
        const int t0 = tile % p.tiles_m * T + lane;
#pragma unroll
        for (int i = 0; i < NCH; ++i) f.v[i] = t0 + 32 * i < p.M ? gload(p.xs + t0 + 32 * i) : 0.f;
        return f;
    };
    auto any_spread = [](const Factors& f) {
        int s = 0;
#pragma unroll
        for (int i = 0; i < NCH; ++i) s |= __float_as_int(f.v[i]);
        return __any_sync(0xffffffffu, s < 0) != 0;
    };

    if (warp == 0) {
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0;
            int tile = (int)(u0 / p.k_iters), kb = (int)(u0 - (int64_t)tile * p.k_iters);
            for (int64_t u = u0; u < u1; ++u) {
                if (!mbar_wait(bar_empty + 8 * stage, phase ^ 1u, abort_s, ST_TIMEOUT_EMPTY)) break;
                const int tn = tile / p.tiles_m, t0 = (tile - tn * p.tiles_m) * T + (int)rank * (T / 2);
                if (leader) mbar_arrive_expect_tx(bar_full + 8 * stage, 2 * stage_bytes);
                const uint32_t full = mapa_shared(bar_full + 8 * stage, 0), dst = base + stage * stage_bytes;
                tma_load_2d_pair(dst, &tmap_w, kb * BK, tn * 2 * BM + (int)rank * BM, full);
                tma_load_3d_pair(dst + w_bytes, &tmap_x, kb * BK, t0, 0, full);
                if (++stage == S) stage = 0, phase ^= 1u;
                if (++kb == p.k_iters) kb = 0, ++tile;
            }
        }
    } else if (warp == 1) {
        if (leader) {
            const bool one = elect_one();
            int stage = 0;
            uint32_t phase = 0, tphase = 0;
            int tile = (int)(u0 / p.k_iters), kb = (int)(u0 - (int64_t)tile * p.k_iters);
            bool fresh = true, spread = any_spread(tile_factors(tile));
            Factors next = tile_factors(tile + 1);      // requested a tile ahead
            for (int64_t u = u0; u < u1; ++u) {
                if (fresh && !__all_sync(0xffffffffu, mbar_wait(bar_tempty, tphase ^ 1u, abort_s, ST_TIMEOUT_TMEM_EMPTY))) break;
                if (fresh) tc_fence_after();
                if (!__all_sync(0xffffffffu, mbar_wait(bar_full + 8 * stage, phase, abort_s, ST_TIMEOUT_FULL))) break;
                const uint32_t w_lo = umma_desc_lo(base + stage * stage_bytes), x_lo = w_lo + (w_bytes >> 4);
                if (one) {
#pragma unroll
                    for (int k = 0; k < BK / UMMA_K; ++k) {
                        umma_pair_lo(tmem_base, w_lo + 2 * k, x_lo + 2 * k, umma_idesc_i8(2 * BM, 2 * r0), !fresh || k != 0);
                        if (r1 > 0) umma_pair_lo(tmem_base + 2 * r0, w_lo + 2 * k, x_lo + 8 * r0 + 2 * k, umma_idesc_i8(2 * BM, 2 * r1), !fresh || k != 0);
                    }
                    umma_commit_pair(bar_empty + 8 * stage);
                }
                __syncwarp();
                if (++stage == S) stage = 0, phase ^= 1u;
                ++kb;
                fresh = kb == p.k_iters || u + 1 == u1 || (spread && (kb & 1) == 0);
                if (fresh) {
                    if (one) umma_commit_pair(bar_tfull);
                    __syncwarp();
                    tphase ^= 1u;
                    if (kb == p.k_iters) {
                        kb = 0, ++tile;
                        spread = any_spread(next);
                        next = tile_factors(tile + 1);
                    }
                }
            }
        }
    } else {
        const int quad = warp & 3, half = (warp - 2) >> 2;
        const int sub = ((int)rank * 4 + quad) * 2 + half;
        constexpr int kTok = T / 2;                    // tokens of this warp
        uint32_t tphase = 0;
        int64_t u = u0;
        while (u < u1) {
            const int tile = (int)(u / p.k_iters), k0 = (int)(u - (int64_t)tile * p.k_iters);
            const int64_t end = min((int64_t)(tile + 1) * p.k_iters, u1);
            const bool whole = k0 == 0 && end == (int64_t)(tile + 1) * p.k_iters;
            const int tn = tile / p.tiles_m, t0 = (tile - tn * p.tiles_m) * T + half * kTok;
            const int n = tn * 2 * BM + (int)rank * BM + quad * 32 + lane;
            const bool n_ok = n < p.N;
            const float ws = n_ok ? gload(p.ws + n) : 0.f;
            constexpr int kRegs = (NCH + 1) / 2;       // lane l: factors of tokens t0 + l, t0 + 32 + l, ...
            float xs[kRegs];
#pragma unroll
            for (int i = 0; i < kRegs; ++i) xs[i] = t0 + 32 * i + lane < p.M ? gload(p.xs + t0 + 32 * i + lane) : 0.f;
            const bool spread = any_spread(tile_factors(tile));
            const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16);
            auto column = [&](int d, int c) {          // of digit d, tokens 16 c .. 16 c + 15 of this warp's half
                const int r = d * kTok + 16 * c;
                return (uint32_t)(r < r0 ? half * r0 + r : 2 * r0 + half * r1 + r - r0);
            };
            auto hand_back = [&]() {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_remote(mapa_shared(bar_tempty, 0));
            };
            float f[kTok];
            if (!spread) {
                if (!mbar_wait_warp_relaxed(bar_tfull, tphase, abort_s, ST_TIMEOUT_TMEM_FULL)) break;
                tphase ^= 1u;
                tc_fence_after();
                // out of tensor memory first: the next tile's MMAs wait for it, not for the stores
#pragma unroll
                for (int c = 0; c < NCH; ++c) {
                    uint32_t a[16], b[16], d[16];
                    tmem_ld16(taddr + column(0, c), a);
                    tmem_ld16(taddr + column(1, c), b);
                    tmem_ld16(taddr + column(2, c), d);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 16; ++i)
                        f[16 * c + i] = __fmaf_rn(__int2float_rn((int)a[i]), 65536.f, __fmaf_rn(__int2float_rn((int)b[i]), 256.f, __int2float_rn((int)d[i])));
                }
                hand_back();
            } else {
                // Group by group. The sums of 256 products of a digit stay below 2^22: the lower two digits join as integers.
#pragma unroll
                for (int i = 0; i < kTok; ++i) f[i] = 0.f;
                bool ok = true;
                for (int64_t v = u; v < end;) {
                    const int kb = (int)(v - (int64_t)tile * p.k_iters);
                    v = min(v + 2 - (kb & 1), end);
                    float rel[kRegs];                  // 2^-shift, as two factors (the product may be subnormal)
#pragma unroll
                    for (int i = 0; i < kRegs; ++i) {
                        rel[i] = 1.f;
                        if (__float_as_int(xs[i]) < 0) {
                            const int s = gload(p.shifts + (int64_t)(kb >> 1) * p.M + t0 + 32 * i + lane), h = s >> 1;
                            rel[i] = __uint_as_float((uint32_t)(127 + (xs[i] <= -0x1p-21f ? kWo8Lift : 0) - h) << 23) * __uint_as_float((uint32_t)(127 - (s - h)) << 23);
                        }
                    }
                    if (!mbar_wait_warp_relaxed(bar_tfull, tphase, abort_s, ST_TIMEOUT_TMEM_FULL)) { ok = false; break; }
                    tphase ^= 1u;
                    tc_fence_after();
#pragma unroll
                    for (int c = 0; c < NCH; ++c) {
                        uint32_t a[16], b[16], d[16];
                        tmem_ld16(taddr + column(0, c), a);
                        tmem_ld16(taddr + column(1, c), b);
                        tmem_ld16(taddr + column(2, c), d);
                        tmem_ld_wait();
                        if (c + 1 == NCH) hand_back();
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            const float lower = __int2float_rn((int)(b[i] * 256u + d[i]));
                            f[16 * c + i] = __fmaf_rn(__fmaf_rn(__int2float_rn((int)a[i]), 65536.f, lower), __shfl_sync(0xffffffffu, rel[c >> 1], 16 * (c & 1) + i), f[16 * c + i]);
                        }
                    }
                }
                if (!ok) break;
#pragma unroll
                for (int i = 0; i < kRegs; ++i)
                    if (__float_as_int(xs[i]) < 0) xs[i] = xs[i] <= -0x1p-21f ? xs[i] * -0x1p-40f : -xs[i];
            }
            u = end;
            if (!whole) {
                // this cluster's share of the tile into its slot; the last to arrive at the tile's counter adds the slots up
                const int64_t u_first = (int64_t)tile * p.k_iters;
                int c0 = cluster_id, c1 = cluster_id;
                while (wo8_start(p, c0) > u_first) --c0;
                while (wo8_start(p, c1 + 1) < u_first + p.k_iters) ++c1;
                auto slot = [&](int c) {               // a share's first piece of a tile begun before it: slot 0, its last piece: slot 1
                    const int which = wo8_start(p, c) > u_first ? 0 : 1;
                    return p.parts + ((int64_t)(2 * c + which) * kWo8Counters + sub) * (kTok * 32) + lane;
                };
                float* own = slot(cluster_id);
#pragma unroll
                for (int i = 0; i < kTok; ++i) own[32 * i] = f[i];
                __threadfence();
                __syncwarp();
                int old = 0;
                if (lane == 0) old = atomicAdd(p.counters + c0 * kWo8Counters + sub, 1);
                if (__shfl_sync(0xffffffffu, old, 0) != c1 - c0) continue;
                __threadfence();
#pragma unroll 1
                for (int c = c0; c <= c1; ++c) {
                    const float* s = slot(c);
#pragma unroll
                    for (int i = 0; i < kTok; ++i) f[i] = __fadd_rn(c == c0 ? 0.f : f[i], __ldcg(s + 32 * i));
                }
            }
            float* out = p.D + (int64_t)t0 * p.N + n;      // the column's factor first: the row's may be near f32's ends
            if (p.add) {
#pragma unroll
                for (int c = 0; c < NCH; ++c) {
                    float r[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) r[i] = n_ok && t0 + 16 * c + i < p.M ? out[(int64_t)(16 * c + i) * p.N] : 0.f;
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const float x = __shfl_sync(0xffffffffu, xs[c >> 1], 16 * (c & 1) + i);
                        if (n_ok && t0 + 16 * c + i < p.M) out[(int64_t)(16 * c + i) * p.N] = __fadd_rn(__fmul_rn(__fmul_rn(f[16 * c + i], ws), x), r[i]);
                    }
                }
            } else {
#pragma unroll
                for (int i = 0; i < kTok; ++i) {
                    const float x = __shfl_sync(0xffffffffu, xs[i >> 5], i & 31);
                    if (n_ok && t0 + i < p.M) out[(int64_t)i * p.N] = __fmul_rn(__fmul_rn(f[i], ws), x);
                }
            }
        }
    }

    __syncwarp();
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();
    if (*abort_s != 0) {
        for (int i = 0; i < 2000; ++i) __nanosleep(1000);      // leave time for copies and MMAs still in flight, then report
        if (threadIdx.x == 0) atomicCAS(&g_kernel_status, 0, *abort_s);
        __syncthreads();
    }
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, 512);
    }
}

// The digits [3][M, K] in boxes of 128 bytes x box_rows tokens x 3 digits; tokens beyond M read as zero
bool make_digits_tmap(CUtensorMap* tm, const void* ptr, int64_t M, int64_t K, int box_rows) {
    const TmapKey k{ptr, K, M, K, BK, box_rows, 4};
    if (const CUtensorMap* hit = g_tmaps.find(k)) { *tm = *hit; return true; }
    EncodeTiledFn enc = encode_fn();
    if (!enc) return false;
    const cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)M, 3};
    const cuuint64_t strides[2] = {(cuuint64_t)K, (cuuint64_t)(M * K)};
    const cuuint32_t box[3] = {(cuuint32_t)BK, (cuuint32_t)box_rows, 3};
    const cuuint32_t estr[3] = {1, 1, 1};
    if (enc(tm, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return false;
    g_tmaps.put(k, *tm);
    return true;
}

template <int NCH>
int launch_wo8(const CUtensorMap& tw, const CUtensorMap& tx, const Wo8Params& p, int clusters, cudaStream_t st) {
    auto kern = gemm_wo8_kernel<NCH>;
    static std::atomic<uint64_t> configured{0};
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = 1ull << (dev & 63);
    if (!(configured.load(std::memory_order_acquire) & bit)) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
        if (e != cudaSuccess) return (int)e;
        configured.fetch_or(bit, std::memory_order_release);
    }
    return launch_pdl(kern, dim3(2 * clusters), kWo8Threads, kSmemBytes, st, tw, tx, p);
}

// How a call is cut, and what it leaves in the caller's scratch: the digits [3][M, K], the row factors [M] and the groups' shifts
// [K / 256][M] in a_scratch (4 M K bytes, K >= 256), the counters and the shared tiles' values in w_scratch (2 N K bytes).
struct Wo8Plan {
    int tokens, tiles_m, tiles, clusters;
    bool whole;
    size_t counter_bytes;
};
Wo8Plan plan_wo8(int64_t M, int64_t N, int64_t K, int max_clusters) {
    Wo8Plan r{};
    const int64_t k_iters = K / BK, tiles_n = (N + 2 * BM - 1) / (2 * BM);
    // Token tiles: the fewest cycles of a K box over all of them, of the tensor core (12 T / 2) or of the operands' way in (64 bytes a
    // cycle), whichever is longer.
    int64_t best = INT64_MAX;
    const int64_t least = (M + kWo8MaxTokens - 1) / kWo8MaxTokens;
    for (int64_t m = least; m < least + 4; ++m) {
        const int64_t T = ((M + m - 1) / m + 31) / 32 * 32, tiles_m = (M + T - 1) / T;
        const int64_t cost = tiles_m * std::max<int64_t>(6 * T, 256 + 3 * T);
        if (cost < best) best = cost, r.tokens = (int)T, r.tiles_m = (int)tiles_m;
    }
    const int64_t tiles = tiles_n * r.tiles_m;
    if (tiles > INT32_MAX) return r;
    r.tiles = (int)tiles;
    r.counter_bytes = ((size_t)max_clusters * kWo8Counters * 4 + 127) & ~(size_t)127;
    const size_t need = r.counter_bytes + (size_t)max_clusters * 2 * (2 * BM) * r.tokens * 4;
    // Equal shares where they save more than the exchange costs, about six K boxes; whole tiles otherwise.
    const int64_t rounds = (tiles + max_clusters - 1) / max_clusters;
    const int64_t share = (tiles * k_iters + max_clusters - 1) / max_clusters;
    r.whole = need > (size_t)2 * N * K || rounds * k_iters <= share + 6 || share < 4;
    r.clusters = r.whole && tiles < max_clusters ? (int)tiles : max_clusters;
    return r;
}
int run_wo8(bool add, const Wo8Plan& r, const int8_t* digits, const float* xs, const uint8_t* shifts, const int8_t* W, const float* ws, float* D, void* w_scratch,
            int64_t M, int64_t N, int64_t K, cudaStream_t st) {
    Wo8Params p{};
    p.xs = xs, p.shifts = shifts, p.ws = ws, p.D = D;
    p.M = (int)M, p.N = (int)N, p.add = add;
    p.tiles_m = r.tiles_m;
    p.k_iters = (int)(K / BK);
    p.unit = r.whole ? p.k_iters : 1;
    const int64_t pieces = r.whole ? r.tiles : (int64_t)r.tiles * p.k_iters;
    p.share = pieces / r.clusters, p.extra = (int)(pieces % r.clusters);
    p.stages = (kSmemBytes - 1024 - kTailBytes) / (BM * BK + 3 * r.tokens / 2 * BK);
    if (p.stages > kMaxStages) p.stages = kMaxStages;
    p.counters = reinterpret_cast<int*>(w_scratch);
    p.parts = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(w_scratch) + r.counter_bytes);
    CUtensorMap tw, tx;
    if (!make_operand_tmap(&tw, W, N, K, BM) || !make_digits_tmap(&tx, digits, M, K, r.tokens / 2)) return -203;
    switch (r.tokens / 32) {
        case 1: return launch_wo8<1>(tw, tx, p, r.clusters, st);
        case 2: return launch_wo8<2>(tw, tx, p, r.clusters, st);
        case 3: return launch_wo8<3>(tw, tx, p, r.clusters, st);
        case 4: return launch_wo8<4>(tw, tx, p, r.clusters, st);
        default: return launch_wo8<5>(tw, tx, p, r.clusters, st);
    }
}
