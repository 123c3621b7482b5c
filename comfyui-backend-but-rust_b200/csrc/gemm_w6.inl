// W6A8 GEMM: the CTA-pair kernel of gemm_i8.cu with the W operand arriving as 6-bit codes and expanded to int8 in
// shared memory. Included by gemm_i8.cu inside its anonymous namespace (shares its parameters and epilogue).
//
// Storage (the reference's, csrc/h3.cu:8-37, csrc/vendor/w6a8_requant.cu:128-151): a weight row is K/2 bytes of low
// nibbles (element e in byte e/2, even e in the low nibble) followed by K/4 bytes holding the top two bits of four
// consecutive elements; one fp8-e4m3 scale s_rel per G = 32 columns; the int8 the GEMM multiplies is
// clamp(rint((code - 32) * s_rel), +-127). The reference decodes the whole matrix to int8 before every GEMM
// (src/h3.rs:1208-1216); here the packed planes are what crosses HBM and L2 (0.78 bytes per weight).
//
// Per 128-byte K box and CTA: TMA brings bn/2 rows x 64 B of nibbles and x 32 B of top bits (64-byte and 32-byte
// swizzles, so that one thread per row reads without bank conflicts); eight unpack warps, two threads per weight
// row, expand them into the 128-byte-swizzled int8 tile the MMA descriptor expects, make the writes visible to the
// async proxy and arrive on the leader's "full" barrier, which also counts the A bytes. Four epilogue warps.
// The arithmetic is exact in half precision: code - 32 has 6 bits, e4m3 has 4, the product at most 10; rint is one
// addition of 1536 (ulp 1), ties to even, after the clamp.

constexpr int kW6EpiWarps = 4;
constexpr int kW6Groups = 3;                     // unpack groups of four warps, taking K boxes in turn
constexpr int kW6UnpackWarps = 4 * kW6Groups;
constexpr int kW6Threads = 32 * (2 + kW6EpiWarps + kW6UnpackWarps);
constexpr int kW6StagingPerWarp = 6144;   // output chunk (2 KB, or 4 KB for 4-byte outputs) + 3 KB of staged vectors
constexpr int kW6StagingBytes = kW6EpiWarps * kW6StagingPerWarp;

struct W6Extra {
    const uint8_t* s_rel;   // [N, K / 32] e4m3
    int srel_pitch;         // K / 32
    int sb;                 // depth of the ring of expanded tiles
};

// Whole-warp wait for the unpack warps: lane 0 polls (256 threads polling one shared-memory word would compete with
// the tensor core's operand reads), then every lane observes the completed phase itself, which is what orders its
// reads after the TMA writes.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile int* abort_flag, int code) {
    int ok = 1;
    if ((threadIdx.x & 31) == 0) ok = mbar_wait_suspended(bar, parity, abort_flag, code) ? 1 : 0;
    ok = __shfl_sync(0xffffffffu, ok, 0);
    if (!ok) return false;
    return mbar_try_wait(bar, parity) || mbar_wait_suspended(bar, parity, abort_flag, code);
}

constexpr int kW6BStages = 4;    // ring of expanded W tiles: only has to span unpack -> MMA

// Rings: (A, packed planes) SA deep, filled by TMA far ahead of use; expanded W tiles kW6BStages deep, written by
// the unpack warps. Barriers: afull (leader: A bytes of both CTAs), pfull (per CTA: its packed planes), aempty (per
// CTA: MMAs have read A slot -> its packed slot is free too, the unpack that fed those MMAs being long done),
// bfull (leader: 16 unpack-warp arrivals), bempty (per CTA: MMAs have read the expanded slot).
// A tile has MH = 2 halves of 256 rows and 128 columns: an expanded W tile feeds two sets of MMAs (rows 0-255 and 256-511 of
// the tile, two accumulators per buffer), so the unpack work per MMA halves. A weight narrower than 128 columns takes one half
// and up to 128 columns (16896 x 64 x 1024: 11.0 us, 13.0 as two halves). Few rows take the kernel further down.
template <typename OutT, int EPI, int MH>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kW6Threads, 1)
gemm_w6a8_pair_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_lo,
                      const __grid_constant__ CUtensorMap tmap_hi, const __grid_constant__ CUtensorMap tmap_d,
                      const GemmParams p, const W6Extra x6) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    const uint32_t base = (raw_addr + 1023u) & ~1023u;
    uint8_t* sm = smem_raw + (base - raw_addr);
    const int SA = p.stages;
    const int SB = x6.sb;
    const int BN = p.bn;
    const int rows_w = BN / 2;                              // weight rows this CTA expands
    constexpr uint32_t a_box = BM * BK;                    // one 128-row, 128-byte K box of A
    const uint32_t a_bytes = MH * a_box, b_bytes = (uint32_t)rows_w * BK, lo_bytes = (uint32_t)rows_w * 64, hi_bytes = (uint32_t)rows_w * 32;
    uint8_t* staging = sm;
    const uint32_t sA = base + kW6StagingBytes;
    const uint32_t sB = sA + SA * a_bytes;
    const uint32_t sLo = sB + SB * b_bytes;
    const uint32_t sHi = sLo + SA * lo_bytes;
    uint8_t* tail = sm + kW6StagingBytes + SA * (a_bytes + lo_bytes + hi_bytes) + SB * b_bytes;
    const uint32_t bar_afull = smem_u32(tail);
    const uint32_t bar_aempty = bar_afull + 8 * kMaxStages;
    const uint32_t bar_pfull = bar_aempty + 8 * kMaxStages;
    const uint32_t bar_bfull = bar_pfull + 8 * kMaxStages;
    const uint32_t bar_bempty = bar_bfull + 8 * kMaxStages;
    const uint32_t bar_tfull = bar_bempty + 8 * kMaxStages;
    const uint32_t bar_tempty = bar_tfull + 16;
    uint32_t* tmem_ptr_s = reinterpret_cast<uint32_t*>(tail + 8 * (5 * kMaxStages + 4));
    volatile int* abort_s = reinterpret_cast<volatile int*>(tmem_ptr_s + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const bool leader = rank == 0;
    const int nclusters = gridDim.x >> 1, cluster_id = blockIdx.x >> 1;

    if (threadIdx.x == 0) {
        for (int i = 0; i < SA; ++i) {
            mbar_init(bar_afull + 8 * i, 1);
            mbar_init(bar_aempty + 8 * i, 1);
            mbar_init(bar_pfull + 8 * i, 1);
        }
        for (int i = 0; i < SB; ++i) {
            mbar_init(bar_bfull + 8 * i, 2 * 4);   // the four warps of one group in each CTA
            mbar_init(bar_bempty + 8 * i, 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(bar_tfull + 8 * i, 1);
            mbar_init(bar_tempty + 8 * i, 2 * kW6EpiWarps);
        }
        *abort_s = 0;
        fence_mbar_init();
        prefetch_tmap(&tmap_a), prefetch_tmap(&tmap_lo), prefetch_tmap(&tmap_hi);
        if (p.tma_store) prefetch_tmap(&tmap_d);
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

    if (warp == 0) {
        // ---------------- TMA producer: A tile (credited to the leader) and this CTA's packed planes ----------------
        if (lane == 0) {
            int sa = 0;
            uint32_t pa = 0;
            bool ok = true;
            for (int t = cluster_id; t < p.num_tiles && ok; t += nclusters) {
                int tm, tn;
                tile_coords(t, p.tiles_m, p.tiles_n, tm, tn);
                const int row_a = tm * (2 * BM * MH) + (int)rank * BM;
                const int row_w = tn * BN + (int)rank * rows_w;
                for (int kb = 0; kb < p.k_iters; ++kb) {
                    if (!mbar_wait_suspended(bar_aempty + 8 * sa, pa ^ 1u, abort_s, ST_TIMEOUT_EMPTY)) { ok = false; break; }
                    mbar_arrive_expect_tx(bar_pfull + 8 * sa, lo_bytes + hi_bytes);
                    tma_load_2d(sLo + sa * lo_bytes, &tmap_lo, kb * 64, row_w, bar_pfull + 8 * sa);
                    tma_load_2d(sHi + sa * hi_bytes, &tmap_hi, kb * 32, row_w, bar_pfull + 8 * sa);
                    if (leader) mbar_arrive_expect_tx(bar_afull + 8 * sa, 2 * a_bytes);
#pragma unroll
                    for (int h = 0; h < MH; ++h)
                        tma_load_2d_pair(sA + sa * a_bytes + h * a_box, &tmap_a, kb * BK, row_a + h * 2 * BM,
                                         mapa_shared(bar_afull + 8 * sa, 0));
                    if (++sa == SA) { sa = 0; pa ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer (leader CTA) ----------------
        if (leader && lane == 0) {
            const uint32_t a_lo0 = umma_desc_lo(sA), b_lo0 = umma_desc_lo(sB);
            const uint32_t a_step = a_bytes >> 4, b_step = b_bytes >> 4;
            const uint32_t idesc = p.idesc;
            int sa = 0, sb = 0;
            uint32_t pa = 0, pb = 0;
            uint32_t a_lo = a_lo0, b_lo = b_lo0;
            int buf = 0;
            uint32_t tphase = 0;
            bool ok = true;
            for (int t = cluster_id; t < p.num_tiles && ok; t += nclusters) {
                {
                    if (!mbar_wait(bar_tempty + 8 * buf, tphase ^ 1u, abort_s, ST_TIMEOUT_TMEM_EMPTY)) break;
                }
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + buf * 256;
                for (int kb = 0; kb < p.k_iters; ++kb) {
                    if (!mbar_wait(bar_afull + 8 * sa, pa, abort_s, ST_TIMEOUT_FULL)) { ok = false; break; }
                    if (!mbar_wait(bar_bfull + 8 * sb, pb, abort_s, ST_TIMEOUT_FULL)) { ok = false; break; }
                    tc_fence_after();
#pragma unroll
                    for (int h = 0; h < MH; ++h) {
                        const uint32_t dh = d_tmem + h * 128, ah = a_lo + h * (a_box >> 4);
                        umma_pair_lo(dh, ah, b_lo, idesc, kb);
                        umma_pair_lo(dh, ah + 2, b_lo + 2, idesc, 1);
                        umma_pair_lo(dh, ah + 4, b_lo + 4, idesc, 1);
                        umma_pair_lo(dh, ah + 6, b_lo + 6, idesc, 1);
                    }
                    umma_commit_pair(bar_bempty + 8 * sb);
                    umma_commit_pair(bar_aempty + 8 * sa);
                    ++sa, a_lo += a_step;
                    if (sa == SA) sa = 0, pa ^= 1u, a_lo = a_lo0;
                    ++sb, b_lo += b_step;
                    if (sb == SB) sb = 0, pb ^= 1u, b_lo = b_lo0;
                }
                if (!ok) break;
                umma_commit_pair(bar_tfull + 8 * buf);
                buf ^= 1;
                if (buf == 0) tphase ^= 1u;
            }
        }
    } else if (warp >= 2 + kW6EpiWarps) {
        // ---------------- unpack warps: groups of four warps take K boxes in turn; one thread per weight row ----------------
        // Every barrier operation and the proxy fence cost a warp on the order of a hundred cycles whatever the amount of
        // data, so a group pays them once per 128 elements of its rows, and the groups overlap one another's waits.
        const int uw = warp - (2 + kW6EpiWarps);
        const int grp = uw >> 2;
        // 64 rows per CTA: two threads per row, 64 elements each
        const int r = 32 * (uw & 1) + lane;                                   // row of the half tile
        const int hf = (uw >> 1) & 1;                                         // which 64 elements of the box
        const bool has_row = MH == 2 || r < rows_w;                           // one half: tiles of 64 and 96 columns too
        const uint32_t bfull_leader = mapa_shared(bar_bfull, 0);
        const int sw_lo = (r >> 1) & 3, sw_hi = (r >> 2) & 1, sw_out = r & 7;
        const bool wide = (x6.srel_pitch & 15) == 0 && ((uintptr_t)x6.s_rel & 15) == 0;   // scale rows readable 16 bytes at a time
        int sa = 0, sb = 0, turn = 0;           // turn: which group takes the current K box
        uint32_t pa = 0, pb = 0;
        bool ok = true;
        for (int t = cluster_id; t < p.num_tiles && ok; t += nclusters) {
            int tm, tn;
            tile_coords(t, p.tiles_m, p.tiles_n, tm, tn);
            const int n = min(tn * BN + (int)rank * rows_w + r, p.N - 1);
            const uint8_t* srow = x6.s_rel + (size_t)n * x6.srel_pitch;
            // scale bytes of four K boxes at a time, fetched four boxes ahead of their use
            uint4 sc_cur = make_uint4(0, 0, 0, 0), sc_next = make_uint4(0, 0, 0, 0);
            auto fetch = [&](int kb4) -> uint4 {     // scales of boxes 4*kb4 .. 4*kb4+3
                uint4 v = make_uint4(0x38383838u, 0x38383838u, 0x38383838u, 0x38383838u);
                if (!has_row) return v;
                if (wide && 4 * kb4 + 4 <= p.k_iters) return gload(reinterpret_cast<const uint4*>(srow) + kb4);
                const uint32_t* s32 = reinterpret_cast<const uint32_t*>(srow) + 4 * kb4;
                const int left = p.k_iters - 4 * kb4;
                if (left > 0) v.x = gload(s32);
                if (left > 1) v.y = gload(s32 + 1);
                if (left > 2) v.z = gload(s32 + 2);
                if (left > 3) v.w = gload(s32 + 3);
                return v;
            };
            sc_next = fetch(0);
            for (int kb = 0; kb < p.k_iters; ++kb) {
                if ((kb & 3) == 0) {
                    sc_cur = sc_next;
                    if (kb + 4 < p.k_iters) sc_next = fetch((kb >> 2) + 1);
                }
                if (turn == grp) {
                    const int q = kb & 3;
                    const uint32_t sr = q == 0 ? sc_cur.x : q == 1 ? sc_cur.y : q == 2 ? sc_cur.z : sc_cur.w;
                    // usually both are complete already: one probe by every lane, the polling form only when not. The expanded
                    // slot first: a parity says nothing about a barrier that is two phases behind, and a free slot means that
                    // every box up to the ring's depth ago has been loaded and multiplied, hence that the packed slot (a ring
                    // at least as deep) is in the phase awaited or the one before.
                    if (!__all_sync(0xffffffffu, mbar_try_wait(bar_bempty + 8 * sb, pb ^ 1u)) &&
                        !mbar_wait_warp(bar_bempty + 8 * sb, pb ^ 1u, abort_s, ST_TIMEOUT_UNPACK)) { ok = false; break; }
                    if (!__all_sync(0xffffffffu, mbar_try_wait(bar_pfull + 8 * sa, pa)) &&
                        !mbar_wait_warp(bar_pfull + 8 * sa, pa, abort_s, ST_TIMEOUT_UNPACK)) { ok = false; break; }
                    {
                        const int rr = has_row ? r : 0;    // lanes beyond the tile's rows redo row 0 (warp votes below) and store nothing
                        const uint8_t* lo = sm + (sLo - base) + sa * lo_bytes + rr * 64;
                        const uint8_t* hi = sm + (sHi - base) + sa * hi_bytes + rr * 32;
                        uint8_t* out = sm + (sB - base) + sb * b_bytes + rr * 128;
                        const uint4 h0 = *reinterpret_cast<const uint4*>(hi + ((hf ^ sw_hi) << 4));
                        const uint32_t hw[4] = {h0.x, h0.y, h0.z, h0.w};
                        const int mode = w6_mode<false>(sr);      // the other thread's half with it: the row's scales of the box
#pragma unroll
                        for (int c = 0; c < 4; ++c) {      // 32 elements = one scale group per 16-byte piece of nibbles
                            if ((c >> 1) != hf) continue;  // the other thread of the row (the same for the whole warp)
                            const int hi_w = 2 * (c & 1);
                            const uint4 l = *reinterpret_cast<const uint4*>(lo + ((c ^ sw_lo) << 4));
                            uint32_t o[8];
                            w6_group_of<false>(mode, l, hw[hi_w], hw[hi_w + 1], (sr >> (8 * c)) & 0xffu, o);
                            if (has_row) {
                                *reinterpret_cast<uint4*>(out + (((2 * c) ^ sw_out) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
                                *reinterpret_cast<uint4*>(out + (((2 * c + 1) ^ sw_out) << 4)) = make_uint4(o[4], o[5], o[6], o[7]);
                            }
                        }
                    }
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_remote(bfull_leader + 8 * sb);
                }
                if (++turn == kW6Groups) turn = 0;
                if (++sa == SA) { sa = 0; pa ^= 1u; }
                if (++sb == SB) { sb = 0; pb ^= 1u; }
            }
        }
    } else {
        // ---------------- epilogue: four warps, each draining every 32-column chunk of its TMEM lane quarter ----------------
        constexpr int kEsz = EPI == EPI_ACC ? 4 : (int)sizeof(OutT);
        constexpr bool kStageVec = kEsz == 2;            // 2-byte outputs: 2 KB chunk + 3 KB of per-column vectors
        const int ew = warp - 2;
        const int quad = warp & 3;
        const int nchunks = BN / 32;
        uint8_t* my_stage = staging + ew * kW6StagingPerWarp;
        const uint32_t my_stage_u32 = smem_u32(my_stage);
        float* my_vec = reinterpret_cast<float*>(my_stage + 2048);   // ws[256] | bias[256] | rscale[256]
        int buf = 0;
        uint32_t tphase = 0;
        for (int t = cluster_id; t < p.num_tiles; t += nclusters) {
            int tm, tn;
            tile_coords(t, p.tiles_m, p.tiles_n, tm, tn);
            const int n0 = tn * BN;
            const bool staged = kStageVec && p.tma_store;
            if (staged) {
                // the tile's columns of ws / bias / rscale, fetched while the mainloop still runs
                if (lane == 0) bulk_wait_read<0>();
                __syncwarp();
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const int n = n0 + 32 * k + lane;
                    const bool in = n < p.N && k < nchunks;
                    my_vec[32 * k + lane] = in ? p.ws[n] : 0.f;
                    my_vec[256 + 32 * k + lane] = (in && p.bias) ? to_f<OutT>(reinterpret_cast<const OutT*>(p.bias)[n]) : 0.f;
                    if (EPI == EPI_RESID)
                        my_vec[512 + 32 * k + lane] = in ? to_f<OutT>(reinterpret_cast<const OutT*>(p.rscale)[n]) : 0.f;
                }
                __syncwarp();
            }
            if (!mbar_wait_warp_relaxed(bar_tfull + 8 * buf, tphase, abort_s, ST_TIMEOUT_TMEM_FULL)) break;
            tc_fence_after();
            uint32_t ra[32];
#pragma unroll 1
            for (int hc = 0; hc < MH * nchunks; ++hc) {
                const int h = MH == 1 ? 0 : hc / nchunks, c = hc - h * nchunks;
                const int row0 = tm * (2 * BM * MH) + h * 2 * BM + (int)rank * BM + quad * 32;
                const int row = row0 + lane;
                const bool row_ok = row < p.M;
                const int rrow = row_ok ? row : p.M - 1;
                const float xs_r = EPI != EPI_ACC ? p.xs[rrow] : 0.f;
                const uint32_t taddr = tmem_base + buf * 256 + h * 128 + ((uint32_t)(quad * 32) << 16);
                tmem_ld32(taddr + c * 32, ra);
                tmem_ld_wait();
                const int col0 = n0 + c * 32;
                if (col0 >= p.N) continue;
                if (p.tma_store) {
                    if constexpr (kStageVec) {
                        uint4 pk[4];
                        chunk_compute16<OutT, EPI, 256>(p, ra, rrow, col0, xs_r, my_vec + 32 * c, pk);
                        if (lane == 0) bulk_wait_read<0>();   // the previous chunk's store has read the buffer
                        __syncwarp();
                        chunk_write16(pk, my_stage, lane);
                    } else {
                        if (lane == 0) bulk_wait_read<0>();
                        __syncwarp();
                        chunk_to_smem<OutT, EPI>(p, ra, rrow, col0, xs_r, my_stage, lane);
                    }
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0) {
                        tma_store_2d(&tmap_d, my_stage_u32, col0, row0);
                        bulk_commit();
                    }
                } else if (row_ok) {
                    chunk_direct<OutT, EPI>(p, ra, row, col0, xs_r);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(mapa_shared(bar_tempty + 8 * buf, 0));
            buf ^= 1;
            if (buf == 0) tphase ^= 1u;
        }
        if (p.tma_store && lane == 0) bulk_wait_read<0>();   // the staged rows have been read; the grid's end completes the writes
    }

    __syncwarp();
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();
    if (*abort_s != 0) {
        for (int i = 0; i < 2000; ++i) __nanosleep(1000);
        if (threadIdx.x == 0) atomicCAS(&g_kernel_status, 0, *abort_s);
        __syncthreads();
    }
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, 512);
    }
}

// ---- few rows: weight rows as the MMA's M, tokens as its N ---------------------------------------------------------------
// Up to 256 tokens (the block on a short clip, a text prompt), or beside a narrow weight, the kernel above is bound by neither
// memory nor the tensor core but by its chain from the packed tile to the MMA: remote arrivals and commits across the CTA pair for every K box,
// an accumulator of 256 rows of which a quarter is used, and no way to share a long K between SMs. Here one CTA takes 128
// weight rows and up to 256 tokens (tcgen05.mma.cta_group::1, M = 128 weight rows, N = tokens rounded up to 16), so every
// barrier is local and nothing is spent on rows that do not exist; a row tile's K is cut between the CTAs of a cluster
// (integer sums: any cut gives the same bits), which leave their accumulators in shared memory and finish a share of the
// outputs each, reading one another's through distributed shared memory: no scratch in global memory, nothing to clear.
// The four linears of a 5120-wide block with FFN 13824 at 64 rows, under ncu: 231 us on the pair kernel, 128 here.
// Warp 0 loads (packed planes and tokens of a K box, one barrier), warp 1 issues the MMAs, warps 2..21 expand: five groups
// of four warps take K boxes in turn (the expansion is what bounds the kernel, a few instructions per code; three groups left the
// issue slots idle two cycles in five). A lane expands one scale group of one row at a time, eight rows of a box to a warp's step, so
// that a tile need not have 128 rows: the host side picks the height (a multiple of eight; the MMA's other rows are never read) that
// spreads the weight's rows evenly over the SMs. 15360 rows are 120 tiles of 128 for 148 SMs, or 148 of 104. Many tokens beside whole tiles have a row a lane
// (w6_row_a_lane()). All warps run the epilogue: a lane owns an output column.
// Back to back, us, tiles of 128 rows with a row a lane and one lane issuing | this: 64 tokens 5120 -> 15360 31.6 | 26.6, 5120 -> 5120 17.1 | 16.0, 5120 -> 13824
// 31.3 | 25.2, 13824 -> 5120 29.7 | 26.3; 200 tokens 38.1 | 38.7, 20.9 | 20.6, 37.7 | 37.0, 34.0 | 33.8; 64 x 1024 -> 64 7.2 | 7.3.
constexpr int kW6RowsWarps = 20;
constexpr int kW6RowsThreads = 32 * (2 + kW6RowsWarps);
constexpr int kW6RowsMaxTokens = 256;
struct W6RowsParams {
    const uint8_t* s_rel;   // [N, K / 32] e4m3
    int srel_pitch;         // K / 32
    int tokens;             // tokens of a tile, a multiple of 16; tiles of tokens lie along the grid's y
    int splits, kps;        // CTAs of a cluster share a row tile's K: kps boxes each
    int sa, sb;             // ring depths: packed planes + tokens, expanded tiles
    int groups;             // expanding groups of four warps in use
    int height;             // weight rows of a tile, a multiple of 8, at most 128
};
__device__ __forceinline__ int ld_shared_cluster(uint32_t addr) {
    int v;
    asm volatile("ld.shared::cluster.b32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}

// TILED: several tiles of tokens. With one the offsets are left out: computed, they cost the epilogue of the activation form 0.4 us.
template <typename OutT, int EPI, bool TILED, bool ROW_A_LANE>
__global__ void __launch_bounds__(kW6RowsThreads, 1)
gemm_w6a8_rows_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_lo,
                      const __grid_constant__ CUtensorMap tmap_hi, const GemmParams p, const W6RowsParams x6) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    const uint32_t base = (raw_addr + 1023u) & ~1023u;     // the same offset in every CTA of the cluster
    uint8_t* sm = smem_raw + (base - raw_addr);
    const int SA = x6.sa, SB = x6.sb, T = x6.tokens;
    const int R = x6.height;
    const uint32_t w_bytes = BM * BK, lo_bytes = (uint32_t)(R * 64 + 1023) & ~1023u, hi_bytes = (uint32_t)R * 32;
    const uint32_t a_bytes = ((uint32_t)T * BK + 1023u) & ~1023u;      // a tile of 16-row pieces, 1024-byte aligned
    const uint32_t sW = base, sA = sW + SB * w_bytes, sLo = sA + SA * a_bytes, sHi = sLo + SA * lo_bytes;
    // barriers sit at the end of the allocation: the accumulators overwrite the rings when these are done with
    uint8_t* tail = sm + SB * w_bytes + SA * (a_bytes + lo_bytes + hi_bytes);
    if (tail < sm + (uint32_t)T * 512u) tail = sm + (uint32_t)T * 512u;
    const uint32_t bar_full = smem_u32(tail), bar_empty = bar_full + 8 * kMaxStages, bar_wfull = bar_empty + 8 * kMaxStages,
                   bar_wempty = bar_wfull + 8 * kMaxStages, bar_tfull = bar_wempty + 8 * kMaxStages;
    uint32_t* tmem_ptr_s = reinterpret_cast<uint32_t*>(tail + 8 * (4 * kMaxStages + 1));
    volatile int* abort_s = reinterpret_cast<volatile int*>(tmem_ptr_s + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t tmem_cols = T <= 32 ? 32u : T <= 64 ? 64u : T <= 128 ? 128u : 256u;
    const int tn = blockIdx.x / x6.splits, rank = blockIdx.x - tn * x6.splits;     // a cluster = the slices of one row tile
    const int n0 = tn * R;
    const int t0 = TILED ? blockIdx.y * T : 0, rows = TILED ? min(p.M - t0, T) : p.M;      // this tile's tokens
    const int k0 = rank * x6.kps, k1 = min(k0 + x6.kps, p.k_iters);                // never empty: the host side sees to it

    if (threadIdx.x == 0) {
        for (int i = 0; i < SA; ++i) mbar_init(bar_full + 8 * i, 1), mbar_init(bar_empty + 8 * i, 1);
        for (int i = 0; i < SB; ++i) mbar_init(bar_wfull + 8 * i, 4), mbar_init(bar_wempty + 8 * i, 1);
        mbar_init(bar_tfull, 1);
        *abort_s = 0;
        fence_mbar_init();
        prefetch_tmap(&tmap_a), prefetch_tmap(&tmap_lo), prefetch_tmap(&tmap_hi);
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(tmem_ptr_s), tmem_cols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_wait();
    const uint32_t tmem_base = *tmem_ptr_s;

    if (warp == 0) {
        if (lane == 0) {
            int s = 0;
            uint32_t ph = 0;
            for (int kb = k0; kb < k1; ++kb) {
                if (!mbar_wait(bar_empty + 8 * s, ph ^ 1u, abort_s, ST_TIMEOUT_EMPTY)) break;
                mbar_arrive_expect_tx(bar_full + 8 * s, (uint32_t)(T * BK + R * 96));
                tma_load_2d(sLo + s * lo_bytes, &tmap_lo, kb * 64, n0, bar_full + 8 * s);
                tma_load_2d(sHi + s * hi_bytes, &tmap_hi, kb * 32, n0, bar_full + 8 * s);
                tma_load_2d(sA + s * a_bytes, &tmap_a, kb * BK, t0, bar_full + 8 * s);
                if (++s == SA) s = 0, ph ^= 1u;
            }
        }
    } else if (warp == 1) {
        const bool one = elect_one();          // the whole warp walks the boxes, one lane issues: see the one-CTA int8 kernel
        const uint32_t idesc = p.idesc;
        int sa = 0, sb = 0;
        uint32_t pa = 0, pb = 0;
        bool ok = true;
        for (int kb = k0; kb < k1; ++kb) {
            if (!__all_sync(0xffffffffu, mbar_wait(bar_full + 8 * sa, pa, abort_s, ST_TIMEOUT_FULL) &&
                                             mbar_wait(bar_wfull + 8 * sb, pb, abort_s, ST_TIMEOUT_FULL))) { ok = false; break; }
            tc_fence_after();
            const uint32_t dw = umma_desc_lo(sW + sb * w_bytes), da = umma_desc_lo(sA + sa * a_bytes);
            if (one) {
#pragma unroll
                for (int k = 0; k < BK / UMMA_K; ++k) umma_i8_lo(tmem_base, dw + 2 * k, da + 2 * k, idesc, (kb - k0) | k);
                umma_commit(bar_wempty + 8 * sb);
                umma_commit(bar_empty + 8 * sa);
            }
            __syncwarp();
            if (++sa == SA) sa = 0, pa ^= 1u;
            if (++sb == SB) sb = 0, pb ^= 1u;
        }
        if (ok && one) umma_commit(bar_tfull);
    } else {
        const int uw = warp - 2, grp = uw >> 2;
        bool ok = true;
        if constexpr (ROW_A_LANE) {
            const int r = 32 * (uw & 3) + lane;                        // weight row of the tile
            const uint8_t* srow = x6.s_rel + (size_t)min(n0 + r, p.N - 1) * x6.srel_pitch;
            const bool wide = (x6.srel_pitch & 15) == 0 && ((uintptr_t)x6.s_rel & 15) == 0;   // scale rows readable 16 bytes at a time
            auto fetch = [&](int kb4) -> uint4 {                       // scales of boxes 4 kb4 .. 4 kb4 + 3
                if (wide) return gload(reinterpret_cast<const uint4*>(srow) + kb4);
                uint4 v = make_uint4(0, 0, 0, 0);
                const uint32_t* s32 = reinterpret_cast<const uint32_t*>(srow) + 4 * kb4;
                const int left = p.k_iters - 4 * kb4;
                if (left > 0) v.x = gload(s32);
                if (left > 1) v.y = gload(s32 + 1);
                if (left > 2) v.z = gload(s32 + 2);
                if (left > 3) v.w = gload(s32 + 3);
                return v;
            };
            const int sw_lo = (r >> 1) & 3, sw_hi = (r >> 2) & 1, sw_out = r & 7;
            int sa = 0, sb = 0, turn = 0;
            uint32_t pa = 0, pb = 0;
            uint4 sc_cur = make_uint4(0, 0, 0, 0), sc_next = fetch(k0 >> 2);
            for (int kb = grp < x6.groups ? k0 : k1; kb < k1; ++kb) {
                if ((kb & 3) == 0 || kb == k0) {
                    sc_cur = sc_next;
                    if ((kb & ~3) + 4 < k1) sc_next = fetch((kb >> 2) + 1);
                }
                if (turn == grp) {
                    const int q = kb & 3;
                    const uint32_t sr = q == 0 ? sc_cur.x : q == 1 ? sc_cur.y : q == 2 ? sc_cur.z : sc_cur.w;
                    // the expanded slot first, as above: groups <= sb <= sa keeps every awaited phase the current or the last one
                    if (!__all_sync(0xffffffffu, mbar_try_wait(bar_wempty + 8 * sb, pb ^ 1u)) &&
                        !mbar_wait_warp(bar_wempty + 8 * sb, pb ^ 1u, abort_s, ST_TIMEOUT_UNPACK)) { ok = false; break; }
                    if (!__all_sync(0xffffffffu, mbar_try_wait(bar_full + 8 * sa, pa)) &&
                        !mbar_wait_warp(bar_full + 8 * sa, pa, abort_s, ST_TIMEOUT_UNPACK)) { ok = false; break; }
                    const uint8_t* lo = sm + (sLo - base) + sa * lo_bytes + r * 64;
                    const uint8_t* hi = sm + (sHi - base) + sa * hi_bytes + r * 32;
                    uint8_t* out = sm + sb * w_bytes + r * 128;
                    const uint4 h0 = *reinterpret_cast<const uint4*>(hi + (sw_hi << 4)), h1 = *reinterpret_cast<const uint4*>(hi + ((1 ^ sw_hi) << 4));
                    const uint32_t hw[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
                    auto expand = [&](auto mode) {
#pragma unroll
                        for (int c = 0; c < 4; ++c) {                  // 32 codes = one scale group per 16-byte piece of nibbles
                            const uint4 l = *reinterpret_cast<const uint4*>(lo + ((c ^ sw_lo) << 4));
                            uint32_t o[8];
                            w6_group<decltype(mode)::value>(l, hw[2 * c], hw[2 * c + 1], (sr >> (8 * c)) & 0xffu, o);
                            *reinterpret_cast<uint4*>(out + (((2 * c) ^ sw_out) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
                            *reinterpret_cast<uint4*>(out + (((2 * c + 1) ^ sw_out) << 4)) = make_uint4(o[4], o[5], o[6], o[7]);
                        }
                    };
                    const int mode = w6_mode(sr);
                    if (mode == W6_MID) expand(std::integral_constant<int, W6_MID>());
                    else if (mode == W6_SMALL) expand(std::integral_constant<int, W6_SMALL>());
                    else if (mode == W6_UNIT) expand(std::integral_constant<int, W6_UNIT>());
                    else expand(std::integral_constant<int, W6_ANY>());
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_wfull + 8 * sb);
                }
                if (++turn == x6.groups) turn = 0;
                if (++sa == SA) sa = 0, pa ^= 1u;
                if (++sb == SB) sb = 0, pb ^= 1u;
            }
        } else {
            // Step i of a box: its rows 8 i .. 8 i + 7; lane = (row, scale group). Warp j of a group takes every fourth step, counted from
            // where its last box left off, so that all four do as much.
            const int steps = R / 8, c = lane & 3;
            auto row_of = [&](int i) { return 8 * i + (lane >> 2); };
            // where a lane's pieces lie among a step's rows: the swizzles look at the row's low three bits, which are the lane's
            const uint32_t l8 = lane >> 2, lo_at = l8 * 64 + ((c ^ ((l8 >> 1) & 3)) << 4), hi_at = l8 * 32 + (((c >> 1) ^ (l8 >> 2)) << 4) + ((c & 1) << 3),
                           out_at = l8 * 128 + (((2 * c) ^ l8) << 4);
            const int out_next = (int)((out_at ^ 16u) - out_at);
            auto first = [&](int kb) { return ((uw & 3) + 4 - (kb / x6.groups * steps & 3)) & 3; };
            const int g = x6.groups;
            // The scales of four turns at a time, a word (a row's four groups) a load: lane (row, c) requests those of its rows for the c-th of the turns and
            // the lanes of a row hand them round. The first turn's come by themselves, before what can wait.
            uint32_t sc_cur[4], sc_next[4];
            const uint32_t pick = (uint32_t)(c | (c + 4) << 4);        // byte c of two words
            auto fetch = [&](uint32_t (&w)[4], int k) {                // of box k
                const int i0 = first(k);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    w[j] = 0x38383838u;
                    if (i0 + 4 * j < steps && k < k1) w[j] = gload(reinterpret_cast<const uint32_t*>(x6.s_rel + (size_t)min(n0 + row_of(i0 + 4 * j), p.N - 1) * x6.srel_pitch) + k);
                }
            };
            int sa = grp, sb = grp;                                    // a group beyond the boxes has none
            uint32_t pa = 0, pb = 0;
            fetch(sc_cur, k0 + grp);
            fetch(sc_next, k0 + grp + (c + 1) * g);
            for (int kb = grp < g ? k0 + grp : k1, turn = 0; kb < k1; kb += g, ++turn) {
                if ((turn & 3) == 1) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) sc_cur[j] = sc_next[j];
                    fetch(sc_next, kb + (c + 4) * g);
                }
                uint32_t w[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) w[j] = __shfl_sync(0xffffffffu, sc_cur[j], (lane & 28) | ((turn + 3) & 3));
                const uint32_t sc = __byte_perm(__byte_perm(w[0], w[1], pick), __byte_perm(w[2], w[3], pick), 0x5410);
                // the expanded slot first, as above: groups <= sb <= sa keeps every awaited phase the current or the last one
                if (!__all_sync(0xffffffffu, mbar_try_wait(bar_wempty + 8 * sb, pb ^ 1u)) &&
                    !mbar_wait_warp(bar_wempty + 8 * sb, pb ^ 1u, abort_s, ST_TIMEOUT_UNPACK)) { ok = false; break; }
                if (!__all_sync(0xffffffffu, mbar_try_wait(bar_full + 8 * sa, pa)) &&
                    !mbar_wait_warp(bar_full + 8 * sa, pa, abort_s, ST_TIMEOUT_UNPACK)) { ok = false; break; }
                const int i0 = first(kb);
                const uint8_t* lo = sm + (sLo - base) + sa * lo_bytes + i0 * 512 + lo_at;
                const uint8_t* hi = sm + (sHi - base) + sa * hi_bytes + i0 * 256 + hi_at;
                uint8_t* out = sm + sb * w_bytes + i0 * 1024 + out_at;
                // Up to four steps in a straight line: one by one, a warp waits for each (64 x 5120 -> 15360 27.5 us, 26.5 with the next line's scales).
                uint32_t s4 = sc;
                auto expand = [&](auto mode) {
                    auto lines = [&](auto count) {
                        constexpr int kN = decltype(count)::value;
                        uint4 l[kN];
                        uint2 h[kN];
#pragma unroll
                        for (int j = 0; j < kN; ++j) l[j] = *reinterpret_cast<const uint4*>(lo + 2048 * j), h[j] = *reinterpret_cast<const uint2*>(hi + 1024 * j);
#pragma unroll
                        for (int j = 0; j < kN; ++j) {
                            uint32_t o[8];
                            w6_group<decltype(mode)::value>(l[j], h[j].x, h[j].y, (s4 >> (8 * j)) & 0xffu, o);
                            *reinterpret_cast<uint4*>(out + 4096 * j) = make_uint4(o[0], o[1], o[2], o[3]);
                            *reinterpret_cast<uint4*>(out + 4096 * j + out_next) = make_uint4(o[4], o[5], o[6], o[7]);
                        }
                    };
                    if (i0 + 12 < steps) lines(std::integral_constant<int, 4>());
                    else if (i0 + 8 < steps) lines(std::integral_constant<int, 3>());
                    else lines(std::integral_constant<int, 2>());      // tiles have eight steps or more
                };
                const int mode = w6_mode(sc);
                if (mode == W6_MID) expand(std::integral_constant<int, W6_MID>());
                else if (mode == W6_SMALL) expand(std::integral_constant<int, W6_SMALL>());
                else if (mode == W6_UNIT) expand(std::integral_constant<int, W6_UNIT>());
                else expand(std::integral_constant<int, W6_ANY>());
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_wfull + 8 * sb);
                sa += g, sb += g;
                if (sa >= SA) sa -= SA, pa ^= 1u;
                if (sb >= SB) sb -= SB, pb ^= 1u;
            }
        }
        // accumulators to shared memory, [token][weight row] int32, over the rings (all copies have landed and all MMAs have
        // read them when the accumulator is complete)
        if (ok && mbar_wait_warp(bar_tfull, 0, abort_s, ST_TIMEOUT_TMEM_FULL)) {
            tc_fence_after();
            const int quad = warp & 3;                             // TMEM lane quarter this warp may read
            int* red = reinterpret_cast<int*>(sm) + quad * 32 + lane;
            for (int c = grp; c < T / 16; c += kW6RowsWarps / 4) {
                uint32_t v[16];
                tmem_ld16(tmem_base + ((uint32_t)(quad * 32) << 16) + c * 16, v);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 16; ++j) red[(c * 16 + j) * BM] = (int)v[j];
            }
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();
    if (warp >= 2 && *abort_s == 0) {
        // eight tokens x 32 columns at a time, dealt out over the cluster's warps
        const int quads = (rows + 7) / 8 * 4;
        const int64_t tile = (int64_t)t0 * p.N;                    // the tile's first output
        for (int u = rank + x6.splits * (warp - 2); u < quads; u += x6.splits * kW6RowsWarps) {
            const int quad = u & 3, m0 = (u >> 2) * 8;
            const int n = n0 + quad * 32 + lane;
            if (n >= p.N || quad * 32 + lane >= R) continue;
            const uint32_t src = base + (uint32_t)(m0 * BM + quad * 32 + lane) * 4u;
            int acc[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[i] = 0;
            for (int s = 0; s < x6.splits; ++s) {
                const uint32_t a = mapa_shared(src, (uint32_t)s);
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[i] += ld_shared_cluster(a + i * BM * 4);      // rows up to the next multiple of 16 exist
            }
            if constexpr (EPI == EPI_ACC) {
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (m0 + i < rows) reinterpret_cast<int*>(p.D)[tile + (int64_t)(m0 + i) * p.N + n] = acc[i];
            } else {
                const float ws = p.ws[n], bias = p.bias ? to_f<OutT>(reinterpret_cast<const OutT*>(p.bias)[n]) : 0.f;
                const float rs = EPI == EPI_RESID ? to_f<OutT>(reinterpret_cast<const OutT*>(p.rscale)[n]) : 0.f;
                float rr[8];
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    rr[i] = EPI == EPI_RESID && m0 + i < rows ? to_f<OutT>(reinterpret_cast<const OutT*>(p.resid)[tile + (int64_t)(m0 + i) * p.N + n]) : 0.f;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    if (m0 + i >= rows) break;
                    reinterpret_cast<OutT*>(p.D)[tile + (int64_t)(m0 + i) * p.N + n] =
                        from_f<OutT>(epilogue1<OutT, EPI>(acc[i], p.xs[t0 + m0 + i], ws, bias, rs, rr[i], p.act));
                }
            }
        }
    }
    __syncwarp();
    cluster_sync_all();            // nobody leaves while another CTA may read its accumulators
    if (*abort_s != 0) {
        for (int i = 0; i < 2000; ++i) __nanosleep(1000);
        if (threadIdx.x == 0) atomicCAS(&g_kernel_status, 0, *abort_s);
        __syncthreads();
    }
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, tmem_cols);
    }
}

// ---- host side ------------------------------------------------------------------------------------------------------
// Tensor map of one plane of the packed rows: `cols` bytes per row at `pitch` bytes, boxes of box_x bytes x box_rows.
bool make_plane_tmap(CUtensorMap* tm, const void* ptr, int64_t rows, int64_t cols, int64_t pitch, int box_x, int box_rows,
                     CUtensorMapSwizzle swz) {
    EncodeTiledFn enc = encode_fn();
    if (!enc) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)pitch};
    const cuuint32_t box[2] = {(cuuint32_t)box_x, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return enc(tm, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(ptr), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, swz, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <typename OutT, int EPI, int MH>
int launch_w6_mh(const CUtensorMap& ta, const CUtensorMap& tlo, const CUtensorMap& thi, const CUtensorMap& td,
                 const GemmParams& p, const W6Extra& x6, int grid, cudaStream_t st) {
    auto kern = gemm_w6a8_pair_kernel<OutT, EPI, MH>;
    static std::atomic<uint64_t> configured{0};
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = 1ull << (dev & 63);
    if (!(configured.load(std::memory_order_acquire) & bit)) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
        if (e != cudaSuccess) return (int)e;
        configured.fetch_or(bit, std::memory_order_release);
    }
    return launch_pdl(kern, dim3(grid), kW6Threads, kSmemBytes, st, ta, tlo, thi, td, p, x6);
}

template <typename OutT, int EPI>
int launch_w6(const CUtensorMap& ta, const CUtensorMap& tlo, const CUtensorMap& thi, const CUtensorMap& td,
              const GemmParams& p, const W6Extra& x6, int mh, int grid, cudaStream_t st) {
    return mh == 2 ? launch_w6_mh<OutT, EPI, 2>(ta, tlo, thi, td, p, x6, grid, st)
                   : launch_w6_mh<OutT, EPI, 1>(ta, tlo, thi, td, p, x6, grid, st);
}

template <typename OutT, int EPI, bool TILED, bool ROW_A_LANE>
int launch_w6_rows_tiled(const CUtensorMap& ta, const CUtensorMap& tlo, const CUtensorMap& thi, const GemmParams& p, const W6RowsParams& x6,
                         size_t smem, cudaStream_t st) {
    auto kern = gemm_w6a8_rows_kernel<OutT, EPI, TILED, ROW_A_LANE>;
    static std::atomic<uint64_t> configured{0};
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = 1ull << (dev & 63);
    if (!(configured.load(std::memory_order_acquire) & bit)) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
        if (e != cudaSuccess) return (int)e;
        configured.fetch_or(bit, std::memory_order_release);
    }
    return launch_pdl_cluster(kern, dim3(p.tiles_n * x6.splits, p.tiles_m), kW6RowsThreads, smem, st, x6.splits, ta, tlo, thi, p, x6);
}

template <typename OutT, int EPI>
int launch_w6_rows(const CUtensorMap& ta, const CUtensorMap& tlo, const CUtensorMap& thi, const GemmParams& p, const W6RowsParams& x6,
                   size_t smem, cudaStream_t st) {
    return p.tiles_m > 1 ? launch_w6_rows_tiled<OutT, EPI, true, false>(ta, tlo, thi, p, x6, smem, st)
           : w6_row_a_lane(x6.tokens, x6.height, true) ? launch_w6_rows_tiled<OutT, EPI, false, true>(ta, tlo, thi, p, x6, smem, st)
                                                 : launch_w6_rows_tiled<OutT, EPI, false, false>(ta, tlo, thi, p, x6, smem, st);
}

// Clusters of 1 .. 8 CTAs of the kernel above that the current device holds at once ([0] unused): asked of the runtime once per device.
const int* w6_rows_clusters() {
    static int count[64][kW6RowsMaxSplits + 1];
    static std::mutex mu;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(mu);
    int* c = count[dev & 63];
    if (c[0] == 0) {
        auto kern = gemm_w6a8_rows_kernel<bf16, EPI_PLAIN, false, false>;
        c[1] = device_sm_count(dev);
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes) == cudaSuccess) {
            for (int i = 2; i <= kW6RowsMaxSplits; ++i) {
                cudaLaunchConfig_t cfg = {};
                cfg.gridDim = dim3(i), cfg.blockDim = dim3(kW6RowsThreads), cfg.dynamicSmemBytes = kSmemBytes;
                cudaLaunchAttribute at;
                at.id = cudaLaunchAttributeClusterDimension;
                at.val.clusterDim.x = (unsigned)i, at.val.clusterDim.y = 1, at.val.clusterDim.z = 1;
                cfg.attrs = &at, cfg.numAttrs = 1;
                if (cudaOccupancyMaxActiveClusters(&c[i], kern, &cfg) != cudaSuccess) c[i] = 0;
            }
        }
        (void)cudaGetLastError();
        c[0] = 1;
    }
    return c;
}

int run_w6_rows(int epi, const int8_t* A, const uint8_t* Wq6, const uint8_t* s_rel, GemmParams& p, int out_dt, cudaStream_t st) {
    const int64_t M = p.M, N = p.N, K = p.K;
    W6RowsParams x6{s_rel, (int)(K / 32), 0, 1, p.k_iters, 0, 0, 0, BM};
    int dev = 0;
    cudaGetDevice(&dev);
    const W6RowsPlan plan = w6_rows_plan(dev, M, N, p.k_iters, w6_rows_clusters());
    x6.tokens = plan.tokens, x6.splits = plan.splits, x6.kps = plan.kps, x6.height = plan.height;
    p.tiles_m = (int)((M + x6.tokens - 1) / x6.tokens);
    p.tiles_n = (int)((N + x6.height - 1) / x6.height);
    p.idesc = umma_idesc_i8(BM, x6.tokens);
    const int a_bytes = (x6.tokens * BK + 1023) & ~1023;
    const int stage = a_bytes + ((x6.height * 64 + 1023) & ~1023) + x6.height * 32;
    // rings: as many expanded tiles as the packed ring beside them is deep (see the waits of the expanding warps), six at most
    for (x6.sb = 6; x6.sb > 1; --x6.sb) {
        x6.sa = (kSmemBytes - 1024 - kTailBytes - x6.sb * BM * BK) / stage;
        if (x6.sa >= x6.sb) break;
    }
    if (x6.sa > kMaxStages) x6.sa = kMaxStages;
    x6.groups = x6.sb < kW6RowsWarps / 4 ? x6.sb : kW6RowsWarps / 4;
    if (x6.sa > x6.kps) x6.sa = x6.kps;      // no slot is used twice then
    size_t rings = (size_t)x6.sb * BM * BK + (size_t)x6.sa * stage;
    if (rings < (size_t)x6.tokens * BM * 4) rings = (size_t)x6.tokens * BM * 4;
    const size_t smem = 1024 + rings + kTailBytes;
    const int64_t pitch = 3 * K / 4;
    CUtensorMap ta, tlo, thi;
    if (!make_operand_tmap(&ta, A, M, K, x6.tokens)) return -203;
    if (!make_plane_tmap(&tlo, Wq6, N, K / 2, pitch, 64, x6.height, CU_TENSOR_MAP_SWIZZLE_64B)) return -203;
    if (!make_plane_tmap(&thi, Wq6 + K / 2, N, K / 4, pitch, 32, x6.height, CU_TENSOR_MAP_SWIZZLE_32B)) return -203;
    if (epi == EPI_ACC) return launch_w6_rows<float, EPI_ACC>(ta, tlo, thi, p, x6, smem, st);
#define W6_ROWS_DISPATCH(T)                                                                    \
    (epi == EPI_RESID ? launch_w6_rows<T, EPI_RESID>(ta, tlo, thi, p, x6, smem, st)            \
     : epi == EPI_ACT ? launch_w6_rows<T, EPI_ACT>(ta, tlo, thi, p, x6, smem, st)              \
                      : launch_w6_rows<T, EPI_PLAIN>(ta, tlo, thi, p, x6, smem, st))
    if (out_dt == DT_F32) return W6_ROWS_DISPATCH(float);
    if (out_dt == DT_F16) return W6_ROWS_DISPATCH(half);
    return W6_ROWS_DISPATCH(bf16);
#undef W6_ROWS_DISPATCH
}

int run_w6_gemm(int epi, const int8_t* A, const uint8_t* Wq6, const uint8_t* s_rel, const float* xs, const float* ws,
                const void* bias, const void* rscale, const void* resid, void* D, int64_t M, int64_t N, int64_t K, int G,
                int out_dt, cudaStream_t st, int act = 0) {
    if (M == 0 || N == 0) return 0;
    if (G != 32) return -206;                                  // the fused unpack is built for the reference's group size
    if (epi == EPI_RESID && (!rscale || !resid)) return -201;
    if (epi != EPI_ACC && (out_dt < 0 || out_dt > 2)) return -200;
    if (M > INT32_MAX || N > INT32_MAX || K > INT32_MAX) return -200;
    // whole 128-element K boxes; planes and scale rows must be addressable by TMA / 32-bit loads
    if (K <= 0 || (K % 128) != 0 || ((uintptr_t)A & 15) || ((uintptr_t)Wq6 & 15) || ((uintptr_t)s_rel & 3)) return -202;
    int dev = 0;
    cudaGetDevice(&dev);
    const int clusters = device_sm_count(dev) / 2;
    GemmParams p{};
    p.xs = xs, p.ws = ws, p.bias = bias, p.rscale = rscale, p.resid = resid, p.D = D;
    p.M = (int)M, p.N = (int)N, p.K = (int)K;
    p.act = act;
    p.act_lut = nullptr;
    const int esz = epi == EPI_ACC ? 4 : (out_dt == DT_F32 ? 4 : 2);
    p.k_iters = (int)(K / BK);
    // Up to 256 rows, and beside a weight narrower than the pair kernel's 128 columns up to 4 K rows: that kernel gives a cluster
    // the whole K of 256 rows, the other one spreads K over more SMs but starts and ends once per 256 rows or fewer. 64 columns, the
    // few-rows kernel | one half: K = 1024, 2048 rows 8.7 | 10.2 us, 4608 10.4 | 10.3, 8448 11.7 | 10.6; K = 2560, 8448 rows 14.8 |
    // 16.1, 12288 16.4 | 16.2; K = 5120, 300 rows 9.9 | 24.1, 16896 23.9 | 25.9.
    const bool narrow = N < BM;
    if (M <= kW6RowsMaxTokens || (narrow && M <= 4 * K && M <= 65535 * 64)) return run_w6_rows(epi, A, Wq6, s_rel, p, out_dt, st);
    auto al16 = [](const void* q) { return ((uintptr_t)q & 15) == 0; };
    p.vec_ok = (N % 8 == 0) && al16(D) && al16(ws) && al16(bias) && al16(rscale) && al16(resid);
    p.tma_store = al16(D) && ((N * esz) % 16 == 0);
    p.ksub = 1;
    const int mh = narrow ? 1 : 2, bn = narrow ? choose_bn(M, N, clusters) : 128;
    p.bn = bn;
    p.idesc = umma_idesc_i8(2 * BM, bn);
    const int stage_bytes = mh * BM * BK + (bn / 2) * (64 + 32);     // A boxes + packed planes; the expanded ring is separate
    const int sbs = kW6BStages;
    const int stages = (kSmemBytes - 1024 - 512 - kW6StagingBytes - sbs * (bn / 2) * BK) / stage_bytes;
    p.stages = stages > kMaxStages ? kMaxStages : stages;
    p.tiles_m = (int)((M + 2 * BM * mh - 1) / (2 * BM * mh));
    p.tiles_n = (int)((N + bn - 1) / bn);
    p.num_tiles = p.tiles_m * p.tiles_n;
    p.whole_tiles = p.num_tiles, p.num_items = p.num_tiles, p.kps = p.k_iters;
    const int64_t pitch = 3 * K / 4;
    CUtensorMap ta, tlo, thi, td;
    if (!make_operand_tmap(&ta, A, M, K, BM)) return -203;
    if (!make_plane_tmap(&tlo, Wq6, N, K / 2, pitch, 64, bn / 2, CU_TENSOR_MAP_SWIZZLE_64B)) return -203;
    if (!make_plane_tmap(&thi, Wq6 + K / 2, N, K / 4, pitch, 32, bn / 2, CU_TENSOR_MAP_SWIZZLE_32B)) return -203;
    if (p.tma_store) {
        if (!make_output_tmap(&td, D, M, N, esz)) return -203;
    } else {
        td = ta;
    }
    W6Extra x6{s_rel, (int)(K / 32), sbs};
    const int grid = 2 * (p.num_tiles < clusters ? p.num_tiles : clusters);
    if (epi == EPI_ACC) return launch_w6<float, EPI_ACC>(ta, tlo, thi, td, p, x6, mh, grid, st);
#define W6_DISPATCH(T)                                                                                   \
    (epi == EPI_RESID ? launch_w6<T, EPI_RESID>(ta, tlo, thi, td, p, x6, mh, grid, st)                      \
     : epi == EPI_ACT ? launch_w6<T, EPI_ACT>(ta, tlo, thi, td, p, x6, mh, grid, st)                        \
                      : launch_w6<T, EPI_PLAIN>(ta, tlo, thi, td, p, x6, mh, grid, st))
    if (out_dt == DT_F32) return W6_DISPATCH(float);
    if (out_dt == DT_F16) return W6_DISPATCH(half);
    return W6_DISPATCH(bf16);
#undef W6_DISPATCH
}
