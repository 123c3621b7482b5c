// How the few-rows W6A8 GEMM (gemm_w6.inl) cuts a problem: tokens of a tile, rows of a weight tile, K slices. Host code without CUDA.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdint>

namespace b200q {
constexpr int kW6RowsMaxSplits = 8, kW6RowsTall = 128;
struct W6RowsPlan {
    int tokens, splits, kps, height;
};
// A lane expands one row of a box instead of one scale group of one row at a time: straight-line code for tiles of whole height, which a warp gets
// through in less time, at the price of issue slots. From 112 tokens on the rings have five slots or fewer and wait for the expansion of a box: 2048 to
// 13824 columns, whole tiles, one tile of tokens, in 137 plans each: 128 and 160 tokens 2 % less time, 208 and 256 tokens 5 and 4 %; at 64 tokens a box takes 5 % more.
inline bool w6_row_a_lane(int tokens, int height, bool one_tile) { return one_tile && tokens > 112 && height == kW6RowsTall; }

// Rounds of clusters times the cost of one, in K boxes. A CTA's rings take a whole SM and a cluster has to lie in one GPC, so the
// device holds fewer clusters than SMs / s (`clusters`: 148, 74, 45, 33, 26, 22, 15, 15 of 1 to 8 CTAs); a second round costs as much as the first. A box
// costs the longer of its expansion, two steps of eight rows and those of the tile, and of the wait for a slot of the ring, which grows with the tokens
// in it (the two run into one another: fourth powers). The constants are fitted to 19 sizes of N and K (512 x 14336 to 20480 x 5120) at 12 to
// 256 tokens, every height, slice count and up to four tiles of tokens: the plan chosen is 0.6 % above the best of them on average, 9 % at most (180 x 8192 -> 2048);
// without the tokens it was 1.1 % and 17 %. Narrower token tiles expand the weight once more each, which pays where SMs would idle (256 x 120 x 1024 in
// four: 7.9 us, 10.9 in one); they have to promise 5 %.
inline W6RowsPlan w6_rows_search(int64_t M, int64_t N, int k_iters, const int* clusters) {
    W6RowsPlan r{0, 1, k_iters, kW6RowsTall};
    int slices[kW6RowsMaxSplits], boxes[kW6RowsMaxSplits], n = 0;
    for (int s = 1; s <= kW6RowsMaxSplits && s <= k_iters; ++s) {
        const int k = (k_iters + s - 1) / s;
        if ((k_iters + k - 1) / k != s || clusters[s] < 1) continue;          // a slice would be empty; no such cluster fits
        slices[n] = s, boxes[n++] = k;
    }
    double best = 1e30;
    int last = 0;
    for (const int width : {256, 192, 128, 96, 64}) {
        const int64_t tiles_m = (M + width - 1) / width;
        const int tokens = (int)(((M + tiles_m - 1) / tiles_m + 15) / 16 * 16);      // equal shares, at most 256
        if (tokens == last) continue;
        last = tokens;
        double cost = 1e30;
        int at = 0, height = kW6RowsTall;
        const double wait = 0.4 + 0.0025 * tokens, wait4 = wait * wait * wait * wait;
        for (int h = kW6RowsTall; h >= 64; h -= 8) {
            const double steps = (h / 8 + 2) / 18.0;
            const double box = std::sqrt(std::sqrt(steps * steps * steps * steps + wait4)) * (w6_row_a_lane(tokens, h, tiles_m == 1) ? 0.9 : 1.0);
            const int64_t tiles = (N + h - 1) / h * tiles_m;
            for (int i = 0; i < n; ++i) {
                const int s = slices[i];
                const double rounds = (double)((tiles + clusters[s] - 1) / clusters[s]);
                const double c = rounds * (boxes[i] * box + (s == 1 ? 8 + tokens / 28.0 : 10.5 + tokens / (s <= 4 ? 40.0 : 26.0)));
                if (c < cost) cost = c, at = i, height = h;
            }
        }
        if (n && cost < 0.95 * best) best = cost, r = W6RowsPlan{tokens, slices[at], boxes[at], height};
    }
    return r;
}
// The same from a thread's memory of the sizes that it has met: a plan depends on nothing else, and a step of a model asks for the same few
// again and again. The search takes 0.4 us at up to 64 rows and 1.3 at 256, a call in all about 3.
inline W6RowsPlan w6_rows_plan(int dev, int64_t M, int64_t N, int k_iters, const int* clusters) {
    struct Entry {
        int dev, k_iters;
        int64_t M, N;
        W6RowsPlan plan;
    };
    static thread_local Entry memory[64] = {};          // k_iters 0: empty
    const uint64_t mix = ((uint64_t)M * 0x9E3779B97F4A7C15ull) ^ ((uint64_t)N * 0xC2B2AE3D27D4EB4Full) ^ ((uint64_t)k_iters * 0x165667B19E3779F9ull) ^ (uint64_t)dev << 56;
    Entry& e = memory[mix >> 58];
    if (e.k_iters != k_iters || e.M != M || e.N != N || e.dev != dev) e = Entry{dev, k_iters, M, N, w6_rows_search(M, N, k_iters, clusters)};
    return e.plan;
}
}  // namespace b200q
