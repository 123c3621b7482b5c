"""The plan of the few-rows W6A8 GEMM (csrc/w6_rows_plan.h, host code without CUDA): valid for every size, the best by its own cost, and worked
out once per size and thread, since a call in all takes about three microseconds of host time."""
from __future__ import annotations

import os
import random
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "comfyui-backend-but-rust_b200", "csrc")
PROGRAM = r"""
#include <chrono>
#include <cstdio>
#include <thread>
#include "w6_rows_plan.h"
using namespace b200q;
static const int clusters[9] = {1, 148, 74, 45, 33, 26, 22, 15, 15};
template <typename F> double ns(F f) {
    double best = 1e30;
    for (int r = 0; r < 7; ++r) {
        const auto t0 = std::chrono::steady_clock::now();
        int sum = 0;
        for (int i = 0; i < 2000; ++i) sum += f(i);
        const double t = std::chrono::duration<double, std::nano>(std::chrono::steady_clock::now() - t0).count() / 2000;
        if (t < best && sum != 0x7fffffff) best = t;
    }
    return best;
}
static volatile long long kM = 256;
int main() {
    long long M, N;
    int k;
    while (scanf("%lld %lld %d", &M, &N, &k) == 3) {
        const W6RowsPlan a = w6_rows_search(M, N, k, clusters), b = w6_rows_plan(0, M, N, k, clusters), c = w6_rows_plan(0, M, N, k, clusters);
        W6RowsPlan d{};
        std::thread([&] { d = w6_rows_plan(0, M, N, k, clusters); }).join();
        const bool same = !__builtin_memcmp(&a, &b, sizeof a) && !__builtin_memcmp(&a, &c, sizeof a) && !__builtin_memcmp(&a, &d, sizeof a);
        printf("%d %d %d %d %d\n", a.tokens, a.splits, a.kps, a.height, same ? 1 : 0);
    }
    const int Ns[4] = {15360, 5120, 13824, 5120}, ks[4] = {40, 40, 40, 108};
    printf("%f %f\n", ns([&](int i) { return w6_rows_search(kM, Ns[i & 3], ks[i & 3], clusters).tokens; }),
           ns([&](int i) { return w6_rows_plan(0, kM, Ns[i & 3], ks[i & 3], clusters).tokens; }));
}
"""
CLUSTERS = [1, 148, 74, 45, 33, 26, 22, 15, 15]


def _cost(M, N, k_iters, tokens, s, kps, h):
    tiles_m = -(-M // tokens)
    wait = 0.4 + 0.0025 * tokens
    box = (((h // 8 + 2) / 18) ** 4 + wait ** 4) ** 0.25 * (0.9 if tiles_m == 1 and tokens > 112 and h == 128 else 1.0)
    rounds = -(-(-(-N // h) * tiles_m) // CLUSTERS[s])
    return rounds * (kps * box + (8 + tokens / 28 if s == 1 else 10.5 + tokens / (40 if s <= 4 else 26)))


def _plans(k_iters):
    for h in range(64, 129, 8):
        for s in range(1, min(8, k_iters) + 1):
            k = -(-k_iters // s)
            if -(-k_iters // k) == s:
                yield s, k, h


@pytest.fixture(scope="module")
def planned(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I" + CSRC, str(d / "plan.cpp"), "-o", str(d / "plan")], check=True)
    rng = random.Random(5)
    sizes = [(M, N, K // 128) for M in (1, 16, 17, 64, 112, 113, 192, 255, 256) for N, K in ((15360, 5120), (5120, 13824), (640, 1024), (96, 5120), (1, 128))]
    sizes += [(rng.randint(1, 256), rng.randint(1, 20480), rng.randint(1, 120)) for _ in range(200)]
    sizes += [(rng.randint(257, 40000), rng.randint(1, 127), rng.randint(1, 40)) for _ in range(50)]      # beside a narrow weight: more rows
    out = subprocess.run([str(d / "plan")], input="\n".join(" ".join(map(str, s)) for s in sizes) + "\n", capture_output=True, text=True, check=True).stdout.split("\n")
    return [(s, tuple(map(int, line.split()))) for s, line in zip(sizes, out)], tuple(map(float, out[len(sizes)].split()))


def test_plans_are_valid_and_the_best_of_their_cost(planned):
    for (M, N, k_iters), (tokens, s, kps, h, same) in planned[0]:
        what = (M, N, k_iters, tokens, s, kps, h)
        assert same, what                                                  # searched, remembered, and on another thread
        assert tokens % 16 == 0 and 16 <= tokens <= 256 and h % 8 == 0 and 64 <= h <= 128, what
        assert 1 <= s <= 8 and kps * (s - 1) < k_iters <= kps * s, what
        mine = _cost(M, N, k_iters, tokens, s, kps, h)
        assert mine <= min(_cost(M, N, k_iters, tokens, *p) for p in _plans(k_iters)) * (1 + 1e-12), what
        for width in (256, 192, 128, 96, 64):                              # other token tiles promise less than 5 % (each step of the search)
            tm = -(-M // width)
            t = -(-(-(-M // tm)) // 16) * 16
            assert mine <= min(_cost(M, N, k_iters, t, *p) for p in _plans(k_iters)) / 0.95 ** 4, (what, t)


def test_a_plan_is_searched_once(planned):
    search, remembered = planned[1]
    assert remembered < search / 4, planned[1]
