"""The radix selection of the sampler (``csrc/radix.cuh``) built for the host, a thread of the CTA
a thread of the process, under ThreadSanitizer: two descents one after the other over the same
shared memory find the same keys as a sort, and no thread reads what another writes without a
barrier between them.  Needs g++ only."""
import os
import shutil
import subprocess

import pytest

from util import ROOT

HARNESS = r"""
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <pthread.h>
#include <thread>
#include <vector>
using std::min;
constexpr int SM_THREADS = 256;
#define __device__
#define __forceinline__ inline
struct Index { unsigned x; };
static thread_local Index threadIdx;
static pthread_barrier_t of_cta, of_warp[SM_THREADS / 32];
static unsigned long long lanes[SM_THREADS];
static void __syncthreads() { pthread_barrier_wait(&of_cta); }
static void __syncwarp() { pthread_barrier_wait(&of_warp[threadIdx.x / 32]); }
template <typename T> static T exchange(T v, int from, bool valid) {
    lanes[threadIdx.x] = (unsigned long long)v;
    __syncwarp();
    const T got = valid ? (T)lanes[threadIdx.x / 32 * 32 + from] : v;
    __syncwarp();
    return got;
}
template <typename T> static T __shfl_sync(unsigned, T v, int lane) { return exchange(v, lane, true); }
template <typename T> static T __shfl_down_sync(unsigned, T v, int by) {
    const int from = (int)(threadIdx.x % 32) + by;
    return exchange(v, from, from < 32);
}
static unsigned __ballot_sync(unsigned, bool p) {
    unsigned all = 0;
    for (int l = 0; l < 32; ++l) all |= exchange((unsigned)p, l, true) << l;
    return all;
}
static int __clz(unsigned v) { return v ? __builtin_clz(v) : 32; }
template <typename T> static void atomicAdd(T* p, T v) { __atomic_fetch_add(p, v, __ATOMIC_RELAXED); }
static void cluster_meet() {}
static unsigned long long peer_u64(const unsigned long long* p, int) { return *p; }
#include "radix.cuh"

int main() {
    constexpr int PER = 3, N = PER * SM_THREADS;
    pthread_barrier_init(&of_cta, nullptr, SM_THREADS);
    for (auto& w : of_warp) pthread_barrier_init(&w, nullptr, 32);
    std::vector<unsigned> keys(N);
    srand(5);
    for (auto& k : keys) k = (unsigned)rand() * 2u + 1u;
    std::vector<unsigned> order(keys);
    std::sort(order.rbegin(), order.rend());
    static RadixShared sh;
    int wrong = 0;
    std::vector<std::thread> cta;
    for (int t = 0; t < SM_THREADS; ++t)
        cta.emplace_back([&, t] {
            threadIdx.x = t;
            int turn = 0;
            auto each = [&](int e0, int e1, auto&& add) {
                for (int e = e0; e < e1; ++e) add(keys[t + e * SM_THREADS], 1ull);
            };
            // as the sampler calls it: a bound from above, then the key, then by weight
            const unsigned a = radix_descend<true>(sh, 1, turn, 10, PER, each);
            const unsigned b = radix_descend<true>(sh, 1, turn, 64, PER, each);
            const unsigned c = radix_descend<false>(sh, 1, turn, N, PER, each);
            if (a != order[9] || b != order[63] || c != order[N - 1])
                __atomic_fetch_add(&wrong, 1, __ATOMIC_RELAXED);
        });
    for (auto& t : cta) t.join();
    printf("wrong %d\n", wrong);
    return wrong ? 1 : 0;
}
"""


def test_descents_share_no_unsynchronised_memory(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    flags = ["-std=c++17", "-O1", "-g", "-pthread", "-fsanitize=thread"]
    (tmp_path / "empty.cc").write_text("int main() { return 0; }\n")
    probe = subprocess.run([gxx, *flags, str(tmp_path / "empty.cc"), "-o", str(tmp_path / "empty")],
                           capture_output=True, text=True)
    if probe.returncode or subprocess.run([str(tmp_path / "empty")], capture_output=True).returncode:
        pytest.skip("ThreadSanitizer does not run here")
    (tmp_path / "radix.cc").write_text(HARNESS)
    subprocess.run([gxx, *flags, "-Wno-unknown-pragmas", "-I", os.path.join(ROOT, "agave_b200", "csrc"),
                    str(tmp_path / "radix.cc"), "-o", str(tmp_path / "radix")], check=True)
    run = subprocess.run([str(tmp_path / "radix")], capture_output=True, text=True, timeout=300,
                         env=dict(os.environ, TSAN_OPTIONS="halt_on_error=0 exitcode=66"))
    assert "data race" not in run.stderr, run.stderr[:4000]
    assert run.returncode == 0, (run.returncode, run.stdout, run.stderr[:2000])
