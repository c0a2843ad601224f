"""CPU tests of what orders the two CTAs of a pair (gemm_umma.cu).

Sources: an arrival without release on the other CTA's barrier publishes no
shared memory, so it may only hand over TMEM columns (tcgen05's fences order
those); tiles that TMA loads complete on the barrier of the CTA that issues the
MMAs; planes that warps write into shared memory are released to the cluster.

pair_drain, the end of a pair whose wait gave up, compiled for the host against
counting barriers: whatever stages the two producers had issued, every stage's
phase completes and none is waited for before it can."""
from __future__ import annotations

import os
import re
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rblas_b200", "csrc")


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read()


def test_arrivals_without_release_hand_over_tmem_only():
    src = source("gemm_umma.cu")
    calls = re.findall(r"([^\n]*)mbar_arrive_rank_relaxed\(&bar->(\w+)", src)
    assert calls
    for before, bar in calls:
        # accumulators drained, or A's planes stored with tcgen05.st
        assert bar == "acc_empty" or (bar == "a_full" and "if constexpr (A_TMEM)" in before), (before, bar)


def test_pair_loads_complete_on_the_issuing_ctas_barrier():
    src = source("gemm_umma.cu")
    for kernel, loads in (("umma_pair_kernel(const", 4), ("umma_split_fused_kernel(const", 1), ("ozaki_pair_body(const Src", 2)):
        body = src[src.index(kernel):]
        body = body[:body.index("tmem_dealloc_pair")]
        assert len(re.findall(r"tma_load_3d_pair\(", body)) == loads, kernel
        assert not re.search(r"tma_load_3d\(", body), kernel  # (A's f32 tiles of the fused kernel: 2-D, read by this CTA)
        assert "mbar_arrive_expect_tx_cluster(" in body and "pair_fail(" in body and "pair_drain(" in body, kernel


HOST = r"""
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#define __device__
#define __noinline__
static uint64_t* ring;
static int count[16];   // arrivals on each slot's barrier, two a phase
static int n_stages;
static void mbar_arrive(uint64_t* b) { ++count[b - ring]; }
static uint32_t waited;
static bool mbar_wait_drain(uint64_t* b, uint32_t parity) {
    const int phase = count[b - ring] / 2;  // phases complete
    if (count[b - ring] %% 2 || phase == 0 || ((phase - 1) & 1) != (int)parity) { std::printf("wait fails\n"); std::exit(1); }
    ++waited;
    return true;
}
%s
int main() {
    uint64_t bars[16];
    ring = bars;
    for (uint32_t stages = 2; stages <= 11; ++stages)
        for (uint32_t a = 0; a < 40; ++a)
            for (uint32_t b = a > stages ? a - stages : 0; b <= a + stages && b < 40; ++b) {  // (a slot is refilled once both were read)
                for (uint32_t s = 0; s < 16; ++s) count[s] = 0;
                const uint32_t issued[2] = {a, b};
                for (int c = 0; c < 2; ++c)
                    for (uint32_t j = 0; j < issued[c]; ++j) ++count[j %% stages];
                waited = 0;
                pair_drain(bars, stages, issued);
                const uint32_t end = a > b ? a : b;
                if (waited != (end < stages ? end : stages)) return 2;
                for (uint32_t s = 0; s < stages; ++s)  // every phase that began has ended
                    if (count[s] %% 2) return 3;
            }
    return 0;
}
"""


def test_pair_drain_ends_every_phase(tmp_path):
    src = source("rb_device.cuh")
    start = src.index("static __device__ __noinline__ void pair_drain(")
    func = src[start:src.index("\n}", start) + 2]
    cpp = tmp_path / "drain.cpp"
    cpp.write_text(HOST % func)
    exe = tmp_path / "drain"
    subprocess.run(["g++", "-O1", "-std=c++17", "-o", str(exe), str(cpp)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
