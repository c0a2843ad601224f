"""CPU test of how the kinds of tile of a grouped Ozaki launch share the SMs
(ozaki_share_sms, gemm_umma.cu), compiled for the host: a kind's time is that of
dealing its tiles one by one, a split fits the SMs and starts every kind at once,
and it ends before the kinds one after the other would (mixed sets did take up to
a third longer that way than before CTA pairs were a kind of their own)."""
from __future__ import annotations

import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rblas_b200", "csrc")

HOST = r"""
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>
#include <utility>
#include <vector>
%s
static double dealt(const OzGroupKind& g, int workers) {  // the fullest worker
    std::vector<double> t(workers, 0.0);
    int i = 0;
    for (const auto& j : g.jobs)
        for (int q = 0; q < j.first; ++q, ++i) t[i %% workers] += j.second * g.per_kt + g.per_tile;
    return *std::max_element(t.begin(), t.end());
}
int main() {
    std::mt19937 rng(1);
    int shared = 0;
    for (int trial = 0; trial < 3000; ++trial) {
        OzGroupKind kinds[3];
        const int sms = trial %% 7 == 0 ? 2 + rng() %% 20 : 148;
        int used = 0;
        for (int q = 0; q < 3; ++q) {
            const int n = rng() %% 3 == 0 ? 0 : 1 + rng() %% 20;
            for (int i = 0; i < n; ++i) kinds[q].jobs.emplace_back(1 + rng() %% (rng() %% 4 ? 8 : 200), 1 + rng() %% 32);
            std::sort(kinds[q].jobs.begin(), kinds[q].jobs.end(), [](auto& a, auto& b) { return a.second > b.second; });
            used += n > 0;
        }
        int workers[3];
        const bool share = ozaki_share_sms(kinds, 2 + rng() %% 11, sms, workers);
        if (used < 2 && share) return 1;
        if (!share) continue;
        ++shared;
        double end = 0, one_by_one = 0;
        const int cap[3] = {sms / 2, sms, sms}, sm[3] = {2, 1, 1};
        int need = 0;
        for (int q = 0; q < 3; ++q) {
            if (kinds[q].jobs.empty()) {
                if (workers[q] != 0) return 2;
                continue;
            }
            if (workers[q] < 1 || workers[q] > cap[q]) return 3;
            need += sm[q] * workers[q];
            const double t = dealt(kinds[q], workers[q]);
            if (std::fabs(t - kinds[q].time(workers[q])) > 1e-9 * t) return 4;
            end = std::max(end, t);
            one_by_one += dealt(kinds[q], cap[q]);
        }
        if (need > sms) return 5;
        if (end > 0.951 * one_by_one) return 6;
    }
    std::printf("%%d\n", shared);
    return shared > 1500 ? 0 : 7;
}
"""


def test_share(tmp_path):
    with open(os.path.join(CSRC, "gemm_umma.cu")) as f:
        src = f.read()
    start = src.index("struct OzGroupKind {")
    end = src.index("\n}\n", src.index("bool ozaki_share_sms(")) + 2
    cpp = tmp_path / "share.cpp"
    cpp.write_text(HOST % src[start:end])
    exe = tmp_path / "share"
    subprocess.run(["g++", "-O2", "-std=c++17", "-o", str(exe), str(cpp)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stdout)
