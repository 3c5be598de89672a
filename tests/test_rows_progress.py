"""The rule that admits an instance to the implicit row-block kernels, where the
blocks outnumber the resident CTAs: a host program walks the kernel's schedule
(blocks claimed in order, a warp's tiles one after another, a tile done once the
maps of the blocks that its fold reads are published) until nothing moves.  What
the rule admits has to finish, on chips with fewer SMs as well; and the walk itself
has to get stuck where the rule is far exceeded, or it would show nothing."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CUDA = Path(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc").resolve().parent.parent / "include"

WALK = r"""
#include <algorithm>
#include <cstdio>
#include <vector>
#include "keq_rows_host.h"

// True if `nblk` blocks of nvt tiles (nt_neg of them against the block order) finish
// on `grid` CTAs of `warps` warps with folds over up to kmax blocks.
static bool finishes(int nblk, int nvt, int nt_neg, int kmax, int warps, int grid) {
    // per block and warp: tiles done; a claimed block has published the maps of the
    // tiles done and of the one behind them
    std::vector<std::vector<int>> done(nblk, std::vector<int>(warps, 0));
    std::vector<int> tiles(warps);
    for (int w = 0; w < warps; ++w) tiles[w] = w < nvt ? (nvt - w + warps - 1) / warps : 0;
    int claimed = std::min(grid, nblk);
    std::vector<int> open(claimed);
    for (int b = 0; b < claimed; ++b) open[b] = b;
    auto there = [&](int b, int w, int k) { return b < claimed && done[b][w] >= k; };
    while (!open.empty()) {
        bool moved = false;
        std::vector<int> still;
        for (int b : open) {
            bool all = true;
            for (int w = 0; w < warps; ++w)
                while (done[b][w] < tiles[w]) {
                    const int k = done[b][w], vt = w + k * warps;
                    const bool up = vt >= nt_neg;  // reads blocks in front of it
                    const int avail = up ? b : nblk - 1 - b, last = std::min(avail, kmax);
                    bool ok = true;
                    for (int j = 1; j <= last && ok; ++j) ok = there(up ? b - j : b + j, w, k);
                    if (!ok) { all = false; break; }
                    ++done[b][w];
                    moved = true;
                }
            if (!all) { still.push_back(b); continue; }
            if (claimed < nblk) still.push_back(claimed++);
        }
        open.swap(still);
        if (!moved) return false;
    }
    return true;
}

int main() {
    int admitted = 0;
    for (int sms : {148, 132, 20}) {
        for (int nvt : {1, 2, 5, 8, 9, 16, 17, 32, 33, 64}) {
            const int kmax = std::min(keq::kRowsKmax, keq::rows_fold_limit(nvt, sms));
            if (!keq::rows_eligible(kmax, nvt, sms)) { printf("not admitted\n"); return 1; }
            // folds go up to the limit, beyond the admission's kmax
            const int fold = keq::rows_fold_limit(nvt, sms);
            for (int warps : {4, 8}) {
                const int grid = sms * (warps == 8 ? 2 : 4);
                if (!keq::rows_progress(fold, nvt, warps, grid)) { printf("rule: %d %d %d\n", sms, nvt, warps); return 1; }
                for (int neg : {0, nvt / 2, nvt})
                    for (int nblk : {grid + 1, 2 * grid + 3})
                        if (!finishes(nblk, nvt, neg, fold, warps, grid)) {
                            printf("stuck: %d SMs, %d tiles (%d), fold %d, %d warps, %d blocks\n", sms, nvt, neg, fold, warps, nblk);
                            return 1;
                        }
                ++admitted;
            }
        }
    }
    // far beyond the rule the schedule does get stuck, and the rule says so
    if (keq::rows_progress(300, 8, 8, 296) || finishes(1000, 8, 8, 300, 8, 296)) { printf("no stall\n"); return 1; }
    if (keq::rows_progress(100, 32, 8, 296) || finishes(1000, 32, 32, 100, 8, 296)) { printf("no stall\n"); return 1; }
    printf("%d ok\n", admitted);
    return 0;
}
"""


def test_admitted_plans_make_progress(tmp_path):
    if not (CUDA / "cuda_runtime.h").exists() or not shutil.which("g++"):
        pytest.skip("no CUDA headers or host compiler")
    (tmp_path / "walk.cpp").write_text(WALK)
    exe = tmp_path / "walk"
    subprocess.run(["g++", "-O2", "-std=c++17", f"-I{ROOT / 'kineticeq_b200' / 'csrc'}", f"-I{CUDA}",
                    str(tmp_path / "walk.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
    assert r.stdout.strip() == "60 ok"
