"""The tile list of a projection of many tokens (linear_plan.hpp), walked on the CPU: every 128 columns of every row tile
once, and no more rounds than the choice of the column width reckoned with."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

WALK = r"""
#include <cstdio>
#include <map>
#include <random>
#include <tuple>
#include <vector>
#include "linear_plan.hpp"
struct Job { int out_features; };
struct Args { Job job[hc::kLinJobs]; int n_jobs, tiles_m, n_wide; };
static int check(const std::vector<int>& outs, int tiles_m, int pairs) {
    const hc::LinPlan plan = hc::plan_pairs(outs.data(), int(outs.size()), tiles_m, pairs);
    if (plan.width != 256) return 0;
    Args args{};
    args.n_jobs = int(outs.size());
    args.tiles_m = tiles_m;
    args.n_wide = int(plan.n_wide);
    long long blocks = 0;
    for (size_t j = 0; j < outs.size(); ++j) {
        args.job[j].out_features = outs[j];
        blocks += (long long)((outs[j] + 127) / 128) * tiles_m;
    }
    std::map<std::tuple<int, int, int>, int> seen;
    double clocks = 0;
    int bad = 0;
    for (long long tile = 0; tile < plan.n_tiles; ++tile) {
        const hc::LinWide t = hc::decode_wide<256>(args, int(tile));
        if (tile % pairs == 0) clocks += t.width == 256 ? 546.0 : 410.0;      // the widest of a round comes first
        bad |= t.job < 0 || t.job >= args.n_jobs || t.tm < 0 || t.tm >= tiles_m || t.col % 128 || t.col < 0 || t.col >= outs[t.job];
        bad |= (t.width == 256) != (tile < plan.n_wide);
        if (bad) break;
        for (int col = t.col; col < t.col + t.width && col < outs[t.job]; col += 128) bad |= seen[{t.job, t.tm, col}]++ != 0;
    }
    bad |= (long long)seen.size() != blocks || clocks > plan.steps;
    if (bad) {
        std::printf("tiles_m %d pairs %d, %.0f clocks of %.0f, columns", tiles_m, pairs, clocks, plan.steps);
        for (int n : outs) std::printf(" %d", n);
        std::printf("\n");
    }
    return bad;
}
int main() {
    int bad = 0;
    for (int pairs : {74, 72, 5, 1}) {
        for (int tiles_m : {1, 2, 3, 16, 32}) {
            for (int n = 1; n < 2600; n += n < 520 ? 1 : 37) bad += check({n}, tiles_m, pairs);
            bad += check({904}, tiles_m, pairs) + check({2200}, tiles_m, pairs) + check({2880}, tiles_m, pairs);
        }
    }
    std::mt19937 rng(1);
    for (int i = 0; i < 3000; ++i) {
        std::vector<int> outs(1 + rng() % hc::kLinJobs);
        for (int& n : outs) n = 1 + rng() % (rng() % 2 ? 300 : 5000);
        bad += check(outs, 1 + rng() % 20, 74);
    }
    return bad != 0;
}
"""


def test_tiles_of_two_widths_cover_every_column_in_the_rounds_reckoned_with(tmp_path):
    (tmp_path / "walk.cpp").write_text(WALK)
    program = str(tmp_path / "walk")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-I", os.path.join(ROOT, "hydra_b200", "csrc"), str(tmp_path / "walk.cpp"), "-o", program])
    done = subprocess.run([program], capture_output=True, text=True)
    assert done.returncode == 0, done.stdout[:2000]
