"""Where single networks step, at measured points on both sides of each line of
group_plan.h: a form that was measured slower than the grid kernel (k_step,
k_det_step) there is not chosen, one that was clearly faster is.  CPU only
(host code, compiled here)."""
import subprocess
from pathlib import Path

from naer_b200.build import nvcc

ROOT = Path(__file__).resolve().parent.parent

CHECK = r"""
#include <cstdio>
#include "group_plan.h"
using namespace naer;
int main() {
    GroupNeed n;
    unsigned window, stdp, det, neurons;
    double row, events;
    while (std::scanf("%u %u %u %u %lf %lf", &window, &stdp, &det, &neurons, &row, &events) == 6) {
        n.window = window, n.stdp = stdp, n.det = det;
        n.chunks = (neurons + 31) / 32;
        n.synapses = (uint64_t)(neurons * row);
        n.act.neurons = n.act.drawn = neurons;
        n.act.events = events;
        n.act.spikes = row > 0 ? events / row : 0.0;
        const GroupForm f = single_form(n, 148);
        std::printf("%s%s\n", !f.group ? "grid kernel" : f.cluster ? "cluster" : "grid", f.local ? " local" : "");
    }
    return 0;
}
"""

# window, plastic, deterministic, neurons, out-degree, events a step -> form; us a step of
# (block-local or cluster, exchange on the grid, grid kernel) there
POINTS = [
    ((1, 0, 0, 2000, 100, 200), "cluster local"),         # 3.2, 5.9, 8.0
    ((1, 0, 0, 2000, 1000, 7600), "cluster local"),       # 5.0, 6.6, 9.1
    ((1, 0, 0, 2000, 4000, 141525), "grid"),              # 27.6, 8.2, 10.9
    ((1, 0, 0, 5000, 4000, 75225), "grid"),               # 13.5, 7.7, 10.9
    ((1, 0, 0, 6100, 2000, 102069), "grid"),              # 11.8, 8.2, 10.9
    ((1, 0, 0, 12000, 300, 3507), "cluster local"),       # 4.2, 6.8, 9.1
    ((1, 0, 0, 50000, 1000, 185916), "grid local"),       # 8.7, 8.7, 11.0
    ((1, 0, 0, 50000, 4000, 3481431), "grid kernel"),     # 41.8, 30.2, 26.7
    ((1, 0, 0, 100000, 2000, 391088), "grid"),            # -, 11.2, 12.0
    ((1, 0, 0, 200000, 1000, 196047), "grid"),            # 9.6, 9.3, 11.9
    ((1, 0, 0, 200000, 4000, 2967294), "grid kernel"),    # 42.5, 30.8, 26.2
    ((1, 0, 0, 20000, 0, 0), "grid local"),               # no synapses
    ((15, 0, 0, 6000, 1000, 5900), "cluster"),            # 1.7, 1.7, 8.6
    ((15, 0, 0, 6000, 4000, 458693), "grid"),             # 15.9, 4.8, 13.3
    ((2, 0, 0, 6000, 4000, 418444), "grid"),              # 21.3, 8.2, 10.5
    ((15, 0, 0, 400000, 1000, 3334387), "grid"),          # -, 22.9, 31.5
    ((1, 1, 0, 5000, 1000, 8949), "cluster"),             # 8.1, 9.0, 10.7
    ((1, 1, 0, 6100, 2000, 53527), "grid"),               # 17.5, 10.0, 13.4
    ((1, 1, 0, 12000, 1000, 66709), "grid"),              # 27.5, 11.1, 13.2 (8M synapses: the grid anyway)
    ((1, 1, 0, 240000, 1000, 488688), "grid"),            # -, 24.5, 28.1
    ((1, 0, 1, 6000, 300, 1797), "cluster"),              # 7.8, 10.2, 15.1
    ((1, 0, 1, 12000, 300, 30175), "grid"),               # 22.3, 12.9, 19.8
    ((1, 0, 1, 2000, 4000, 125261), "grid"),              # 255, 73, 154
    ((1, 0, 1, 100000, 1000, 97878), "grid"),             # -, 19.1, 22.5
    ((1, 0, 1, 100000, 1000, 834330), "grid kernel"),     # -, 70.7, 48.3
    ((1, 0, 1, 240000, 300, 70419), "grid"),              # -, 19.5, 20.1
    ((1, 0, 1, 240000, 100, 200506), "grid kernel"),      # -, 26.5, 20.6
    ((1, 0, 1, 240000, 4000, 938920), "grid kernel"),     # -, 67.9, 44.0
    ((1, 1, 1, 6000, 1000, 33478), "grid"),               # 28.8, 16.0, 28.7
    ((1, 1, 1, 100000, 1000, 198177), "grid"),            # -, 29.1, 31.2
    ((1, 1, 1, 240000, 1000, 1372255), "grid kernel"),    # -, 127, 110
]


def test_measured_points(tmp_path):
    src, exe = tmp_path / "check.cu", tmp_path / "check"
    src.write_text(CHECK)
    subprocess.run([nvcc(), "-std=c++17", "-I", str(ROOT / "naer_b200" / "csrc"), "-o", str(exe), str(src)], check=True)
    inp = "".join(" ".join(str(x) for x in p) + "\n" for p, _ in POINTS)
    out = subprocess.run([str(exe)], input=inp, capture_output=True, text=True, check=True).stdout.strip().split("\n")
    for (point, want), got in zip(POINTS, out, strict=True):
        assert got == want, point


BATCH = r"""
#include <cstdio>
#include "group_plan.h"
using namespace naer;
int main() {
    unsigned stdp, launch, sms;
    double count, neurons, row, rate, slots, c, per;
    while (std::scanf("%u %lf %lf %lf %lf %lf %lf %lf %u %u", &stdp, &count, &neurons, &row, &rate, &slots, &c, &per, &launch,
                      &sms) == 10) {
        GroupNeed n;
        n.stdp = stdp;
        n.synapses = (uint64_t)(neurons * row);
        n.act.neurons = n.act.drawn = neurons;
        n.act.spikes = 1e-4 * rate * neurons;
        n.act.events = n.act.spikes * row;
        const double rounds = std::ceil(std::ceil(neurons / (32 * per)) / (12 * c)), turns = std::ceil(count * c / sms);
        const double clusters = turns * cluster_us(n, (unsigned)c, (unsigned)per, rounds);
        std::printf("%d %.1f\n", (int)clusters_pay(clusters, grid_us(count * neurons, count * n.act.events,
                    4e-6 * slots * count * neurons, stdp, launch)), clusters);
    }
    return 0;
}
"""

# plastic, networks, neurons, out-degree, rate, ring slots, blocks, neurons a lane, steps a launch, usable SMs
# -> clusters; measured us a step, clusters and grid kernel
BATCHES = [
    ((0, 64, 2000, 200, 19.2, 17, 1, 4, 64, 148), 1),     # 5.6, 11.4
    ((0, 8, 20000, 500, 19.2, 17, 8, 4, 64, 120), 1),     # 9.9, 12.0
    ((0, 16, 50000, 500, 19.2, 17, 4, 4, 64, 148), 0),    # 30.0, 19.7
    ((0, 32, 20000, 300, 19.2, 17, 2, 4, 64, 148), 0),    # 24.1, 17.2
    ((0, 32, 10000, 2000, 37.0, 17, 8, 4, 64, 120), 0),   # 45.5, 26.0
    ((1, 8, 5000, 500, 11.1, 21, 8, 1, 64, 120), 1),      # 8.0, 11.6
    ((1, 8, 50000, 500, 11.1, 21, 8, 4, 64, 120), 0),     # 35.1, 21.0
    ((0, 32, 20000, 300, 19.2, 17, 2, 4, 4, 148), 1),     # four steps a launch (served): the grid's launches cost more
]


def test_measured_batches(tmp_path):
    src, exe = tmp_path / "check.cu", tmp_path / "check"
    src.write_text(BATCH)
    subprocess.run([nvcc(), "-std=c++17", "-I", str(ROOT / "naer_b200" / "csrc"), "-o", str(exe), str(src)], check=True)
    inp = "".join(" ".join(str(x) for x in p) + "\n" for p, _ in BATCHES)
    out = subprocess.run([str(exe)], input=inp, capture_output=True, text=True, check=True).stdout.strip().split("\n")
    for (point, want), got in zip(BATCHES, out, strict=True):
        assert int(got.split()[0]) == want, (point, got)
