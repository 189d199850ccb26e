"""The step kernel and the steps per launch that a server's parameters select:
an explicit value is kept, on the grid and in clusters.  CPU only (the rule is
host code, compiled here)."""
import subprocess
from pathlib import Path

from naer_b200 import _capi as capi
from naer_b200.build import nvcc

ROOT = Path(__file__).resolve().parent.parent

CHECK = r"""
#include <cstdio>
#include "forms.h"
using namespace naer;
int main() {
    unsigned launch, kernel, blocks;
    while (std::scanf("%u %u %u", &launch, &kernel, &blocks) == 3) {
        ServerParams p;
        p.launch_steps = launch;
        p.step_kernel = kernel;
        p.blocks_per_sm = blocks;
        const Tuning t = served_tuning(p);
        std::printf("%u %u %u %u %u\n", t.step_kernel, t.group_launch_steps(false), t.group_launch_steps(true),
                    (unsigned)t.group_allowed(false), (unsigned)t.group_allowed(true));
    }
    const Tuning own;  // a network or a batch
    std::printf("%u %u %u %u\n", own.group_launch_steps(false), own.group_launch_steps(true),
                (unsigned)own.group_allowed(false), (unsigned)own.group_allowed(true));
    return 0;
}
"""


def test_explicit_choices_are_kept(tmp_path):
    src, exe = tmp_path / "check.cu", tmp_path / "check"
    src.write_text(CHECK)
    subprocess.run([nvcc(), "-std=c++17", "-I", str(ROOT / "naer_b200" / "csrc"), "-o", str(exe), str(src)], check=True)
    S, T = capi.KERNEL_SPLIT, capi.KERNEL_TWO_BARRIER
    # launch_steps, step_kernel, blocks_per_sm -> kernel, steps on the grid and in clusters, the window
    # kernel open (atomic or exact-sum, deterministic)
    want = {(0, T, 0): (T, 4, 32, 1, 1),
            (1, T, 0): (T, 1, 1, 1, 1),
            (16, T, 0): (T, 16, 16, 1, 1),
            (64, T, 0): (T, 64, 64, 1, 1),
            (0, S, 0): (S, 4, 32, 0, 1),
            (8, S, 0): (S, 8, 8, 0, 1),
            (0, T, 2): (T, 4, 32, 0, 0)}
    inp = "".join("%u %u %u\n" % k for k in want)
    out = subprocess.run([str(exe)], input=inp, capture_output=True, text=True, check=True).stdout.split("\n")
    for (k, v), line in zip(want.items(), out):
        assert tuple(int(x) for x in line.split()) == v, k
    assert out[len(want)].split() == ["64", "64", "1", "1"]
