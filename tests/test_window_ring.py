"""Windows of the window kernel stay inside the delay ring.  A network's ring
has one slot more than its largest delay, so networks without synapses, or
whose connections touch an empty population, have rings of a few slots.

The rule is checked on the host for every smallest delay and ring; the
networks themselves against the oracle (-m gpu), bit for bit."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

from naer_b200 import _capi as capi
from naer_b200 import spec as S
from naer_b200.build import nvcc
from naer_b200.forms import Batch, Server

ROOT = Path(__file__).resolve().parent.parent

CHECK = r"""
#include <cstdio>
#include "engine_types.cuh"
using namespace naer;
int main() {
    for (uint32_t slots = 2; slots <= 255; ++slots)
        for (uint32_t dmin = 1; dmin <= 254; ++dmin) {
            const uint32_t w = window_steps(dmin, slots);
            if (w < 1 || w > kGroupMaxWindow || w > dmin) return 1;
            for (uint32_t at = 0; at < slots; ++at)   // ring_slot: one subtraction
                for (uint32_t k = 0; k < w; ++k)
                    if ((at + k >= slots ? at + k - slots : at + k) >= slots) return 2;
            // as long as a connected network allows: its ring has more slots than its smallest delay
            if (dmin < slots && w != (dmin < kGroupMaxWindow ? dmin : kGroupMaxWindow)) return 3;
        }
    return 0;
}
"""


def test_window_rule(tmp_path):
    src, exe = tmp_path / "check.cu", tmp_path / "check"
    src.write_text(CHECK)
    subprocess.run([nvcc(), "-std=c++17", "-I", str(ROOT / "naer_b200" / "csrc"), "-o", str(exe), str(src)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0


def driven(n, empty_delay=None, **kw):
    """Driven LIF neurons that receive nothing; with empty_delay connected to
    and from an empty population with delays up to it."""
    s = S.NetSpec(name="driven", poisson_seed=5, **kw)
    E = s.add_pop(S.NOP, n, drive_rate_hz=200.0, drive_weight=21.0, drive_seed=n)
    if empty_delay:
        Z = s.add_pop(S.NOP, 0)
        for a, b in [(E, Z), (Z, E)]:
            s.connect(a, b, capi.CONN_REF_BERNOULLI, 1.0, probability=0.5, dmin=1, dmax=empty_delay, seed=n)
    return s


def connected(n, **kw):
    s = S.NetSpec(name="connected", poisson_seed=6, **kw)
    E = s.add_pop(S.NOP, n, drive_rate_hz=200.0, drive_weight=21.0, drive_seed=n + 1)
    s.connect(E, E, capi.CONN_FIXED_OUTDEGREE, 1.0, degree=20, dmin=3, dmax=9, seed=n)
    return s


RUNS = [1, 64, 150]


def expected(oracle_mod, s):
    o = oracle_mod.OracleNet(s, deterministic=None if s.exact else True)
    o.run(sum(RUNS))
    out = o.spikes() + o.state()
    o.close()
    return out


def same(got, want):
    assert len(want[1]) > 100
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    assert np.array_equal(got[2].view(np.uint32), want[2].view(np.uint32)) and np.array_equal(got[3], want[3])


@pytest.mark.gpu
@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("empty_delay", [None, 4, 13])
@pytest.mark.parametrize("n", [700, 5000, 20000])
def test_no_synapses(oracle_mod, lib, n, empty_delay, exact):
    s = driven(n, empty_delay, exact=exact)
    with S.build(s) as net:
        for c in RUNS:
            net.run(c)
        net.finish()
        got = net.read_spikes() + net.read_state()
    same(got, expected(oracle_mod, s))


@pytest.mark.gpu
@pytest.mark.parametrize("exact", [False, True])
def test_no_synapses_beside_others(oracle_mod, lib, exact):
    """As batch members and as served jobs, beside connected networks."""
    ms = [f(n, exact=exact) for n in (700, 5000, 20000) for f in (driven, connected)] + [driven(900, 4, exact=exact)]
    want = [expected(oracle_mod, m) for m in ms]
    with Batch(ms, exact=exact, raster_capacity=1 << 22).compile() as b:
        for c in RUNS:
            b.run(c)
        b.finish()
        spikes = b.read_spikes()
        for i, m in enumerate(ms):
            same(b.member_spikes(i, spikes) + b.read_state(i, m.neurons), want[i])
    with Server(budget_bytes=2 * 10**9, exact=exact) as srv:
        jobs = [srv.submit(m, sum(RUNS)) for m in ms]
        for i, j in enumerate(jobs):
            srv.wait(j)
            st, ids = srv.spikes(j)
            assert np.array_equal(st, want[i][0]) and np.array_equal(ids, want[i][1]), i
