"""The window kernel (k_group) against the oracle, at the sizes where it can
go wrong: chunks of 32 and 128 neurons and their remainders, one and two
chunks per warp, cluster and grid, windows of one step, of a few, of the
longest a kernel takes and of smallest delays past that, launches that end
within a window, more spikes in a window than a block keeps in shared memory,
a raster that fills up within a launch.

Weights are integers (or the aggregation is exact-sum), so every ring sum is
exact whatever the order of the reductions and everything is bit for bit.
"""
import numpy as np
import pytest

from naer_b200 import _capi as capi
from naer_b200 import spec as S
from naer_b200.forms import Batch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def O(oracle_mod, lib):
    return oracle_mod


def mixed_net(n, k, dmin, dmax, sources=0, seed=3, rate=200.0, t_ref_ms=2.0, **kw):
    """80/20 LIF neurons, fixed out-degree with integer weights, per-neuron
    drive on the excitatory ones, and POISSON sources (multiplicities)."""
    s = S.NetSpec(name="mixed", poisson_seed=seed, **kw)
    ne = max(1, n * 4 // 5)
    E = s.add_pop(S.NOP, ne, drive_rate_hz=rate, drive_weight=21.0, drive_seed=7 + seed, t_ref_ms=t_ref_ms)
    I = s.add_pop(S.NOP, max(1, n - ne), t_ref_ms=t_ref_ms)
    R = capi.CONN_FIXED_OUTDEGREE
    for src, w, sd in [(E, 2.0, 1), (I, -3.0, 2)]:
        s.connect(src, E, R, w, degree=k, dmin=dmin, dmax=dmax, seed=seed * 100 + sd)
        s.connect(src, I, R, w, degree=k, dmin=dmin, dmax=dmax, seed=seed * 100 + sd + 10)
    if sources:
        P = s.add_pop(S.POISSON, sources, rate_hz=3000.0)
        s.connect(P, E, R, 1.0, degree=k, dmin=dmin, dmax=dmax, seed=seed * 100 + 5)
        s.connect(P, I, R, 1.0, degree=k, dmin=dmin, dmax=dmax, seed=seed * 100 + 6)
    return s


def assert_matches(O, spec, runs, launches_per_run=None):
    """The network after the given runs of grid steps, bit for bit."""
    steps = sum(runs)
    with S.build(spec) as net:
        for c in runs:
            net.run(c)
        net.finish()
        st, ids = net.read_spikes()
        v, r = net.read_state()
        stats = net.stats()
        w = net.read_csr()[2] if spec.stdp_enabled else None
    o = O.OracleNet(spec, deterministic=None if spec.exact else True)
    o.run(steps)
    ost, oids = o.spikes()
    ov, orr = o.state()
    oev, ow = o.events, o.weights() if spec.stdp_enabled else None
    o.close()
    # one launch for up to 64 steps: the window kernel, not k_drive + k_step
    assert stats["kernel_launches"] == sum((c + 63) // 64 for c in runs)
    assert len(oids) > 20
    assert np.array_equal(st, ost) and np.array_equal(ids, oids)
    assert np.array_equal(v.view(np.uint32), ov.view(np.uint32)) and np.array_equal(r, orr)
    assert stats["events"] == oev and stats["step"] == steps
    if w is not None:
        assert np.array_equal(w.view(np.uint32), ow.view(np.uint32))


@pytest.mark.parametrize("n", [5, 40, 161, 6100, 6200, 12200, 12400])
@pytest.mark.parametrize("dmin,dmax", [(1, 12), (4, 9)])
def test_sizes(O, n, dmin, dmax):
    """Less than a chunk, remainders, 16 blocks x 12 warps full (6,144
    neurons), two chunks a warp, the first sizes of the grid form."""
    assert_matches(O, mixed_net(n, 20 if n > 100 else 5, dmin, dmax, sources=70), [1, 63, 150])


@pytest.mark.parametrize("dmin,dmax", [(2, 2), (3, 40), (15, 15), (16, 16), (17, 90), (200, 254)])
@pytest.mark.parametrize("n", [700, 15000])
def test_windows(O, n, dmin, dmax):
    """Windows of 2, 3, 15 and 16 steps and smallest delays past the longest
    window; runs that end within one."""
    assert_matches(O, mixed_net(n, 12, dmin, dmax, sources=33), [2, 64, 31, 65, 300])


@pytest.mark.parametrize("n,dmin,dmax", [(120_000, 1, 16), (130_001, 5, 5)])
def test_four_neurons_a_lane(O, n, dmin, dmax):
    assert_matches(O, mixed_net(n, 10, dmin, dmax, sources=130, rate=60.0), [65, 35])


def test_exchange_with_one_step_windows(O):
    """Past the size of block-local delivery: spikes exchanged between blocks."""
    assert_matches(O, mixed_net(6000, 700, 1, 8, sources=50, rate=100.0), [70])


@pytest.mark.parametrize("n", [900, 5000, 14000])
def test_plasticity(O, n):
    s = S.plastic_indegree(n=n, k=60, seed=5, drive_rate_hz=60.0).with_(exact=True)
    assert_matches(O, s, [1, 200, 64])


def test_two_plastic_populations_and_odd_sizes(O):
    s = S.NetSpec(name="two", exact=True, stdp_enabled=True, poisson_seed=3, stdp_history=3)
    A = s.add_pop(S.STDP, 333, drive_rate_hz=80.0, drive_weight=20.5, drive_seed=1)
    B = s.add_pop(S.STDP, 31, drive_rate_hz=80.0, drive_weight=20.5, drive_seed=2)
    C = s.add_pop(S.NOP, 65)
    R = capi.CONN_FIXED_INDEGREE
    for i, (a, b) in enumerate([(A, A), (A, B), (B, A), (A, C), (C, A), (B, C)]):
        s.connect(a, b, R, -0.3 if a == C else 0.2, degree=20, dmin=1, dmax=7, seed=40 + i)
    assert_matches(O, s, [500])


@pytest.mark.parametrize("n,k,dmin,dmax,rate,t_ref", [
    (5, 3, 1, 3, 500.0, 2.0),
    (161, 150, 1, 1, 3000.0, 0.0),       # lists past the fold's registers
    (6100, 20, 1, 12, 200.0, 2.0),       # one chunk a warp, piece by piece
    (6000, 700, 2, 30, 200.0, 2.0),      # more list starts than a warp keeps
    (12200, 40, 4, 9, 200.0, 2.0),       # two chunks a warp; delays past one step
    (12400, 150, 1, 254, 100.0, 2.0),    # the grid
    (30000, 1300, 3, 40, 200.0, 2.0),    # the grid, more list starts than a warp keeps
    (130001, 30, 1, 16, 60.0, 2.0),      # four neurons a lane
])
def test_deterministic(O, n, k, dmin, dmax, rate, t_ref):
    """Random weights: sums in the canonical order, bit for bit."""
    s = mixed_net(n, k, dmin, dmax, sources=50, rate=rate, t_ref_ms=t_ref)
    for c in s.conns[:2]:
        c.weight, c.wmin, c.wmax = 0.0, 0.05, 0.9
    assert_matches(O, s.with_(deterministic=True), [1, 64, 40])


@pytest.mark.parametrize("n,k", [(900, 60), (14000, 60), (5000, 600)])
def test_deterministic_plasticity(O, n, k):
    s = S.plastic_indegree(n=n, k=k, seed=5, drive_rate_hz=60.0).with_(deterministic=True)
    assert_matches(O, s, [1, 200, 64])


@pytest.mark.parametrize("n", [5000, 14000])
def test_more_spikes_than_the_shared_list(O, n):
    """Every driven neuron fires nearly every step (no refractory period):
    thousands of spikes per block and window."""
    assert_matches(O, mixed_net(n, 3, 12, 14, rate=9000.0, t_ref_ms=0.0), [40])


def test_no_recording_and_idle_network(O):
    s = mixed_net(3000, 10, 2, 5).with_(record=False)
    with S.build(s) as net:
        net.run(100)
        net.finish()
        v, r = net.read_state()
        assert net.stats()["spikes"] == 0 and net.stats()["raster_dropped"] == 0
    with S.build(s.with_(record=True)) as net:
        net.run(100)
        net.finish()
        v1, r1 = net.read_state()
    assert np.array_equal(v.view(np.uint32), v1.view(np.uint32)) and np.array_equal(r, r1)


@pytest.mark.parametrize("n", [3000, 20000])
def test_full_raster_keeps_the_first_records(O, n):
    """A raster that fills up within a launch keeps whole earlier steps and
    counts the rest as dropped."""
    s = mixed_net(n, 10, 3, 6)
    with S.build(s) as net:
        net.run(60)
        net.finish()
        st, ids = net.read_spikes()
    cap = len(st) // 2
    with S.build(s.with_(raster_capacity=cap)) as net:
        net.run(60)
        net.finish()
        st2, ids2 = net.read_spikes()
        assert net.stats()["raster_dropped"] == len(st) - cap
    assert np.array_equal(st2, st[:cap]) and np.array_equal(ids2, ids[:cap])


@pytest.mark.parametrize("n", [2000, 20000])
def test_same_state_as_the_grid_kernels(O, n):
    """A checkpoint passes between the window kernel and k_step in the middle
    of a window; the rest of the run is the same."""
    s = mixed_net(n, 15, 6, 11, sources=40)
    with S.build(s) as net:
        net.run(100)
        net.finish()
        ck = net.checkpoint()
        net.clear_spikes()
        net.run(97)
        net.finish()
        a = net.read_spikes() + net.read_state()
    with S.build(s) as net:
        net.set_tuning(blocks_per_sm=1)  # k_step
        net.restore(ck)
        net.run(97)
        net.finish()
        b = net.read_spikes() + net.read_state()
    assert len(a[0]) > 100
    assert all(np.array_equal(x, y) for x, y in zip(a, b))


def test_grid_wait_runs_out(lib):
    """The grid form's barriers are bounded like k_step's."""
    net = S.build(mixed_net(20000, 10, 3, 6))
    try:
        net.run(5)
        net.finish()
        capi.call("naer_net_set_wait_limit", net.handle, 1000)  # 1 ms
        capi.call("naer_test_set_barrier_skew", net.handle, 1)
        net.run(130)
        assert lib.naer_net_finish(net.handle) == capi.NAER_E_TIMEOUT
        assert lib.naer_net_step(net.handle, 1) == capi.NAER_E_STATE
    finally:
        net.close()


def uneven_members():
    """Cluster sizes of 1 to 8 blocks, one and four neurons a lane, static and
    plastic, windows of one and of many steps."""
    ms = [S.plastic_indegree(n=n, k=k, seed=i, drive_rate_hz=30.0, stdp=i % 2 == 0).with_(exact=True)
          for i, (n, k) in enumerate([(600, 40), (1601, 90), (5003, 150), (2222, 300), (9001, 200), (800, 60), (3100, 25),
                                      (12000, 100), (1000, 500), (450, 20)])]
    ms += [mixed_net(n, 12, dmin, dmax, sources=src, seed=40 + n, exact=True)
           for n, dmin, dmax, src in [(700, 15, 15, 90), (2500, 3, 30, 0), (6500, 7, 9, 260)]]
    return ms


@pytest.mark.parametrize("record", [True, False])
def test_batch_members_as_alone(lib, record):
    ms = uneven_members()
    runs = [64, 7, 130]
    with Batch(ms, exact=True, raster_capacity=1 << 22 if record else 1).compile() as b:
        l0 = b.stats()["kernel_launches"]
        for c in runs:
            b.run(c)
        b.finish()
        assert b.stats()["kernel_launches"] - l0 == 2 * sum((c + 63) // 64 for c in runs)
        spikes = b.read_spikes()
        states = [b.read_state(i, m.neurons) for i, m in enumerate(ms)]
    if record:
        assert np.all(np.diff(spikes[1].astype(np.int64)) >= 0)  # step by step
    for i, m in enumerate(ms):
        with S.build(m) as net:
            net.run(sum(runs))
            net.finish()
            st, ids = net.read_spikes()
            v, r = net.read_state()
        assert np.array_equal(states[i][0].view(np.uint32), v.view(np.uint32)), i
        assert np.array_equal(states[i][1], r), i
        if record:
            bst, bids = b.member_spikes(i, spikes)
            assert len(ids) > 5 and np.array_equal(bst, st) and np.array_equal(bids, ids), i
