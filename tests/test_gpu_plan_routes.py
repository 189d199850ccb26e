"""Networks far more active than their description lets expect: the form chosen
for a few events a step must deliver hundreds of thousands.  Against the
oracle, bit for bit; launches show that the window kernel stepped them."""
import numpy as np
import pytest

from naer_b200 import _capi as capi
from naer_b200 import spec as S

from test_gpu_group import assert_matches, mixed_net

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def O(oracle_mod, lib):
    return oracle_mod


def chain_reaction(n, k, dmin=1, dmax=3, **kw):
    """A few driven neurons set off the others, each of whose spikes fires its
    targets: nearly all of them fire as often as they can."""
    s = S.NetSpec(name="chain_reaction", poisson_seed=11, **kw)
    A = s.add_pop(S.NOP, 40, drive_rate_hz=400.0, drive_weight=21.0, drive_seed=3)
    B = s.add_pop(S.NOP, n)
    R = capi.CONN_FIXED_OUTDEGREE
    s.connect(A, B, R, 25.0, degree=k, dmin=dmin, dmax=dmax, seed=1)
    s.connect(B, B, R, 25.0, degree=k, dmin=dmin, dmax=dmax, seed=2)
    return s


@pytest.mark.parametrize("n,k,dmin", [
    (6000, 700, 1),     # one cluster, block-local delivery
    (6000, 1500, 1),    # one cluster, spikes exchanged
    (11000, 600, 1),    # one cluster, two chunks a warp
    (6000, 400, 5),     # one cluster, windows of five steps
    (20000, 500, 1),    # the grid, block-local
    (60000, 1400, 1),   # the grid, spikes exchanged
])
def test_static(O, n, k, dmin):
    assert_matches(O, chain_reaction(n, k, dmin, dmin + 2), [1, 64, 20])


@pytest.mark.parametrize("n,k", [
    (5900, 400),        # one cluster, more list starts than its warps keep
    (30000, 300),       # the grid
])
def test_deterministic(O, n, k):
    s = chain_reaction(n, k)
    for c in s.conns:
        c.weight, c.wmin, c.wmax = 0.0, 22.0, 25.0
    assert_matches(O, s.with_(deterministic=True), [1, 64, 20])


@pytest.mark.parametrize("n,k,rate,mode", [
    (2000, 3000, 400.0, dict(exact=True)),
    (6000, 700, 200.0, dict(deterministic=True)),
    (12000, 1500, 100.0, dict(exact=True)),
])
def test_expected_to_be_busy(O, n, k, rate, mode):
    """Small networks with many events a step: the grid, not a cluster."""
    s = mixed_net(n, k, 1, 9, rate=rate)
    assert_matches(O, s.with_(**mode), [1, 64, 20])


def test_grid_kernel_for_many_events(O):
    """Where k_step is expected to be faster it runs, with its draws: two
    launches of up to 64 steps."""
    s = S.NetSpec(name="dense", poisson_seed=4)
    E = s.add_pop(S.NOP, 30000, drive_rate_hz=300.0, drive_weight=21.0, drive_seed=3)
    s.connect(E, E, capi.CONN_FIXED_OUTDEGREE, 1.0, degree=2000, dmin=1, dmax=9, seed=2)
    with S.build(s) as net:
        net.run(64)
        net.finish()
        st, ids = net.read_spikes()
        stats = net.stats()
    assert stats["kernel_launches"] == 2
    o = O.OracleNet(s, deterministic=True)
    o.run(64)
    ost, oids = o.spikes()
    assert len(oids) > 1000 and np.array_equal(st, ost) and np.array_equal(ids, oids) and stats["events"] == o.events
    o.close()
