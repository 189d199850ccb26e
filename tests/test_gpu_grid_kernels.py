"""The grid kernels (k_step, k_run, k_det_step with k_drive) on small networks,
which step on the window kernel unless a geometry or the two-barrier kernel is
named: against the oracle, bit for bit, whatever the launches' lengths."""
import numpy as np
import pytest

from naer_b200 import _capi as capi
from naer_b200 import spec as S

from nets import mixed_rules, reference_brunel
from test_gpu_group import mixed_net
from test_window_ring import driven

pytestmark = pytest.mark.gpu

KERNELS = {"k_step": (dict(exact=True), dict(blocks_per_sm=2)),
           "k_run": (dict(exact=True), dict(step_kernel=capi.KERNEL_TWO_BARRIER)),
           "k_det_step": (dict(deterministic=True), dict(blocks_per_sm=2))}

NETS = {"five neurons": lambda: mixed_net(5, 3, 1, 3, sources=70, rate=2000.0),
        "one chunk": lambda: mixed_net(1000, 20, 1, 12, sources=24),
        "several chunks": lambda: mixed_net(6100, 60, 4, 9, sources=1100),
        "longest delays": lambda: mixed_net(700, 12, 200, 254),
        "long rows": lambda: mixed_net(3000, 1400, 1, 20, rate=60.0),
        "no synapses": lambda: driven(1500),
        "bernoulli": lambda: mixed_rules(capi.CONN_REF_BERNOULLI),
        "reference brunel": reference_brunel,
        "plastic": lambda: S.plastic_indegree(n=900, k=60, seed=5, drive_rate_hz=60.0),
        "plastic, several chunks": lambda: S.plastic_indegree(n=5000, k=90, seed=6, drive_rate_hz=60.0)}


@pytest.mark.parametrize("kernel", KERNELS)
@pytest.mark.parametrize("name", NETS)
def test_small_networks(oracle_mod, lib, name, kernel):
    mode, tuning = KERNELS[kernel]
    s = NETS[name]().with_(**mode)
    runs = [1, 64, 150]
    with S.build(s) as net:
        net.set_tuning(**tuning)
        for c in runs:
            net.run(c)
        net.finish()
        st, ids = net.read_spikes()
        v, r = net.read_state()
        stats = net.stats()
        w = net.read_csr()[2] if s.stdp_enabled else None
    o = oracle_mod.OracleNet(s, deterministic=None if s.exact else True)
    o.run(sum(runs))
    ost, oids = o.spikes()
    ov, orr = o.state()
    oev, ow = o.events, o.weights() if s.stdp_enabled else None
    o.close()
    assert stats["kernel_launches"] == 2 * sum((c + 63) // 64 for c in runs)  # k_drive and the step kernel
    assert len(oids) > 20 and stats["events"] == oev
    assert np.array_equal(st, ost) and np.array_equal(ids, oids)
    assert np.array_equal(v.view(np.uint32), ov.view(np.uint32)) and np.array_equal(r, orr)
    if w is not None:
        assert np.array_equal(w.view(np.uint32), ow.view(np.uint32))
