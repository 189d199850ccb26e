"""Device memory of the window kernel: the spike records of a batch's windows
are bounded, and without memory for its buffers a network steps on the grid
kernels instead of failing to compile."""
import numpy as np
import pytest

from naer_b200 import _capi as capi
from naer_b200 import spec as S
from naer_b200.forms import Batch

from test_gpu_group import mixed_net

pytestmark = pytest.mark.gpu


def test_records_of_long_windows_are_bounded(lib):
    """720k neurons with windows of 16 steps would take 370 MB of records;
    at most 8e6 of 32 bytes are kept, and results do not change."""
    ms = [mixed_net(12_000, 3, 16, 20, seed=i, exact=True) for i in range(60)]
    one = [mixed_net(12_000, 3, 1, 20, seed=i, exact=True) for i in range(60)]  # windows of one step, same ring
    with Batch(one, exact=True, raster_capacity=1 << 20).compile() as b:
        base = b.stats()["device_bytes"]
    with Batch(ms, exact=True, raster_capacity=1 << 20).compile() as b:
        assert b.stats()["device_bytes"] - base <= 8_000_000 * 32 + (8 << 20)
        l0 = b.stats()["kernel_launches"]
        b.run(40)
        b.finish()
        assert b.stats()["kernel_launches"] - l0 == 2  # the window kernel and its raster
        spikes = b.read_spikes()
        got = [b.member_spikes(i, spikes) + b.read_state(i, ms[i].neurons) for i in (0, 59)]
    for i, g in zip((0, 59), got):
        with S.build(ms[i]) as net:
            net.run(40)
            net.finish()
            want = net.read_spikes() + net.read_state()
        assert len(want[1]) > 100 and all(np.array_equal(x, y) for x, y in zip(g, want))


def test_no_memory_for_its_buffers(lib):
    """Every allocation of a compile fails in turn: one of the window kernel's
    own leaves the network compiled, on k_drive + k_step (two launches of up to
    64 steps), with the same results and no more memory than those need."""
    s = mixed_net(14_000, 12, 12, 14, sources=33)
    with S.build(s) as net:
        net.run(64)
        net.finish()
        want = net.read_spikes() + net.read_state()
        assert net.stats()["kernel_launches"] == 1
        most = net.stats()["device_bytes"]
    fell_back = 0
    try:
        for k in range(400):
            net = S.describe(s, device=0)
            try:
                capi.call("naer_test_fail_allocation", k)
                rc = lib.naer_net_compile(net.handle)
                capi.call("naer_test_fail_allocation", -1)
                if rc == capi.NAER_E_OOM:
                    continue
                assert rc == capi.NAER_OK
                net.run(64)
                net.finish()
                launches = net.stats()["kernel_launches"]
                got = net.read_spikes() + net.read_state()
                assert all(np.array_equal(x, y) for x, y in zip(got, want)), k
                if launches == 1:
                    break  # no allocation failed
                assert launches == 2 and net.stats()["device_bytes"] < most, k
                fell_back += 1
            finally:
                net.close()
    finally:
        capi.call("naer_test_fail_allocation", -1)
    assert launches == 1 and fell_back >= 6  # chunks, segments, counts, spike bits, records
