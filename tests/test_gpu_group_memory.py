"""Device memory of the window kernel: the spike records of a batch's windows
are bounded."""
import numpy as np
import pytest

from naer_b200.forms import Batch

from test_gpu_group import mixed_net
from naer_b200 import spec as S

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
