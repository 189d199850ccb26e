"""A batch's phase times describe all of its members, also where each steps in
a cluster of its own."""
import pytest

from naer_b200 import spec as S
from naer_b200.forms import Batch

from test_gpu_group import mixed_net

pytestmark = pytest.mark.gpu


def phase_ms(members, steps=640):
    with Batch(members, exact=True).compile() as b:
        b.run(64)
        b.finish()
        p0, l0 = b.phases(), b.stats()["kernel_launches"]
        b.run(steps)
        b.finish()
        p1 = b.phases()
        assert b.stats()["kernel_launches"] - l0 == 2 * steps // 64  # clusters and their raster
    return sum(p1.values()) - sum(p0.values())


def test_mean_over_members(lib):
    """Twelve networks with windows of 15 steps beside a plastic one (windows
    of one step: several times their time per step).  The mean stays near
    theirs; the plastic one's own time is more than twice that."""
    short = [mixed_net(700, 15, 15, 15, sources=90, seed=i, exact=True) for i in range(13)]
    plastic = S.plastic_indegree(n=5000, k=300, seed=2, drive_rate_hz=30.0).with_(exact=True)
    alone = phase_ms(short)
    assert 0 < phase_ms([plastic] + short[1:]) < 2 * alone
    assert phase_ms([plastic] * 4) > 2 * alone
