"""The window kernel in the bounds-checked build: its guards name every kind
of buffer it indexes, and none fires over its forms (cluster and grid, one and
four neurons a lane, windows of one and of several steps, the three
aggregations, plasticity, more spikes than the shared list, batches), networks
without synapses among them, which still equal the oracle."""
import json
import os
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def test_every_buffer_has_a_guard():
    """Synapses, ring, queued sources, neuron state, Poisson counts, event
    lists, spike bits, spike records."""
    text = (ROOT / "naer_b200" / "csrc" / "group_kernel.cuh").read_text()
    for code in ("Synapse", "Ring", "Queue", "State", "Drive", "EventList", "Bits", "Record"):
        assert f"kChk{code})" in text, code


CHILD = r"""
import ctypes as C, json, sys
import numpy as np
sys.path.insert(0, sys.argv[1]); sys.path.insert(0, sys.argv[1] + "/tests")
from naer_b200 import _capi as capi
from naer_b200 import spec as S
from naer_b200.forms import Batch
from test_gpu_group import mixed_net, uneven_members
from test_window_ring import connected, driven
from oracle import oracle as O
lib = capi.load()
flag = C.c_int()
capi.call("naer_build_checked", C.byref(flag))
out = {"checked": flag.value, "runs": []}
cases = [(f"driven {n} {d} {e}", driven(n, d, exact=e), True)
         for n in (700, 5000, 20000) for d in (None, 13) for e in (False, True)]
cases += [
    ("cluster", mixed_net(6100, 20, 1, 12, sources=70), False),
    ("cluster, windows", mixed_net(700, 12, 15, 15, sources=33), False),
    ("exchange", mixed_net(6000, 700, 1, 8, sources=50), False),
    ("grid, windows", mixed_net(15000, 12, 3, 40, sources=33), False),
    ("four a lane", mixed_net(120_000, 10, 1, 16, sources=130), False),
    ("four a lane, windows", mixed_net(130_001, 10, 5, 5, sources=130), False),
    ("list overflow", mixed_net(5000, 3, 12, 14, rate=9000.0, t_ref_ms=0.0), False),
    ("det cluster", mixed_net(6000, 700, 2, 30, sources=50).with_(deterministic=True), False),
    ("det grid", mixed_net(30000, 1300, 3, 40, sources=50).with_(deterministic=True), False),
    ("plastic cluster", S.plastic_indegree(n=5000, k=60, seed=5, drive_rate_hz=60.0).with_(exact=True), False),
    ("plastic grid", S.plastic_indegree(n=14000, k=60, seed=5, drive_rate_hz=60.0).with_(exact=True), False),
    ("plastic det", S.plastic_indegree(n=5000, k=600, seed=5, drive_rate_hz=60.0).with_(deterministic=True), False),
]
for name, s, oracle in cases:
    with S.build(s) as net:
        for c in (1, 64, 35):
            net.run(c)
        net.finish()
        code, idx = C.c_uint32(), C.c_uint64()
        capi.call("naer_net_check_report", net.handle, C.byref(code), C.byref(idx))
        st, ids = net.read_spikes()
        r = {"net": name, "code": code.value, "index": idx.value, "spikes": len(ids),
             "launches": int(net.stats()["kernel_launches"])}
        if oracle:
            o = O.OracleNet(s, deterministic=None if s.exact else True)
            o.run(100)
            ost, oids = o.spikes()
            r["same"] = bool(np.array_equal(st, ost) and np.array_equal(ids, oids))
            o.close()
        out["runs"].append(r)
ms = uneven_members() + [driven(900, None, exact=True), driven(4000, 13, exact=True), connected(900, exact=True)]
with Batch(ms, exact=True).compile() as b:
    b.run(100)
    b.finish()  # fails if an access was out of bounds
    out["runs"].append({"net": "batch", "code": 0, "spikes": int(b.stats()["spikes"]), "launches": 0})
print(json.dumps(out))
"""


@pytest.mark.gpu
def test_no_access_out_of_bounds(lib):
    from naer_b200 import build as b
    b.build(checked=True)
    r = subprocess.run([sys.executable, "-c", CHILD, str(ROOT)], capture_output=True, text=True,
                       env=dict(os.environ, NAER_CHECKED="1"), timeout=900)
    assert r.returncode == 0, r.stderr[-4000:]
    out = json.loads(r.stdout.strip().splitlines()[-1])
    assert out["checked"] == 1 and len(out["runs"]) == 25
    for run in out["runs"]:
        assert run["code"] == 0 and run["spikes"] > 0 and run.get("same", True), run
        assert run["launches"] in (0, 4) if run["net"] == "batch" else run["launches"] == 3, run
