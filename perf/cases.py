"""Performance cases of the framework: what a user has it do, at the sizes users run.

A case is one network (or a batch, or a stream of jobs) and one pass over
it: a number of grid steps through the public API, then the results a program
reads back (spikes, membrane potentials and refractory counters, weights
where they are learned).  A pass continues the simulation where the last one
ended, as a program's own loop does.

Network families (all from the reference's builders or this repository's
workloads):

  brunel    the reference's Brunel network in volts: N/2 Poisson sources, 0.4 N
            excitatory and 0.1 N inhibitory neurons, p = 0.1, weights 2/N and
            -10/N, one axonal delay of 1.5 ms, stepped window by window
  explicit  the same shape with the caller's own CSR and a driving weight of 1 mV
  outdegree LIF neurons 80/20, fixed out-degree, delays of 1 to 16 steps,
            a Poisson drive per neuron
  indegree  fixed in-degree, delays of 1 to 20 steps, random excitatory weights
  plastic   fixed in-degree with pair STDP on the excitatory synapses

Atomic aggregation adds floats in whatever order they land.  Its cases carry
weights of few significant bits, whose sums are exact in 32 bits, so that a
run can be compared with another spike by spike; the others use the exact-sum
or the deterministic mode, whose results do not depend on the order.
"""
import math

import numpy as np
import torch

from naer_b200 import _capi as capi
from naer_b200 import spec as S
from naer_b200.forms import Batch, Server

DT_US = 100
WINDOW = 15  # grid steps of the reference's 1.5 ms window


def listed():
    return [
        # a controller that advances a small network by one window and reads what it did: pure latency
        dict(name="closed_loop_window", kind="net", family="explicit", n=1003, k=20, agg="atomic", windows=1, settle=300),
        # the reference's benchmark network at its smallest size, driven as its main() does, 0.3 s
        dict(name="brunel_2k", kind="net", family="brunel", n=2000, k=0, agg="atomic", windows=200),
        # the same at the size of its larger sweeps (1.8e8 synapses), 90 ms
        dict(name="brunel_60k", kind="net", family="brunel", n=60001, k=0, agg="atomic", windows=60),
        # a desktop-sized network with heterogeneous delays, 100 ms
        dict(name="outdegree_5k", kind="net", family="outdegree", n=4999, k=100, agg="atomic", steps=1000),
        # an ordinary cortical-scale network: 2e8 synapses, 50 ms
        dict(name="outdegree_200k", kind="net", family="outdegree", n=200000, k=1000, agg="atomic", steps=500),
        # the largest: 1M neurons, 1e9 synapses, 100 ms, raster into pinned memory
        dict(name="outdegree_1m", kind="net", family="outdegree", n=1000000, k=1000, agg="atomic", steps=1000, raw=True),
        # reproducible runs with random weights, 100 ms
        dict(name="indegree_50k_exact", kind="net", family="indegree", n=50001, k=400, agg="exact", steps=1000),
        # float sums in canonical order, for comparison with a CPU run, 30 ms
        dict(name="outdegree_100k_det", kind="net", family="outdegree", n=100000, k=500, agg="det", steps=300),
        # a learning experiment that looks at its weights after every 50 ms
        dict(name="plastic_5k_weights", kind="net", family="plastic", n=5003, k=200, agg="exact", steps=500, weights=True),
        # learning at the size of the plastic benchmark workload, 100 ms
        dict(name="plastic_100k", kind="net", family="plastic", n=100000, k=1000, agg="exact", steps=1000),
        # a parameter sweep: 48 uneven networks in one batch, half of them plastic, 50 ms each
        dict(name="batch_48", kind="batch", members=48, n=50000, k=1000, steps=500),
        # simulation jobs handed to the server at once, rasters back
        dict(name="served_24", kind="served", members=24, n=20000, k=500, steps=2000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    form = rng.choice(["brunel", "brunel", "explicit", "outdegree", "outdegree", "outdegree", "indegree", "det", "plastic", "plastic",
                       "batch", "served"])
    if form == "brunel":
        return dict(kind="net", family="brunel", n=_log(rng, 1500, 60000), k=0, agg=rng.choice(["atomic", "exact"]),
                    windows=_log(rng, 4, 60))
    if form == "explicit":
        return dict(kind="net", family="explicit", n=_log(rng, 200, 4000), k=rng.randint(5, 40), agg="atomic",
                    windows=_log(rng, 1, 40), settle=300)
    if form == "batch":
        return dict(kind="batch", members=rng.randint(3, 40), n=_log(rng, 4000, 30000), k=rng.randint(200, 800),
                    steps=_log(rng, 60, 500))
    if form == "served":
        return dict(kind="served", members=rng.randint(3, 20), n=_log(rng, 3000, 20000), k=rng.randint(150, 500),
                    steps=_log(rng, 300, 1500))
    if form == "plastic":
        return dict(kind="net", family="plastic", n=_log(rng, 1000, 80000), k=rng.randint(50, 800), agg=rng.choice(["exact", "det"]),
                    steps=_log(rng, 30, 500))
    if form == "det":
        return dict(kind="net", family="outdegree", n=_log(rng, 2000, 150000), k=rng.randint(50, 600), agg="det",
                    steps=_log(rng, 30, 300))
    return dict(kind="net", family=form, n=_log(rng, 500, 400000), k=rng.randint(20, 700),
                agg="exact" if form == "indegree" else rng.choice(["atomic", "exact"]), steps=_log(rng, 20, 600))


def _few_bits(x, bits=6):
    """x rounded to `bits` significant bits."""
    m, e = math.frexp(x)
    return math.ldexp(round(m * 2**bits), e - bits)


def _steps(case):
    return case["windows"] * WINDOW if "windows" in case else case["steps"]


def _spec(case, seed):
    """The network of a case as a declarative description."""
    n, k, fam = case["n"], case["k"], case["family"]
    agg = dict(exact=case["agg"] == "exact", deterministic=case["agg"] == "det")
    if fam in ("brunel", "explicit"):
        return _brunel(case, seed, agg)
    if fam == "outdegree":
        s = S.scatter_outdegree(n=n, k=k, seed=seed)
        if case["agg"] == "atomic":  # 0.1 and -0.5 mV in the workload; here sums of them are exact
            for c in s.conns:
                c.weight = 0.125 if c.weight > 0 else -0.5
        return s.with_(**agg)
    s = S.plastic_indegree(n=n, k=k, seed=seed, stdp=fam == "plastic")
    if fam == "indegree":
        for c in s.conns:
            if c.weight > 0:  # weight 0 asks for random weights
                c.weight, c.wmin, c.wmax = 0.0, 0.02, 0.18
    return s.with_(**agg)


def _brunel(case, seed, agg):
    n, fam = case["n"], case["family"]
    s = S.NetSpec(name=fam, poisson_seed=seed & 0xFFFFFFFF, **agg)
    if fam == "brunel":
        np_, ne, ni = n // 2, n * 4 // 10, n // 10
        lif = dict(v_th=0.020, v_reset=0.0, t_ref_ms=2.0, tau_m_ms=20.0)
        we = _few_bits(2.0 / n)
        wi, wp, rate, p = -5.0 * we, we, 20.0, 0.1
    else:  # potentials in mV, 1,000 sources at 10 Hz onto every neuron with 1 mV
        np_, ne = 1000, n * 4 // 5
        ni = n - ne
        lif, we, wi, wp, rate, p = {}, 0.125, -0.5, 1.0, 10.0, 0.0
    P = s.add_pop(S.POISSON, np_, rate_hz=rate)
    E = s.add_pop(S.NOP, ne, **lif)
    I = s.add_pop(S.NOP, ni, **lif)
    rng = np.random.default_rng(seed)
    for i, (src, dst, w) in enumerate([(P, E, wp), (P, I, wp), (E, E, we), (E, I, we), (I, E, wi), (I, I, wi)]):
        if fam == "brunel":
            s.connect(src, dst, capi.CONN_REF_BERNOULLI, w, probability=p, dmin=WINDOW, dmax=WINDOW, seed=seed * 7919 + i)
            continue
        ns, nd = s.pops[src].size, s.pops[dst].size
        deg = rng.binomial(nd, 0.1 if src == P else min(1.0, case["k"] / n), size=ns)
        rp = np.concatenate([[0], np.cumsum(deg)]).astype(np.uint64)
        m = int(rp[-1])
        s.connect_csr(src, dst, rp, rng.integers(0, nd, m), np.full(m, w), np.full(m, WINDOW))
    return s


def _members(case, seed):
    lo = (case["n"] // 20, case["k"] // 8)
    sizes = dict(seed=case["members"], n_range=(lo[0], case["n"]), k_range=(lo[1], case["k"]))  # of the case, not of the seed
    if case["kind"] == "batch":
        ms = S.batch_members(case["members"], **sizes)
    else:
        jobs = S.served_jobs(case["members"], duration_ms=(case["steps"] * 0.02, case["steps"] * 0.1), **sizes)
        ms = [m for _, m, _ in jobs]
    for m in ms:
        for p in m.pops:
            p.drive_seed = (p.drive_seed + 1009 * seed) & 0xFFFFFFFF
        for c in m.conns:
            c.seed += 100_003 * seed
    return ms if case["kind"] == "batch" else [(m, steps) for m, (_, _, steps) in zip(ms, jobs)]


class _Raster:
    """A program's own arrays for the spikes of one pass, unused entries 0."""

    def __init__(self, neurons, steps, columns):
        self.a = np.zeros((columns, int(neurons * (1.0 + 0.01 * steps)) + 1024), dtype=np.uint32)
        self.used = 0

    def keep(self, *columns):
        m = min(len(columns[0]), self.a.shape[1])
        for row, c in zip(self.a, columns):
            row[:m] = c[:m]
            row[m:self.used] = 0
        self.used = m
        return self.a


def prepare(case, seed):
    """The built network, batch or server a program holds between passes."""
    seed = int(seed) % 100_000 + 1
    if case["kind"] == "batch":
        ms = _members(case, seed)
        sizes = [m.neurons for m in ms]
        return dict(case=case, batch=Batch(ms, exact=True).compile(), sizes=sizes, raster=_Raster(sum(sizes), case["steps"], 3))
    if case["kind"] == "served":
        return dict(case=case, server=Server(budget_bytes=8 * 10**9, exact=True), jobs=_members(case, seed),
                    raster=_Raster(case["members"] * case["n"], case["steps"] // 2, 2))
    spec = _spec(case, seed)
    st = dict(case=case, net=S.build(spec), raster=_Raster(spec.neurons, _steps(case), 2))
    if case.get("settle"):  # steps behind it: events are on their way
        st["net"].run(case["settle"])
        st["net"].clear_spikes()
    if case.get("raw"):
        st["records"] = torch.empty((4_000_000, 2), dtype=torch.int32, pin_memory=torch.cuda.is_available()).numpy().view(np.uint32)
    return st


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        b = state["batch"]
        b.run(case["steps"])
        b.finish()
        member, steps, ids = b.read_spikes()
        states = [b.read_state(i, n) for i, n in enumerate(state["sizes"])]
        b.clear_spikes()
        return dict(count=len(ids), raster=state["raster"].keep(member, steps, ids), v=np.concatenate([v for v, _ in states]),
                    refractory=np.concatenate([r for _, r in states]))
    if case["kind"] == "served":
        srv = state["server"]
        jobs = [srv.submit(m, steps) for m, steps in state["jobs"]]
        got = []
        for j in jobs:
            srv.wait(j)
            got.append(srv.spikes(j))
            srv.release(j)
        return dict(count=np.array([len(s) for s, _ in got]),
                    raster=state["raster"].keep(np.concatenate([s for s, _ in got]), np.concatenate([i for _, i in got])))
    net = state["net"]
    if "windows" in case:
        for _ in range(case["windows"]):
            net.step()
    else:
        net.run(case["steps"])
    net.finish()
    out = {}
    if case.get("raw"):
        out["count"] = net.read_raster(state["records"])
    else:
        steps, ids = net.read_spikes()
        out["count"], out["raster"] = len(ids), state["raster"].keep(steps, ids)
    net.clear_spikes()
    out["v"], out["refractory"] = net.read_state()
    if case.get("weights"):
        out["weights"] = net.read_csr()[2]
    return out


# Expected spikes per second and neuron of each family.
_RATE = dict(outdegree=10.0, indegree=5.0, plastic=5.0, brunel=26.0, explicit=10.0)


def _work(n, sources, rows, rate, steps, plastic, n_syn):
    """Bytes and operations of `steps` steps: the rows of the spikes that happen (9 B a synapse, once each where a
    pass visits them again; a plastic one is written back too), neuron state in and out, 8 B a spike."""
    spikes = rate * sources * steps * DT_US * 1e-6
    events = spikes * rows
    visited = min(events, n_syn)
    return visited * (13.0 if plastic else 9.0) + 10.0 * n + 8.0 * spikes, events * (12.0 if plastic else 1.0) + 4.0 * n * steps


def work(case):
    if case["kind"] != "net":
        b = f = 0.0
        for m in _members(case, 1):
            m, steps = m if isinstance(m, tuple) else (m, case["steps"])
            k = sum(c.degree for c in m.conns) / 2.0
            x = _work(m.neurons, m.neurons, k, 5.0, steps, m.stdp_enabled, k * m.neurons)
            built = 9.0 * k * m.neurons if case["kind"] == "served" else 0.0
            b, f = b + x[0] + built, f + x[1]
        return dict(bytes=b, flops=f)
    n, fam, steps = case["n"], case["family"], _steps(case)
    sources, rows = n, float(case["k"])
    if fam == "brunel":
        rows = 0.05 * n
    elif fam == "explicit":
        sources, rows = n + 1000, (100.0 * n + case["k"] * n) / (n + 1000)
    b, f = _work(n, sources, rows, _RATE[fam], steps, fam == "plastic", sources * rows)
    if case.get("weights"):
        b += 4.0 * n * case["k"]
    return dict(bytes=b, flops=f)


# ---------------------------------------------------------------------------
# The same networks in 64 bits, in plain torch: connectivity and Poisson
# streams from the counter-based generator, the membrane, the ring and the
# weights in double.

_M0, _M1, _W0, _W1, _U32 = 0xD2511F53, 0xCD9E8D57, 0x9E3779B9, 0xBB67AE85, 0xFFFFFFFF


def _mulhilo(m, a):
    hi = (((a >> 16) * m) + (((a & 0xFFFF) * m) >> 16)) >> 16
    return hi, (a * m) & _U32


def _philox(c0, c1, c2, k0, k1):
    """Philox4x32-10 of counter {c0, c1, c2, 0}; int64 tensors (or ints) of 32-bit values."""
    c3 = torch.zeros_like(c0)
    c1, c2 = c1 + c3, c2 + c3
    for _ in range(10):
        h0, l0 = _mulhilo(_M0, c0)
        h1, l1 = _mulhilo(_M1, c2)
        c0, c1, c2, c3 = h1 ^ c1 ^ k0, l1, h0 ^ c3 ^ k1, l0
        k0, k1 = (k0 + _W0) & _U32, (k1 + _W1) & _U32
    return c0, c1, c2, c3


def _synapses(spec, base, dev):
    """(source, target, weight, delay) of every synapse; addresses from `base`."""
    parts = []
    for c in spec.conns:
        ns, nd = spec.pops[c.src].size, spec.pops[c.dst].size
        lo, hi = c.seed & _U32, (c.seed >> 32) & _U32
        if c.csr is not None:
            rp, tg, w, d = (torch.from_numpy(np.asarray(a).astype(np.float64 if i == 2 else np.int64)).to(dev) for i, a in enumerate(c.csr))
            src = torch.repeat_interleave(torch.arange(ns, device=dev), rp[1:] - rp[:-1])
            parts.append((src + base[c.src], tg + base[c.dst], w, d))
            continue
        w32 = float(np.float32(c.weight))
        if c.rule == capi.CONN_REF_BERNOULLI:
            rows = max(1, (1 << 24) // max(1, nd))
            dd = torch.arange(nd, device=dev)[None, :]
            for r0 in range(0, ns, rows):
                ss = torch.arange(r0, min(ns, r0 + rows), device=dev)[:, None]
                z = _philox(dd + 0 * ss, 0, 0, (ss * 32 + (dd & 31)) & _U32, lo)[2]
                hit = (z.double() / 4294967295.0 < c.probability).nonzero()
                one = torch.ones(len(hit), dtype=torch.float64, device=dev)
                parts.append((hit[:, 0] + r0 + base[c.src], hit[:, 1] + base[c.dst], w32 * one, (c.dmin * one).long()))
            continue
        indegree = c.rule == capi.CONN_FIXED_INDEGREE
        own, other = (nd, ns) if indegree else (ns, nd)  # who draws its partners
        blocks = (c.degree + 3) // 4
        i = torch.arange(own, device=dev)[:, None]
        b = torch.arange(blocks, device=dev)[None, :]
        word = lambda j: torch.stack(_philox(i + 0 * b, b, j, lo, hi), 2).reshape(own, 4 * blocks)[:, :c.degree].reshape(-1)  # noqa: E731
        span = lambda x, m: (((x >> 16) * m) + (((x & 0xFFFF) * m) >> 16)) >> 16  # noqa: E731
        mate, dly = span(word(0), other), c.dmin + span(word(1), c.dmax - c.dmin + 1)
        if c.weight == 0.0:
            x = (word(2) >> 8).float() * np.float32(1.0 / 16777216.0)
            w = (np.float32(c.wmin) + np.float32(np.float32(c.wmax) - np.float32(c.wmin)) * x).double()
        else:
            w = torch.full((own * c.degree,), w32, dtype=torch.float64, device=dev)
        me = torch.repeat_interleave(torch.arange(own, device=dev), c.degree)
        src, dst = (mate, me) if indegree else (me, mate)
        parts.append((src + base[c.src], dst + base[c.dst], w, dly))
    return [torch.cat(x) for x in zip(*parts)]


def _poisson(rate, seed, n_gen, idx, t0, dt):
    """Events of generators `idx` in the windows [t0, t0 + dt), int64 tensors that broadcast."""
    key = (idx // 2048) * 128 + (idx % 2048) % 128

    def interval(z):
        x = torch.log(1.0 - z.double() / 4294967295.0) / -(rate / 1e6)
        return x.clamp(max=4294967295.0).long()

    zero = torch.zeros_like(idx + t0)
    idx, key, t0 = idx + zero, key + zero, t0 + zero
    time = t0 + interval(_philox((t0 * n_gen + idx) & _U32, 0, 0, key, seed)[2])
    count = zero
    for _ in range(10):
        live = (time < t0 + dt).nonzero(as_tuple=True)
        if not len(live[0]):
            break
        count[live] += 1
        time[live] += interval(_philox((time[live] * n_gen + idx[live]) & _U32, 0, 0, key[live], seed)[2])
    return count


def _simulate(spec, steps, want_weights):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    order = sorted(range(len(spec.pops)), key=lambda i: spec.pops[i].type)
    base, at = {}, 0
    for i in order:
        base[i] = at
        at += spec.pops[i].size
    n = at
    src, tgt, w, dly = _synapses(spec, base, dev)
    # rows of a source in the order read_csr lists them: connections as declared, then the delay-1 synapses first
    perm = torch.sort(src * 2 + (dly > 1), stable=True).indices
    src, tgt, w, dly = src[perm], tgt[perm], w[perm], dly[perm]
    row = torch.searchsorted(src, torch.arange(n + 1, device=dev))
    D = int(dly.max()) + 1
    ring = torch.zeros(D * n, dtype=torch.float64, device=dev)
    full = lambda f: torch.cat([torch.full((spec.pops[i].size,), float(f(spec.pops[i])), dtype=torch.float64, device=dev) for i in order])  # noqa: E731
    f32 = lambda x: float(np.float32(x))  # noqa: E731
    decay = full(lambda p: math.exp(-spec.dt_us / (f32(p.tau_m_ms) * 1000.0)))
    v_th, v_reset, drive_w = full(lambda p: f32(p.v_th)), full(lambda p: f32(p.v_reset)), full(lambda p: f32(p.drive_weight))
    t_ref = full(lambda p: round(f32(p.t_ref_ms) * 1000.0 / spec.dt_us)).long()
    is_source = full(lambda p: p.type == S.POISSON) > 0
    v = full(lambda p: 0.0 if p.type == S.POISSON else f32(p.v_init))
    refr = torch.zeros(n, dtype=torch.int64, device=dev)
    n_sources = sum(p.size for p in spec.pops if p.type == S.POISSON)
    first_source = n - n_sources
    n_plastic = sum(p.size for p in spec.pops if p.type == S.STDP) if spec.stdp_enabled else 0
    post = torch.full((max(1, n_plastic), spec.stdp_history), -1, dtype=torch.int64, device=dev)  # newest first
    post_y = torch.zeros(max(1, n_plastic), dtype=torch.float64, device=dev)
    pre_t = torch.full((max(1, n_plastic),), -1, dtype=torch.int64, device=dev)
    pre_x = torch.zeros(max(1, n_plastic), dtype=torch.float64, device=dev)
    kp, km = spec.dt_us / (f32(spec.tau_plus_ms) * 1000.0), spec.dt_us / (f32(spec.tau_minus_ms) * 1000.0)
    ap, am, w_max = f32(spec.a_plus) * f32(spec.w_max), f32(spec.a_minus) * f32(spec.w_max), f32(spec.w_max)
    block = max(1, (1 << 24) // n)
    for t in range(steps):
        if t % block == 0:
            t0 = torch.arange(t, min(steps, t + block), device=dev)[:, None] * spec.dt_us
            counts = torch.zeros((len(t0), n), dtype=torch.int64, device=dev)
            for i, p in enumerate(spec.pops):
                idx = torch.arange(p.size, device=dev)[None, :]
                if p.type == S.POISSON and p.rate_hz > 0:
                    counts[:, base[i]:base[i] + p.size] = _poisson(f32(p.rate_hz), spec.poisson_seed, n_sources,
                                                                   idx + base[i] - first_source, t0, spec.dt_us)
                elif p.type != S.POISSON and p.drive_rate_hz > 0:
                    counts[:, base[i]:base[i] + p.size] = _poisson(f32(p.drive_rate_hz), p.drive_seed & _U32, p.size, idx, t0, spec.dt_us)
        m = counts[t % block]
        cell = ring[(t % D) * n:(t % D + 1) * n]
        idle = (refr > 0) | is_source
        x = torch.where(idle, v, v * decay + cell + m * drive_w)
        fired = ~idle & (x > v_th)
        v = torch.where(fired, v_reset, x)
        refr = torch.where(fired, t_ref, (refr - 1).clamp(min=0))
        cell.zero_()
        spiking = (fired | (is_source & (m > 0))).nonzero()[:, 0]
        if not len(spiking):
            continue
        mine = spiking[spiking < n_plastic]
        old_t, old_x = pre_t.clone(), pre_x.clone()
        if len(mine):
            lp = post[mine, 0]
            post_y[mine] = torch.where(lp >= 0, post_y[mine] * torch.exp(-km * (t - lp)), 0.0) + 1.0
            post[mine] = torch.cat([torch.full_like(post[mine, :1], t), post[mine, :-1]], 1)
            pre_x[mine] = torch.where(old_t[mine] >= 0, old_x[mine] * torch.exp(-kp * (t - old_t[mine])), 0.0) + 1.0
            pre_t[mine] = t
        lens = row[spiking + 1] - row[spiking]
        start = torch.cumsum(lens, 0) - lens
        who = torch.repeat_interleave(torch.arange(len(spiking), device=dev), lens)
        j = torch.arange(len(who), device=dev) - start[who] + row[spiking][who]
        source = spiking[who]
        if n_plastic:
            learn = ((source < n_plastic) & (tgt[j] < n_plastic)).nonzero()[:, 0]
            js, a, b = j[learn], source[learn], tgt[j[learn]]
            ww = w[js]
            for h in range(spec.stdp_history - 1, -1, -1):
                tp = post[b, h]
                pair = (old_t[a] >= 0) & (tp > old_t[a])
                ww = torch.where(pair, (ww + ap * old_x[a] * torch.exp(-kp * (tp - old_t[a]))).clamp(max=w_max), ww)
            lp = post[b, 0]
            w[js] = torch.where(lp >= 0, (ww - am * post_y[b] * torch.exp(-km * (t - lp))).clamp(min=0.0), ww)
        amount = w[j] * torch.where(is_source[source], m[source], 1)
        ring.index_add_(0, ((t + dly[j]) % D) * n + tgt[j], amount)
    v = torch.where(is_source, 0.0, v)
    return v.cpu().numpy(), (w.cpu().numpy() if want_weights else None)


def exact(case, seed):
    """Potentials and weights of the first pass in 64 bits; None for the largest networks, long mean-driven runs and the
    forms of many."""
    if case["kind"] != "net":
        return None
    n = case["n"]
    synapses = n * n * 0.05 if case["family"] == "brunel" else n * max(case["k"], 100)
    if synapses > 2.1e8 or (case["family"] == "brunel" and n * _steps(case) > 1e7):  # mean-driven: roundings grow to other spikes
        return None
    seed = int(seed) % 100_000 + 1
    out = dict(count=None, raster=None)
    out["v"], weights = _simulate(_spec(case, seed), case.get("settle", 0) + _steps(case), bool(case.get("weights")))
    out["refractory"] = None
    if case.get("weights"):
        out["weights"] = weights
    return out
