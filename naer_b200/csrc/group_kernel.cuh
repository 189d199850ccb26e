// k_group: a step kernel without per-step launches of its own for Poisson
// draws, with fewer barriers than k_step.  Included once, by sim_kernels.cu,
// after the delivery helpers.
//
// Two forms share the code:
//   kGrid = false  a network is stepped by one thread-block cluster,
//                  synchronised by hardware cluster barriers.  Networks do not
//                  interact, so each goes through all the steps of the launch
//                  by itself; the clusters of a launch have one size, larger
//                  networks are launched with larger clusters (Engine::plan_several)
//   kGrid = true   one network is stepped by the whole (cooperative) grid,
//                  synchronised by the bounded grid barrier
// kPer neurons a lane (1 or 4): a warp's time over its neurons is a chain of
// instructions, so networks with few neurons per warp take 1, the others 4
// (vector loads, fewer instructions per neuron).
//
// The steps go in windows of W = the network's smallest synaptic delay (1 for
// a network with plasticity on).  Within a window no spike can reach any
// neuron, so a warp takes its neurons through all W steps with the membrane
// potential in registers and no synchronisation; then the group's spikes of
// the window are delivered together.  Two barriers per window instead of two
// per step, and only one where a block delivers its own spikes (NetDev::local).
//
// kPlastic: with the plasticity code; without it the kernel is shorter, and a
// step passes once through most of its instructions.
//
// kDet: deterministic aggregation of one network, in windows of one step with
// a third barrier (det_link, det_fold).
//
// Of a block's warps, kGroupSteppers step neurons and deliver; the others draw
// the Poisson counts of later steps meanwhile.
//
// What bounds it: a step's chain of latencies (ring loads from L2, 350 to 770
// cycles by die; a few hundred dependent instructions of one warp; row loads;
// the reductions' fence; the barrier), not bytes: on the grid at 200k / 1000
// DRAM is 2.5 % busy, L2 10 %, the SMs 17 %, and 14 of the 23 cycles between a
// warp's instructions are waits at barriers.  Kernel time per grid step (events
// around the launches), against k_drive + k_step: 5k neurons / out-degree 100:
// 3.4 against 8.7 us; 50k / in-degree 400: 5.1 against 9.5; 200k / 1000: 11.0
// against 12.0; 100k plastic / 1000: 11.0 against 13.0; Brunel (delay 15 steps,
// called window by window) 2k: 1.8 against 8.5, 60k / 1.8e8 synapses: 6.3
// against 12.6.
namespace naer {

constexpr uint32_t kGroupWarps = kGroupThreads / 32;
constexpr uint32_t kGroupSteppers = kGroupStepThreads / 32;
constexpr uint32_t kGroupDrawers = kGroupWarps - kGroupSteppers;
constexpr uint32_t kGroupAhead = 4;    // steps drawn ahead of the simulation, at least
constexpr uint32_t kDetStarts = 384;   // list starts a warp keeps (deterministic aggregation)
constexpr uint32_t kGroupQueue = 64;   // windows a warp can hold (31 left over + 32)
static_assert(2 * kGroupMaxWindow <= kDriveSlots, "counts of two windows fit the drive ring");
static_assert(4 * kGroupMaxWindow <= 64, "a lane's spikes of a window fit 64 bits");

// A spike of the current window: source, step within the window, POISSON
// multiplicity or (plastic sources) pre-synaptic state before it, row.
struct __align__(16) GroupSpike {
    uint32_t i;       // storage index
    uint32_t k;       // step within the window
    int32_t aux0;     // SpikeRec::aux0
    float aux1;
    uint4 row;        // row_of
};

struct GroupShared {
    NetDev net;
    PopDev pop[kGroupPops];
    BarrierCfg bcfg;
    int flag, ok;                         // poll_barrier
    unsigned long long ev;
    uint32_t ovf;
    uint32_t n_spikes[2];                 // spikes of the block in this window, by window parity
    uint32_t first[kGroupMaxBlocks + 1];  // grid form: spikes of the blocks before each
    unsigned long long ph[4];             // thread 0 of the group's first block
};

// Barrier of the group.
template <bool kGrid>
__device__ __forceinline__ bool group_barrier(Ctl* ctl, unsigned long long& target, GroupShared& sh) {
    if (kGrid) {
        target += gridDim.x;
        __syncthreads();
        if (threadIdx.x == 0) {
            arrive_barrier(ctl);
            poll_barrier(ctl, target, sh.bcfg, &sh.flag, &sh.ok);
        }
        __syncthreads();
        return sh.ok != 0;
    }
    __syncwarp();  // .aligned
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    return true;
}

// Barrier of the block's stepping warps alone.
__device__ __forceinline__ void steppers_sync() {
    asm volatile("bar.sync 1, %0;" ::"n"(kGroupStepThreads) : "memory");
}

// Address of `p` (this block's shared memory) in block `rank` of the cluster.
__device__ __forceinline__ uint32_t cluster_map(const void* p, uint32_t rank) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ uint32_t cluster_ld(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ uint4 cluster_ld4(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared::cluster.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
    return v;
}

// NAER_CHECKED: a ring cell inside the ring, a spike record inside its
// block's part of the queue.
__device__ __forceinline__ bool ring_ok(const NetDev& np, uint32_t slot, uint32_t i, Ctl* ctl) {
    return NAER_IN_BOUNDS(ctl, slot, np.ring_slots, kChkRing) && NAER_IN_BOUNDS(ctl, i, np.n_storage, kChkRing);
}
__device__ __forceinline__ bool record_ok(const NetDev& np, uint32_t x, Ctl* ctl) {
    return NAER_IN_BOUNDS(ctl, x, np.q_cap, kChkRecord);
}

// Inclusive sum over the warp's lanes.
__device__ __forceinline__ uint32_t warp_scan(uint32_t x, uint32_t lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    return x;
}

// kPer consecutive values of a lane, as one vector access.
template <int kPer>
struct Vals {
    float v[kPer];
};
template <int kPer>
__device__ __forceinline__ Vals<kPer> ld_vals(const float* p) {  // at L2: other blocks' reductions
    Vals<kPer> r;
    if constexpr (kPer == 4) {
        const float4 x = __ldcg(reinterpret_cast<const float4*>(p));
        r.v[0] = x.x, r.v[1] = x.y, r.v[2] = x.z, r.v[3] = x.w;
    } else {
        r.v[0] = __ldcg(p);
    }
    return r;
}
template <int kPer>
__device__ __forceinline__ void clear_vals(float* p) {
    if constexpr (kPer == 4) __stcg(reinterpret_cast<float4*>(p), make_float4(0.f, 0.f, 0.f, 0.f));
    else __stcg(p, 0.0f);
}
// kPer bytes (Poisson counts, refractory counters) of a lane in one word
template <int kPer>
__device__ __forceinline__ uint32_t ld_bytes(const uint8_t* p) {
    if constexpr (kPer == 4) return __ldcg(reinterpret_cast<const unsigned int*>(p));
    else return __ldcg(p);
}

// Resolves n <= 32 queued windows of any populations (drive_resolve; the
// population is in the slot word's upper bits).
__device__ __forceinline__ void group_resolve(const PopDev* pops, uint8_t* drive, uint32_t Ns, uint32_t dt_us,
                                              const DriveWindow* q, uint32_t n, uint32_t lane, Ctl* ctl) {
    __syncwarp();
    if (lane < n) {
        const DriveWindow w = q[lane];
        const PopDev& p = pops[w.slot >> 8];
        const uint32_t idx = (p.type == kPOISSON ? p.rng_idx_base : 0u) + (w.i - p.storage_base);
        const uint32_t cnt = poisson_exact_call(p.rate_hz, p.rng_seed, p.rng_n, idx, w.z0, w.t0, w.t0 + dt_us);
        if (NAER_IN_BOUNDS(ctl, w.i, Ns, kChkDrive))
            __stcg(drive + (size_t)(w.slot & 0xFFu) * Ns + w.i, (unsigned char)cnt);
    }
    __syncwarp();
}

// Poisson counts for step s of 128 neurons, four a lane (of the block's
// chunks [at, at + 4 / kPer)), as k_drive draws them: the common path proves a
// window empty from its first draw, the rest are queued per warp and resolved
// up to 32 at a time.  Bound by the integer-multiply pipe: four draws in
// flight per lane keep it busy from one warp per scheduler.  Returns the
// queue's length.
template <int kPer>
__device__ __forceinline__ uint32_t group_draw(const NetDev& np, const PopDev* pops, const uint2* s_gc, uint32_t at,
                                               uint32_t places, unsigned long long s, DriveWindow* q, uint32_t qn,
                                               uint32_t lane, Ctl* ctl) {
    const uint32_t Ns = np.n_storage, dt = np.dt_us;
    const uint32_t t0 = (uint32_t)(s - np.start_step) * dt, slot = (uint32_t)s % kDriveSlots;
    uint8_t* drive = np.drive + (size_t)slot * Ns;
    uint32_t z[4], i[4], info[4], rare = 0, any = 0;
#pragma unroll
    for (uint32_t u = 0; u < 4; ++u) {
        const uint32_t c = kPer == 4 ? at : at + u;
        const uint2 gc = c < places ? s_gc[c] : make_uint2(0u, 0u);
        info[u] = gc.y;
        i[u] = gc.x + (kPer == 4 ? 4 * lane + u : lane);
        any |= gc.y;
    }
    if (!(any & kGcDrawn)) return qn;  // the same in every lane
#pragma unroll
    for (uint32_t u = 0; u < 4; ++u) {
        const PopDev& p = pops[info[u] & 0xFFu];
        const uint32_t idx = (p.type == kPOISSON ? p.rng_idx_base : 0u) + (i[u] - p.storage_base);
        z[u] = philox_ref_z(t0 * p.rng_n + idx, ref_global_id(idx, kPoissonCapacity, kPoissonWorkgroup), p.rng_seed);
        const uint32_t o = kPer == 4 ? 4 * lane + u : lane;
        const bool live = (info[u] & kGcDrawn) && o < ((info[u] >> 8) & 0xFFu);
        rare |= (live && !poisson_quiet(p, z[u], t0) ? 1u : 0u) << u;
        if (kPer == 1 && live && NAER_IN_BOUNDS(ctl, i[u], Ns, kChkDrive)) __stcg(drive + i[u], (unsigned char)0);
    }
    if (kPer == 4 && 4 * lane < ((info[0] >> 8) & 0xFFu) && NAER_IN_BOUNDS(ctl, i[3], Ns, kChkDrive))
        __stcg(reinterpret_cast<unsigned int*>(drive + i[0]), 0u);
    if (__any_sync(0xFFFFFFFFu, rare != 0)) {
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u) {
            const bool r = (rare >> u) & 1u;
            const uint32_t bal = __ballot_sync(0xFFFFFFFFu, r);
            if (r) q[qn + __popc(bal & ((1u << lane) - 1u))] = DriveWindow{i[u], slot | ((info[u] & 0xFFu) << 8), t0, z[u]};
            qn += __popc(bal);
            if (qn >= 32) {
                qn -= 32;
                group_resolve(pops, np.drive, Ns, dt, q + qn, 32, lane, ctl);
            }
        }
    }
    return qn;
}

struct GroupLif {
    double prop;
    float v_th, v_reset, drive_w, fx_inv;
    uint32_t t_ref;
};

// One step of a lane's neurons; returns their spikes (bit k = neuron k).
// Straight-line code: a branch per neuron (refractory or not) costs more
// than the updates it saves.  Only a step with a drive event (dr: one byte
// per neuron) takes the branch.
template <int kPer>
__device__ __forceinline__ uint32_t group_lif(Vals<kPer>& v, uint32_t& r4, const GroupLif& p, const Vals<kPer>& cell,
                                              uint32_t dr) {
    float x[kPer];
#pragma unroll
    for (int k = 0; k < kPer; ++k) x[k] = lif_update(v.v[k], p.prop, ring_input(cell.v[k], p.fx_inv), 0u, p.drive_w);
    if (dr) {
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            const uint32_t m = (dr >> (8 * k)) & 0xFFu;
            if (m) x[k] = lif_update(v.v[k], p.prop, ring_input(cell.v[k], p.fx_inv), m, p.drive_w);
        }
    }
    uint32_t hit = 0, r_new = 0;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const uint32_t r = (r4 >> (8 * k)) & 0xFFu;
        const bool idle = r > 0, spike = !idle && x[k] > p.v_th;
        v.v[k] = idle ? v.v[k] : spike ? p.v_reset : x[k];
        r_new |= (idle ? r - 1u : spike ? p.t_ref : 0u) << (8 * k);
        hit |= (spike ? 1u : 0u) << k;
    }
    r4 = r_new;
    return hit;
}

// One piece of a static source's row (kWide: 128 synapses in 128-bit loads,
// else 32, one a lane): the weights reduced into the ring.
template <bool kWide>
__device__ __forceinline__ void group_row(const NetDev& np, uint32_t slot, float mult, uint64_t beg, uint32_t len,
                                          uint32_t piece, uint32_t split, uint32_t lane, unsigned long long& ev,
                                          Ctl* ctl) {
    const uint32_t D = np.ring_slots, Ns = np.n_storage;
    float* __restrict__ ring = np.ring;
    const float qs = np.fx_scale;  // exact-sum aggregation: 2^S, else 0
    const uint32_t* __restrict__ tgt_a = np.tgt + beg;
    const float* __restrict__ w_a = np.w + beg;
    const uint8_t* __restrict__ d_a = np.dly + beg;
    uint32_t n = 0;
    auto deliver = [&](uint32_t tgt, float w, uint32_t d) {
        if (tgt == kTgtSentinel || !ring_ok(np, ring_slot(slot, d, D), tgt, ctl)) return;
        if (mult != 1.0f) w = __fmul_rn(w, mult);
        float* cell = ring + (size_t)ring_slot(slot, d, D) * Ns + tgt;
        if (qs != 0.0f) red_add_s32(cell, __float2int_rn(__fmul_rn(w, qs)));
        else red_add_f32(cell, w);
        ++n;
    };
    if (kWide) {
        for (uint32_t off = (piece * 32 + lane) * 4; off < len; off += split * 128) {
            if (!NAER_IN_BOUNDS(ctl, beg + off + 3, np.syn_cap, kChkSynapse)) break;
            const uint4 tg = ld_stream_u4(tgt_a + off);
            const float4 ww = __ldcs(reinterpret_cast<const float4*>(w_a + off));
            const uint32_t dd = ld_stream_u32(d_a + off);
#pragma unroll
            for (int j = 0; j < 4; ++j) deliver(u4_get(tg, j), f4_get(ww, j), (dd >> (8 * j)) & 0xFFu);
        }
    } else {
        for (uint32_t off = piece * 32 + lane; off < len; off += split * 32) {
            if (!NAER_IN_BOUNDS(ctl, beg + off, np.syn_cap, kChkSynapse)) break;
            const uint32_t tgt = __ldcs(tgt_a + off);
            const float w = __ldcs(w_a + off);
            const uint32_t d = __ldcs(d_a + off);
            deliver(tgt, w, d);
        }
    }
    ev += n;
}

// Raster of a launch.  Spikes are left as one bit per neuron (word u of a
// chunk: neuron u of each lane).  raster_count: spikes of step k in segment
// g, by one warp.
__device__ __forceinline__ uint4 raster_bits(const EngineDev& eng, const GroupSeg& seg, uint32_t k, uint32_t x) {
    uint4 m = make_uint4(0u, 0u, 0u, 0u);
    if (x < seg.count && NAER_IN_BOUNDS(eng.ctl, seg.word + (x + 1) * seg.per - 1, eng.group_words, kChkBits)) {
        const uint32_t* bits = eng.group_bits + (size_t)k * eng.group_words + seg.word;
        if (seg.per == 4) m = __ldcg(reinterpret_cast<const uint4*>(bits) + x);
        else m.x = __ldcg(bits + x);
    }
    return m;
}

__device__ __forceinline__ void raster_count(const EngineDev& eng, uint32_t k, uint32_t g, uint32_t lane) {
    const GroupSeg seg = eng.group_segs[g];
    uint32_t n = 0;
    for (uint32_t u = lane; u < seg.count; u += 32) {
        const uint4 m = raster_bits(eng, seg, k, u);
        n += __popc(m.x) + __popc(m.y) + __popc(m.z) + __popc(m.w);
    }
    n = __reduce_add_sync(0xFFFFFFFFu, n);
    if (lane != 0 || n == 0) return;
    if (eng.group_seg_n == 1) {
        __stcg(eng.group_tot + k, n);
        return;
    }
    __stcg(eng.group_q + (size_t)k * eng.group_seg_n + g, n);
    atomicAdd(eng.group_tot + k, n);
}

// Records of segment g in step k, by one warp: in step order and within a
// step in ascending address.  Their place follows from the spikes of the
// earlier steps and of the step's earlier segments.
__device__ __forceinline__ void raster_write(const EngineDev& eng, unsigned long long s0, uint32_t k, uint32_t g,
                                             unsigned long long rbase, uint32_t lane) {
    // with one segment in all, the step's spikes are the segment's
    const uint32_t* q = eng.group_q + (size_t)k * eng.group_seg_n;
    unsigned long long before = 0;
    const uint32_t mine = __ldcg(eng.group_seg_n > 1 ? q + g : eng.group_tot + k);
    for (uint32_t x = lane; x < k; x += 32) before += __ldcg(eng.group_tot + x);
    if (mine == 0) return;  // silent, or its network does not run in this step
    for (uint32_t x = lane; x < g; x += 32) before += __ldcg(q + x);
    const GroupSeg seg = eng.group_segs[g];
    const GroupChunk* chunks = eng.group_chunks + seg.first;
    const PopDev* pops = eng.pops + seg.pop_first;
    unsigned long long at = rbase + warp_sum_u64(before);
    constexpr uint32_t kTile = 2;
    for (uint32_t u0 = lane; u0 - lane < seg.count; u0 += 32 * kTile) {
        uint4 m[kTile];
#pragma unroll
        for (uint32_t u = 0; u < kTile; ++u) m[u] = raster_bits(eng, seg, k, u0 + u * 32);
#pragma unroll
        for (uint32_t u = 0; u < kTile; ++u) {
            const uint32_t c = __popc(m[u].x) + __popc(m[u].y) + __popc(m[u].z) + __popc(m[u].w);
            if (!__any_sync(0xFFFFFFFFu, c != 0)) continue;
            const uint32_t y = warp_scan(c, lane);
            unsigned long long pos = at + (y - c);
            at += __shfl_sync(0xFFFFFFFFu, y, 31);
            if (!c) continue;
            const GroupChunk ch = chunks[u0 + u * 32];
            const PopDev& p = pops[ch.info & 0xFFu];
            const uint32_t id0 = p.id_base + (ch.first - p.storage_base);
            for (uint32_t lanes = m[u].x | m[u].y | m[u].z | m[u].w; lanes; lanes &= lanes - 1) {
                const uint32_t l = __ffs(lanes) - 1;
#pragma unroll
                for (uint32_t v = 0; v < 4; ++v)
                    if ((u4_get(m[u], v) >> l) & 1u) {
                        if (pos < eng.raster_cap)
                            __stcg(eng.raster + pos, make_uint2((uint32_t)(s0 + k), id0 + seg.per * l + v));
                        ++pos;
                    }
            }
        }
    }
}

// End of a launch (one block, after every raster_write): the step and the
// raster cursor advance, the counts are cleared for the next launch.
__device__ __forceinline__ void raster_end(const EngineDev& eng, unsigned long long s0, uint32_t nsteps,
                                           unsigned long long rbase) {
    Ctl* ctl = eng.ctl;
    if (eng.record)
        for (size_t x = threadIdx.x; eng.group_seg_n > 1 && x < (size_t)nsteps * eng.group_seg_n; x += blockDim.x)
            __stcg(eng.group_q + x, 0u);
    if (threadIdx.x < 32) {
        unsigned long long n = 0;
        if (eng.record)
            for (uint32_t k = threadIdx.x; k < nsteps; k += 32) {
                n += __ldcg(eng.group_tot + k);
                __stcg(eng.group_tot + k, 0u);
            }
        n = warp_sum_u64(n);
        if (threadIdx.x == 0) {
            const unsigned long long cap = eng.raster_cap;
            const unsigned long long kept = rbase + n <= cap ? n : (rbase >= cap ? 0ull : cap - rbase);
            if (eng.record) {
                ctl->raster_next = rbase + kept;
                ctl->raster_base = rbase + kept;
                ctl->raster_dropped += n - kept;
            }
            ctl->step = s0 + nsteps;
            ctl->raster_done = 0;
        }
    }
}

// Deterministic aggregation.  The order of a step's additions to a ring cell
// is that of the synapse indices j (k_det_step): every event of the step
// stores its weight at ev_w[j] and links itself into its cell's list, and
// after a barrier the event that started a list folds it in ascending j and
// adds the fold to the cell.  The warp that linked a list's first event keeps
// {j, cell, weight} in its own part of shared memory (kDetStarts places), so
// that the fold reads no row again: one load of the list's head, and for a
// list of one event (most of them) nothing else.  A warp with more starts
// than places goes over its rows a second time instead.
// Bound by the same chain of latencies as the rest of k_group, with one
// exchange and one head load more and the third barrier.  Kernel time per grid
// step, against k_drive + k_det_step (whose fold reads the rows and links of all
// events again, between barriers of two blocks an SM): 1k neurons / out-degree
// 50: 6.1 against 10.3 us; 12k / 600: 12.5 against 18.1; 100k / 500: 16.7
// against 22.1; plastic 5k / 200: 8.5 against 22.3, 80k / 800: 15.5 against 28.4.
struct __align__(16) DetStart {
    uint32_t j, cell;
    float w;
    uint32_t pad;  // one 128-bit access
};

// Links one piece of a row (psz synapses, kBatch a lane at a time): all loads
// of a batch before the first exchange, all exchanges before the first of
// their results is used.  Returns the warp's starts (may exceed kDetStarts).
template <int kBatch>
__device__ __forceinline__ uint32_t det_link(const NetDev& np, uint32_t tl, uint32_t tmod, const uint4& spike,
                                             uint64_t beg, uint32_t len, uint32_t piece, uint32_t split, DetStart* starts,
                                             uint32_t n, uint32_t lane, unsigned long long& ev, uint32_t& ovf, Ctl* ctl) {
    const uint32_t D = np.ring_slots, Ns = np.n_storage;
    const uint32_t* __restrict__ tgt_a = np.tgt + beg;
    const uint8_t* __restrict__ d_a = np.dly + beg;
    float* w_a = np.w + beg;
    float* __restrict__ ev_w = np.ev_w + beg;
    uint32_t* __restrict__ ev_next = np.ev_next + beg;
    uint32_t* __restrict__ heads = np.cell_head;
    const bool plastic = np.stdp_on && spike.x < np.n_plastic;
    const int32_t aux0 = (int32_t)spike.z;
    const float mult = !plastic && aux0 > 1 ? (float)aux0 : 1.0f;
    StdpView sv;
    if (plastic) sv = stdp_view(np);
    for (uint32_t off = piece * 32 * kBatch; off < len; off += split * 32 * kBatch) {
        uint32_t cell[kBatch], tgt[kBatch], d[kBatch], old[kBatch];
        float w[kBatch];
#pragma unroll
        for (uint32_t u = 0; u < (uint32_t)kBatch; ++u) {
            const uint32_t x = off + 32 * u + lane;
            tgt[u] = kTgtSentinel;
            if (x < len && NAER_IN_BOUNDS(ctl, beg + x, np.syn_cap, kChkEventList)) {
                tgt[u] = __ldcg(tgt_a + x);
                d[u] = __ldcg(d_a + x);
                w[u] = __ldcg(w_a + x);
            }
        }
#pragma unroll
        for (uint32_t u = 0; u < (uint32_t)kBatch; ++u) {
            const bool on = tgt[u] != kTgtSentinel && ring_ok(np, ring_slot(tmod, d[u], D), tgt[u], ctl);
            cell[u] = on ? ring_slot(tmod, d[u], D) * Ns + tgt[u] : kTgtSentinel;
            if (!on) continue;
            const uint32_t x = off + 32 * u + lane;
            old[u] = atomicExch(heads + cell[u], (uint32_t)(beg + x));
            if (plastic && tgt[u] < np.n_plastic) {
                w[u] = stdp_update(sv, w[u], tgt[u], (int32_t)tl, aux0, __uint_as_float(spike.w), ovf);
                __stcg(w_a + x, w[u]);
            }
            if (mult != 1.0f) w[u] = __fmul_rn(w[u], mult);
            __stcg(ev_w + x, w[u]);
            ++ev;
        }
#pragma unroll
        for (uint32_t u = 0; u < (uint32_t)kBatch; ++u) {
            const bool on = cell[u] != kTgtSentinel;
            const uint32_t x = off + 32 * u + lane;
            if (on) __stcg(ev_next + x, old[u]);
            const bool first = on && old[u] == kNoEvent;
            const uint32_t bal = __ballot_sync(0xFFFFFFFFu, first);
            const uint32_t pos = n + __popc(bal & ((1u << lane) - 1u));
            if (first && pos < kDetStarts) starts[pos] = DetStart{(uint32_t)beg + x, cell[u], w[u], 0u};
            n += __popc(bal);
        }
    }
    return n;
}

// Empties a list and adds its fold to the cell (j: its first event, of weight
// w).  No other thread touches the list or the cell in this phase.
__device__ __forceinline__ void det_add(const NetDev& np, uint32_t cell, uint32_t hd, uint32_t j, float w) {
    __stcg(np.cell_head + cell, kNoEvent);
    red_add_f32(np.ring + cell, hd == j ? w : fold_from_start(np.ev_w, np.ev_next, hd, j, w));
}

// The fold over a warp's starts, kFold a lane with their heads in flight.
__device__ __forceinline__ void det_fold(const NetDev& np, const DetStart* starts, uint32_t n, uint32_t lane) {
    constexpr uint32_t kFold = 4;
    for (uint32_t x0 = lane; x0 < n; x0 += 32 * kFold) {
        uint32_t hd[kFold];
#pragma unroll
        for (uint32_t u = 0; u < kFold; ++u)
            if (x0 + 32 * u < n) hd[u] = __ldcg(np.cell_head + starts[x0 + 32 * u].cell);
#pragma unroll
        for (uint32_t u = 0; u < kFold; ++u)
            if (x0 + 32 * u < n) {
                const DetStart st = starts[x0 + 32 * u];
                det_add(np, st.cell, hd[u], st.j, st.w);
            }
    }
}

// The fold over a piece of a row read again: its events without a next one.
template <int kBatch>
__device__ __forceinline__ void det_refold(const NetDev& np, uint32_t tmod, uint64_t beg, uint32_t len, uint32_t piece,
                                           uint32_t split, uint32_t lane, Ctl* ctl) {
    const uint32_t* __restrict__ tgt_a = np.tgt + beg;
    const uint8_t* __restrict__ d_a = np.dly + beg;
    for (uint32_t off = piece * 32 * kBatch; off < len; off += split * 32 * kBatch) {
        uint32_t cell[kBatch], next[kBatch], hd[kBatch];
        float w[kBatch];
#pragma unroll
        for (uint32_t u = 0; u < (uint32_t)kBatch; ++u) {
            const uint32_t x = off + 32 * u + lane;
            cell[u] = kTgtSentinel;
            if (x >= len || !NAER_IN_BOUNDS(ctl, beg + x, np.syn_cap, kChkEventList)) continue;
            const uint32_t tgt = __ldcg(tgt_a + x), d = __ldcg(d_a + x);
            next[u] = __ldcg(np.ev_next + beg + x);
            w[u] = __ldcg(np.ev_w + beg + x);
            if (tgt != kTgtSentinel && ring_ok(np, ring_slot(tmod, d, np.ring_slots), tgt, ctl))
                cell[u] = ring_slot(tmod, d, np.ring_slots) * np.n_storage + tgt;
        }
#pragma unroll
        for (uint32_t u = 0; u < (uint32_t)kBatch; ++u)
            if (cell[u] != kTgtSentinel && next[u] == kNoEvent) hd[u] = __ldcg(np.cell_head + cell[u]);
#pragma unroll
        for (uint32_t u = 0; u < (uint32_t)kBatch; ++u)
            if (cell[u] != kTgtSentinel && next[u] == kNoEvent)
                det_add(np, cell[u], hd[u], (uint32_t)(beg + off + 32 * u + lane), w[u]);
    }
}

template <bool kGrid, int kPer, bool kPlastic, bool kDet>
__global__ void __launch_bounds__(kGroupThreads, 1)
    k_group(EngineDev eng, unsigned long long s0, uint32_t nsteps) {
    constexpr uint32_t kChunk = 32 * kPer;
    constexpr uint32_t kTile = kPer == 4 ? 2 : 4;      // chunks of a warp whose loads are issued together
    constexpr uint32_t kStepTile = kPer == 4 ? 4 : 8;  // steps of a window whose loads are issued together
    extern __shared__ __align__(16) unsigned char s_dyn[];
    __shared__ GroupShared sh;
    const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5;
    const uint32_t csz = kGrid ? gridDim.x : eng.group_size;  // blocks of the group
    const uint32_t rank = kGrid ? blockIdx.x : blockIdx.x % csz, group = kGrid ? 0u : blockIdx.x / csz;
    const bool several = !kGrid && eng.n_nets > 1;
    const bool drawer = wib >= kGroupSteppers;
    // the grid's drawing warps deliver too once they have drawn, with
    // plasticity: its items are one synapse a lane, each a chain of loads, and
    // more warps keep more of them in flight (100k / 1000, a pass of 1,000 steps
    // with its results read: 12.6 -> 11.8 ms; of 500 steps with static rows, 200k
    // / 1000: 7.23 and 7.32, so theirs stay with the others)
    constexpr bool kDrawersDeliver = kGrid && kPlastic && !kDet;
    const uint32_t nwarps = csz * kGroupSteppers, gw = rank * kGroupSteppers + wib;  // stepping warps
    Ctl* ctl = eng.ctl;
    const uint32_t own_max = eng.group_own;  // neurons of a block, at most
    GroupSpike* s_list = reinterpret_cast<GroupSpike*>(s_dyn);
    DriveWindow* q = reinterpret_cast<DriveWindow*>(s_list + kGroupList) + wib * kGroupQueue;
    float* sV = reinterpret_cast<float*>(s_dyn + kGroupList * sizeof(GroupSpike) +
                                         kGroupWarps * kGroupQueue * sizeof(DriveWindow));
    uint4* s_row = reinterpret_cast<uint4*>(sV + own_max);  // with eng.group_rows
    uint2* s_gc = reinterpret_cast<uint2*>(s_row + (eng.group_rows ? own_max : 0u));
    uint8_t* sR = reinterpret_cast<uint8_t*>(s_gc + own_max / kChunk);
    // deterministic aggregation: the warp's list starts
    DetStart* starts = reinterpret_cast<DetStart*>(sR + own_max) + wib * kDetStarts;
    unsigned long long bar_target = 0;
    unsigned long long ev = 0;
    uint32_t ovf = 0;
    if (s0 == kStepFromCtl) s0 = ctl->step;
    const unsigned long long rbase = ctl->raster_next;
    const bool timer = rank == 0 && threadIdx.x == 0;
    if (threadIdx.x == 0) {
        sh.bcfg = barrier_cfg(ctl);
        sh.ok = 1;
        sh.ev = 0;
        sh.ovf = 0;
        for (int x = 0; x < 4; ++x) sh.ph[x] = 0;
    }
    bool ok = true;
    const uint32_t ni = several ? eng.group_order[group] : 0u;
    static_assert(sizeof(NetDev) % 4 == 0 && sizeof(NetDev) / 4 <= kGroupThreads, "NetDev copied in words");
    if (threadIdx.x < sizeof(NetDev) / 4)
        reinterpret_cast<uint32_t*>(&sh.net)[threadIdx.x] =
            __ldg(reinterpret_cast<const uint32_t*>(eng.nets + ni) + threadIdx.x);
    __syncthreads();
    const NetDev& np = sh.net;
    // the block's spike records: in the grid form all of them, in the cluster
    // form those past kGroupList
    const size_t region = np.q_off + (size_t)rank * np.q_cap;
    const unsigned long long a = s0 > np.start_step ? s0 : np.start_step;
    const unsigned long long b = s0 + nsteps < np.end_step ? s0 + nsteps : np.end_step;
    if (np.active && a < b) {
        if (threadIdx.x < np.pop_count) sh.pop[threadIdx.x] = eng.pops[np.pop_first + threadIdx.x];
        // the network's chunks go round the group's stepping warps:
        // place j * kGroupSteppers + x of a block holds the j-th of its warp x
        const uint32_t places = (np.g_chunks + nwarps - 1) / nwarps * kGroupSteppers;
        const uint32_t own =  // the warp's chunks
            !drawer && gw < np.g_chunks ? (np.g_chunks - gw + nwarps - 1) / nwarps : 0u;
        for (uint32_t at = threadIdx.x; at < places; at += blockDim.x) {
            const uint32_t c = at / kGroupSteppers * nwarps + rank * kGroupSteppers + at % kGroupSteppers;
            uint2 gc = make_uint2(0u, 0u);
            if (c < np.g_chunks) {
                const GroupChunk ch = eng.group_chunks[np.g_first + c];
                gc = make_uint2(ch.first, ch.info);
            }
            s_gc[at] = gc;
        }
        if (threadIdx.x < 2) sh.n_spikes[threadIdx.x] = 0;
        __syncthreads();
        for (uint32_t j = 0; j < own; ++j) {
            const uint32_t place = j * kGroupSteppers + wib;
            const uint2 gc = s_gc[place];
            const uint32_t at = place * kChunk + kPer * lane, i = gc.x + kPer * lane;
            if (kPer * lane >= ((gc.y >> 8) & 0xFFu) || !NAER_IN_BOUNDS(ctl, i + kPer - 1, np.n_storage, kChkState))
                continue;
            if (gc.y & kGcLif) {
                if constexpr (kPer == 4) {
                    *reinterpret_cast<float4*>(sV + at) = *reinterpret_cast<const float4*>(np.v + i);
                    *reinterpret_cast<uint32_t*>(sR + at) = *reinterpret_cast<const uint32_t*>(np.refr + i);
                } else {
                    sV[at] = np.v[i];
                    sR[at] = np.refr[i];
                }
            }
            if (eng.group_rows)
#pragma unroll
                for (uint32_t u = 0; u < (uint32_t)kPer; ++u) s_row[at + u] = row_of(np.row_ptr, np.row_mid, i + u);
        }
        const uint32_t D = np.ring_slots, Ns = np.n_storage, W = np.window;
        const float fx_inv = np.fx_inv;
        // Poisson counts: drawn for the steps before `drawn`, final for
        // those before `known` (queued windows resolved); the first ones
        // by all the block's warps
        constexpr uint32_t kDrawStep = 4 / kPer;  // chunks of one group_draw
        const uint32_t ahead = 2 * W > kGroupAhead ? 2 * W : kGroupAhead;  // at most the drive ring's slots
        unsigned long long drawn = b < a + ahead ? b : a + ahead;
        unsigned long long known = drawn;
        uint32_t qn = 0;
        {
            const uint32_t n = (uint32_t)(drawn - a), tiles = (places + kDrawStep - 1) / kDrawStep;
            for (uint32_t it = wib; it < tiles * n; it += kGroupWarps)
                qn = group_draw<kPer>(np, sh.pop, s_gc, it / n * kDrawStep, places, a + it % n, q, qn, lane, ctl);
            if (qn) group_resolve(sh.pop, np.drive, Ns, np.dt_us, q, qn, lane, ctl);
            qn = 0;
        }
        __syncthreads();
        // local: windows of one step without plasticity whose spikes the
        // block that found them delivers, as soon as its neurons have
        // stepped (ring slot s is read and cleared only in step s, and no
        // spike of step s lands in it): one barrier per step
        const bool local = !kDet && np.local;
        uint32_t par = 0;  // window parity
        uint32_t tmod = (uint32_t)(a - np.start_step) % D;
        for (unsigned long long s = a; s < b; s += W, par ^= 1u) {
            const unsigned long long ta = timer ? globaltimer_ns() : 0ull;
            const uint32_t w = (uint32_t)(b - s < W ? b - s : W);
            const uint32_t tl = (uint32_t)(s - np.start_step);
            uint32_t* bits =
                eng.record ? eng.group_bits + (size_t)(s - s0) * eng.group_words + np.g_word : nullptr;
            // spikes of one step of a chunk as bits for the raster
            auto put_bits = [&](uint32_t hit, uint32_t k, uint32_t chunk) {
                if (!NAER_IN_BOUNDS(ctl, s - s0 + k, nsteps, kChkBits) ||
                    !NAER_IN_BOUNDS(ctl, np.g_word + (chunk + 1) * kPer - 1, eng.group_words, kChkBits))
                    return;
                uint32_t* to = bits + (size_t)k * eng.group_words + chunk * kPer;
                if constexpr (kPer == 4) {
                    uint32_t m[4];
#pragma unroll
                    for (uint32_t u = 0; u < 4; ++u) m[u] = __ballot_sync(0xFFFFFFFFu, (hit >> u) & 1u);
                    if (lane == 0) __stcg(reinterpret_cast<uint4*>(to), make_uint4(m[0], m[1], m[2], m[3]));
                } else {
                    const uint32_t m = __ballot_sync(0xFFFFFFFFu, hit);
                    if (lane == 0) __stcg(to, m);
                }
            };
            // the warp's spikes of all the window's steps of a chunk into
            // the block's list: bit kPer * k + u of hits is the spike of
            // neuron i + u in step k (state of the lane's neurons at `at`)
            auto append = [&](unsigned long long hits, uint32_t i, uint32_t at, bool lif) {
                const uint32_t n = __popcll(hits), x = warp_scan(n, lane);
                uint32_t pos = 0;
                if (lane == 31) pos = atomicAdd(&sh.n_spikes[par], x);
                pos = __shfl_sync(0xFFFFFFFFu, pos, 31) + x - n;
                for (; hits; hits &= hits - 1, ++pos) {
                    const uint32_t bit = __ffsll(hits) - 1, k = bit / kPer, u = bit % kPer;
                    if (!NAER_IN_BOUNDS(ctl, i + u, Ns, kChkState) || !record_ok(np, pos, ctl)) continue;
                    // a POISSON source's multiplicity is its count
                    const uint32_t m = lif ? 0u : __ldcg(np.drive + (size_t)((s + k) % kDriveSlots) * Ns + i + u);
                    const uint4 row = eng.group_rows ? s_row[at + u] : row_of(np.row_ptr, np.row_mid, i + u);
                    if (pos < kGroupList) {
                        s_list[pos] = GroupSpike{i + u, k, (int32_t)m, 0.0f, row};
                    } else {
                        __stcg(reinterpret_cast<int4*>(eng.queue[0] + region + pos),
                               make_int4((int)(i + u), (int)k, (int)m, 0));
                        __stcg(eng.qrow[0] + region + pos, row);
                    }
                }
            };
            // drive counts of a POISSON chunk are its spikes
            auto counts_hit = [](uint32_t dr) {
                uint32_t h = 0;
#pragma unroll
                for (uint32_t u = 0; u < (uint32_t)kPer; ++u) h |= ((dr >> (8 * u)) & 0xFFu ? 1u : 0u) << u;
                return h;
            };
            // the lane's neurons of a chunk of `count`
            auto valid_of = [&](uint32_t count) {
                if constexpr (kPer == 1) return lane < count ? 1u : 0u;
                return count >= 4 * lane + 4 ? 0xFu : count > 4 * lane ? (1u << (count - 4 * lane)) - 1u : 0u;
            };
            auto get_state = [&](uint32_t at, Vals<kPer>& v, uint32_t& r) {
                if constexpr (kPer == 4) {
                    const float4 x = *reinterpret_cast<const float4*>(sV + at);
                    v.v[0] = x.x, v.v[1] = x.y, v.v[2] = x.z, v.v[3] = x.w;
                    r = *reinterpret_cast<const uint32_t*>(sR + at);
                } else {
                    v.v[0] = sV[at];
                    r = sR[at];
                }
            };
            auto put_state = [&](uint32_t at, const Vals<kPer>& v, uint32_t r) {
                if constexpr (kPer == 4) {
                    *reinterpret_cast<float4*>(sV + at) = make_float4(v.v[0], v.v[1], v.v[2], v.v[3]);
                    *reinterpret_cast<uint32_t*>(sR + at) = r;
                } else {
                    sV[at] = v.v[0];
                    sR[at] = (uint8_t)r;
                }
            };
            // ---- 1. LIF of the window's steps
            if (drawer) {
                // counts that the next window reads and that are still queued
                if (known < b && known < s + w + W) {
                    if (qn) group_resolve(sh.pop, np.drive, Ns, np.dt_us, q, qn, lane, ctl);
                    qn = 0;
                    known = drawn;
                }
            } else if (w == 1) {
                // a tile of the warp's chunks: every load of the tile is
                // issued before the first is used
                float* ring = np.ring + (size_t)tmod * Ns + kPer * lane;
                const uint8_t* drive = np.drive + (size_t)(s % kDriveSlots) * Ns + kPer * lane;
                for (uint32_t j0 = 0; j0 < own; j0 += kTile) {
                    Vals<kPer> in[kTile];
                    uint32_t dr[kTile];
                    uint2 gc[kTile];
#pragma unroll
                    for (uint32_t u = 0; u < kTile; ++u) {
                        if (u && j0 + u >= own) break;
                        gc[u] = s_gc[(j0 + u) * kGroupSteppers + wib];
                        const bool on = kPer * lane < ((gc[u].y >> 8) & 0xFFu) &&
                                        ring_ok(np, tmod, gc[u].x + kPer * lane + kPer - 1, ctl);
                        dr[u] = on && (gc[u].y & kGcDrawn) ? ld_bytes<kPer>(drive + gc[u].x) : 0u;
                        if (on && (gc[u].y & kGcLif)) {
                            in[u] = ld_vals<kPer>(ring + gc[u].x);
                        } else {
#pragma unroll
                            for (int k = 0; k < kPer; ++k) in[u].v[k] = 0.0f;
                        }
                    }
#pragma unroll
                    for (uint32_t u = 0; u < kTile; ++u) {
                        if (u && j0 + u >= own) break;
                        const uint32_t at = ((j0 + u) * kGroupSteppers + wib) * kChunk + kPer * lane;
                        const uint32_t count = (gc[u].y >> 8) & 0xFFu;
                        const bool lif = gc[u].y & kGcLif;
                        uint32_t hit = 0;
                        if (lif) {
                            if (kPer * lane < count && ring_ok(np, tmod, gc[u].x + kPer * lane + kPer - 1, ctl)) {
                                clear_vals<kPer>(ring + gc[u].x);
                                const PopDev& p = sh.pop[gc[u].y & 0xFFu];
                                const GroupLif prm{p.prop, p.v_th, p.v_reset, p.drive_w, fx_inv, p.t_ref_steps};
                                Vals<kPer> v;
                                uint32_t r;
                                get_state(at, v, r);
                                hit = group_lif<kPer>(v, r, prm, in[u], dr[u]);
                                put_state(at, v, r);
                            }
                        } else {
                            hit = counts_hit(dr[u]);
                        }
                        hit &= valid_of(count);
                        if (bits) put_bits(hit, 0, gw + (j0 + u) * nwarps);
                        if (__any_sync(0xFFFFFFFFu, hit != 0)) append(hit, gc[u].x + kPer * lane, at, lif);
                    }
                }
            } else {
                // a tile of the window's steps of one chunk
                for (uint32_t j = 0; j < own; ++j) {
                    const uint2 gc = s_gc[j * kGroupSteppers + wib];
                    const uint32_t i = gc.x + kPer * lane, at = (j * kGroupSteppers + wib) * kChunk + kPer * lane;
                    const uint32_t valid = valid_of((gc.y >> 8) & 0xFFu);
                    const bool on = valid != 0 && NAER_IN_BOUNDS(ctl, i + kPer - 1, Ns, kChkState);
                    const bool lif = gc.y & kGcLif, drawn_pop = gc.y & kGcDrawn;
                    const PopDev& p = sh.pop[gc.y & 0xFFu];
                    const GroupLif prm{p.prop, p.v_th, p.v_reset, p.drive_w, fx_inv, p.t_ref_steps};
                    Vals<kPer> v;
#pragma unroll
                    for (int k = 0; k < kPer; ++k) v.v[k] = 0.0f;
                    uint32_t r = 0;
                    unsigned long long hits = 0;
                    if (lif && on) get_state(at, v, r);
                    for (uint32_t k0 = 0; k0 < w; k0 += kStepTile) {
                        Vals<kPer> in[kStepTile];
                        uint32_t dr[kStepTile];
#pragma unroll
                        for (uint32_t u = 0; u < kStepTile; ++u) {
                            const bool step_on =
                                on && k0 + u < w && ring_ok(np, ring_slot(tmod, k0 + u, D), i + kPer - 1, ctl);
                            dr[u] = step_on && drawn_pop
                                        ? ld_bytes<kPer>(np.drive + (size_t)((s + k0 + u) % kDriveSlots) * Ns + i)
                                        : 0u;
                            if (step_on && lif) {
                                in[u] = ld_vals<kPer>(np.ring + (size_t)ring_slot(tmod, k0 + u, D) * Ns + i);
                            } else {
#pragma unroll
                                for (int k = 0; k < kPer; ++k) in[u].v[k] = 0.0f;
                            }
                        }
                        if (lif && on) {
#pragma unroll
                            for (uint32_t u = 0; u < kStepTile; ++u)
                                if (k0 + u < w && ring_ok(np, ring_slot(tmod, k0 + u, D), i + kPer - 1, ctl))
                                    clear_vals<kPer>(np.ring + (size_t)ring_slot(tmod, k0 + u, D) * Ns + i);
                        }
#pragma unroll
                        for (uint32_t u = 0; u < kStepTile; ++u) {
                            if (k0 + u >= w) break;
                            const uint32_t hit =
                                (lif ? group_lif<kPer>(v, r, prm, in[u], dr[u]) : counts_hit(dr[u])) & valid;
                            hits |= (unsigned long long)hit << (kPer * (k0 + u));
                            if (bits) put_bits(hit, k0 + u, gw + j * nwarps);
                        }
                    }
                    if (__any_sync(0xFFFFFFFFu, hits != 0)) append(hits, i, at, lif);
                    if (lif && on) put_state(at, v, r);
                }
            }
            if (!drawer) steppers_sync();
            const unsigned long long ta2 = timer ? globaltimer_ns() : 0ull;
            // ---- 2. the block's spikes, one thread each: with plasticity
            // the post-spike update; in the grid form the records
            const uint32_t mine = sh.n_spikes[par];
            if (!local) {
                if (kGrid && threadIdx.x == 0) __stcg(eng.group_cnt + rank, mine);
                if (!drawer && (kGrid || (kPlastic && np.stdp_on))) {
                    for (uint32_t e = threadIdx.x; e < mine && record_ok(np, e, ctl); e += kGroupStepThreads) {
                        int4 head;
                        if (e < kGroupList) head = *reinterpret_cast<const int4*>(s_list + e);
                        else head = __ldcg(reinterpret_cast<const int4*>(eng.queue[0] + region + e));
                        if (kPlastic && np.stdp_on && (uint32_t)head.x < np.n_plastic) {
                            float aux1;
                            stdp_post_spike(&sh.net, (uint32_t)head.x, (int32_t)tl + head.y, head.z, aux1);
                            head.w = __float_as_int(aux1);
                        }
                        if (kGrid || e >= kGroupList) {
                            __stcg(reinterpret_cast<int4*>(eng.queue[0] + region + e), head);
                            if (kGrid && e < kGroupList) __stcg(eng.qrow[0] + region + e, s_list[e].row);
                        } else {
                            *reinterpret_cast<int4*>(s_list + e) = head;
                        }
                    }
                }
                if (!group_barrier<kGrid>(ctl, bar_target, sh)) {
                    ok = false;
                    break;
                }
            }
            const unsigned long long tb = timer ? globaltimer_ns() : 0ull;
            if (threadIdx.x == 0) sh.n_spikes[par ^ 1u] = 0;  // the next window's
            // ---- 3. spikes of the group's blocks and, per block, of the
            // blocks before it: of a cluster every warp for itself
            // (lane = block), of the grid once per block
            uint32_t Q = mine, below = 0;
            if (!local) {
                if (!kGrid) {
                    const uint32_t x = lane < csz ? cluster_ld(cluster_map(&sh.n_spikes[par], lane)) : 0u;
                    const uint32_t y = warp_scan(x, lane);
                    below = y - x;
                    Q = __shfl_sync(0xFFFFFFFFu, y, 31);
                } else {
                    if (wib == 0) {
                        uint32_t run = 0, x[kGroupMaxBlocks / 32];
#pragma unroll
                        for (uint32_t r = 0; r < kGroupMaxBlocks / 32; ++r)
                            x[r] = r * 32 + lane < csz ? __ldcg(eng.group_cnt + r * 32 + lane) : 0u;
#pragma unroll
                        for (uint32_t r = 0; r < kGroupMaxBlocks / 32; ++r) {
                            const uint32_t y = warp_scan(x[r], lane);
                            sh.first[r * 32 + lane + 1] = run + y;
                            run += __shfl_sync(0xFFFFFFFFu, y, 31);
                        }
                        if (lane == 0) sh.first[0] = 0;
                    }
                    __syncthreads();
                    Q = sh.first[csz];
                }
            }
            // ---- 4. every row of the window's spikes
            uint32_t workers = 0, split = 1, items = 0, n_starts = 0;
            bool wide = false;
            // spike e of the window: the block that holds it, and its place there
            auto fetch = [&](uint32_t e, uint4& head, uint4& row) {
                uint32_t reg = rank, x = e;
                if (!local) {
                    if (!kGrid) {
                        reg = __popc(__ballot_sync(0xFFFFFFFFu, lane < csz && below <= e)) - 1u;
                        x = e - __shfl_sync(0xFFFFFFFFu, below, reg);
                    } else {
                        reg = locate(sh.first, csz, e);
                        x = e - sh.first[reg];
                    }
                }
                if (!record_ok(np, x, ctl)) {
                    head = row = make_uint4(kTgtSentinel, 0u, 0u, 0u);  // no source: skipped by the caller
                } else if (local && x < kGroupList) {
                    head = *reinterpret_cast<const uint4*>(s_list + x);
                    row = s_list[x].row;
                } else if (!kGrid && x < kGroupList) {
                    const uint32_t at = cluster_map(s_list + x, reg);
                    head = cluster_ld4(at);
                    row = cluster_ld4(at + 16);
                } else {
                    const size_t at = np.q_off + (size_t)reg * np.q_cap + x;
                    head = __ldcg(reinterpret_cast<const uint4*>(eng.queue[0] + at));
                    row = __ldcg(eng.qrow[0] + at);
                }
            };
            if (drawer) {
                // meanwhile: counts of the steps `ahead` of the next window
                const unsigned long long goal = s + w + ahead < b ? s + w + ahead : b;
                for (unsigned long long d = drawn; d < goal; ++d)
                    for (uint32_t at = (wib - kGroupSteppers) * kDrawStep; at < places; at += kGroupDrawers * kDrawStep)
                        qn = group_draw<kPer>(np, sh.pop, s_gc, at, places, d, q, qn, lane, ctl);
                if (drawn < goal) drawn = goal;
            }
            if (Q && (!drawer || (kDrawersDeliver && !local))) {
                // row pieces: enough items for the workers, no more than
                // the longest row has; one synapse a lane where that
                // still leaves every worker at most one
                workers = local ? kGroupSteppers : kDrawersDeliver ? csz * kGroupWarps : nwarps;
                const uint32_t first = local ? wib : drawer ? nwarps + rank * kGroupDrawers + (wib - kGroupSteppers) : gw;
                const uint32_t narrow = (np.max_row + kPlasticPiece - 1) / kPlasticPiece;
                const bool stdp = kPlastic && np.stdp_on;
                wide = (kDet || !stdp) && Q * narrow > workers;
                const uint32_t pieces = wide ? (np.max_row + 127) / 128 : narrow;
                const uint32_t want = (2u * workers + Q - 1) / Q;
                split = want < pieces ? want : (pieces ? pieces : 1u);
                items = Q * split;  // at most Q + 2 * workers
                BinTable bt{};
                for (uint32_t it = first; it < items; it += workers) {
                    const uint32_t e = it / split, piece = it - e * split;
                    uint4 head, row;
                    fetch(e, head, row);
                    if (!NAER_IN_BOUNDS(ctl, head.x, Ns, kChkQueue)) continue;
                    const uint64_t beg = ((uint64_t)row.y << 32) | row.x;
                    if constexpr (kDet) {
                        n_starts = wide ? det_link<4>(np, tl, tmod, head, beg, row.w, piece, split, starts, n_starts, lane, ev, ovf, ctl)
                                        : det_link<1>(np, tl, tmod, head, beg, row.w, piece, split, starts, n_starts, lane, ev, ovf, ctl);
                    } else if (stdp && head.x < np.n_plastic) {
                        SpikeRec rec;
                        rec.net = 0;
                        rec.src = head.x;
                        rec.aux0 = (int32_t)head.z;
                        rec.aux1 = __uint_as_float(head.w);
                        deliver_span(&sh.net, tl, rec, beg, beg + row.w, piece, split, kPlasticPiece, lane, ev, ovf, ctl, bt);
                    } else {
                        const float mult = (int32_t)head.z > 1 ? (float)(int32_t)head.z : 1.0f;
                        const uint32_t slot = ring_slot(tmod, head.y, D);
                        if (wide) group_row<true>(np, slot, mult, beg, row.w, piece, split, lane, ev, ctl);
                        else group_row<false>(np, slot, mult, beg, row.w, piece, split, lane, ev, ctl);
                    }
                }
            }
            if (kDet && Q) {  // every event is linked: fold
                ok = group_barrier<kGrid>(ctl, bar_target, sh);
                if (!ok) break;
                if (!drawer && n_starts <= kDetStarts) {
                    det_fold(np, starts, n_starts, lane);
                } else if (!drawer) {
                    for (uint32_t it = gw; it < items; it += workers) {
                        const uint32_t e = it / split;
                        uint4 head, row;
                        fetch(e, head, row);
                        if (!NAER_IN_BOUNDS(ctl, head.x, Ns, kChkQueue)) continue;
                        const uint64_t beg = ((uint64_t)row.y << 32) | row.x;
                        if (wide) det_refold<4>(np, tmod, beg, row.w, it - e * split, split, lane, ctl);
                        else det_refold<1>(np, tmod, beg, row.w, it - e * split, split, lane, ctl);
                    }
                }
            }
            const unsigned long long tb2 = timer ? globaltimer_ns() : 0ull;
            if (!group_barrier<kGrid>(ctl, bar_target, sh)) {
                ok = false;
                break;
            }
            tmod = (tmod + w) % D;
            if (timer) {
                const unsigned long long tc = globaltimer_ns();
                sh.ph[0] += ta2 - ta;
                sh.ph[1] += tb - ta2;
                sh.ph[2] += tb2 - tb;
                sh.ph[3] += tc - tb2;
            }
        }
        for (uint32_t j = 0; j < own; ++j) {
            const uint32_t place = j * kGroupSteppers + wib;
            const uint2 gc = s_gc[place];
            const uint32_t at = place * kChunk + kPer * lane, i = gc.x + kPer * lane;
            if (kPer * lane < ((gc.y >> 8) & 0xFFu) && (gc.y & kGcLif) &&
                NAER_IN_BOUNDS(ctl, i + kPer - 1, np.n_storage, kChkState)) {
                if constexpr (kPer == 4) {
                    *reinterpret_cast<float4*>(np.v + i) = *reinterpret_cast<const float4*>(sV + at);
                    *reinterpret_cast<uint32_t*>(np.refr + i) = *reinterpret_cast<const uint32_t*>(sR + at);
                } else {
                    np.v[i] = sV[at];
                    np.refr[i] = sR[at];
                }
            }
        }
        // spikes per (step, segment); the last window's barrier made every
        // block's bits visible
        if (eng.record && ok) {
            const uint32_t segs = np.seg_n, items = (uint32_t)(b - a) * segs;
            for (uint32_t it = rank * kGroupWarps + wib; it < items; it += csz * kGroupWarps)
                raster_count(eng, (uint32_t)(a - s0) + it / segs, np.seg_first + it % segs, lane);
        }
    }
    if (ok && !several) {
        if (eng.record) {
            ok = group_barrier<kGrid>(ctl, bar_target, sh);  // the counts
            const uint32_t items = nsteps * eng.group_seg_n;
            for (uint32_t it = rank * kGroupWarps + wib; ok && it < items; it += csz * kGroupWarps)
                raster_write(eng, s0, it / eng.group_seg_n, it % eng.group_seg_n, rbase, lane);
        }
        if (ok) ok = group_barrier<kGrid>(ctl, bar_target, sh);  // counts read before they are cleared
        if (ok && rank == 0) raster_end(eng, s0, nsteps, rbase);
    }
    finish_counters(eng, ev, ovf, lane, &sh.ev, &sh.ovf, eng.group_part);
    if (timer) {  // phase times: mean over the networks
        unsigned long long ph[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) ph[x] = several ? sh.ph[x] / eng.n_nets : sh.ph[x];
        atomicAdd(&ctl->prof_phase_ns[0], ph[0]);
        atomicAdd(&ctl->prof_phase_ns[1], ph[1]);
        atomicAdd(&ctl->prof_phase_ns[2], ph[2]);
        atomicAdd(&ctl->prof_phase_ns[4], ph[3]);
        atomicAdd(&ctl->prof_lif_ns, ph[0] + ph[1]);
        atomicAdd(&ctl->prof_scatter_ns, ph[2] + ph[3]);
        if (blockIdx.x == 0 && eng.group_part == 0) ctl->prof_steps += nsteps;
    }
}

// Raster of a launch over several networks (of one network, its group writes
// the raster itself): warp by warp over (step, segment); the last block to
// finish ends the launch.
__global__ void __launch_bounds__(kRasterThreads) k_raster(EngineDev eng, unsigned long long s0, uint32_t nsteps) {
    __shared__ bool s_last;
    Ctl* ctl = eng.ctl;
    if (s0 == kStepFromCtl) s0 = ctl->step;
    const unsigned long long rbase = ctl->raster_next;
    const uint32_t items = eng.record ? nsteps * eng.group_seg_n : 0u;
    for (uint32_t it = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; it < items; it += (gridDim.x * blockDim.x) >> 5)
        raster_write(eng, s0, it / eng.group_seg_n, it % eng.group_seg_n, rbase, threadIdx.x & 31u);
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(&ctl->raster_done, 1u) + 1 == gridDim.x;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    raster_end(eng, s0, nsteps, rbase);
}


// (deterministic aggregation in a cluster: one network, always one neuron a lane)
#define NAER_GROUP(grid, per, det)                                                            \
    template __global__ void k_group<grid, per, true, det>(EngineDev, unsigned long long, uint32_t); \
    template __global__ void k_group<grid, per, false, det>(EngineDev, unsigned long long, uint32_t);
NAER_GROUP(true, 1, false)
NAER_GROUP(true, 4, false)
NAER_GROUP(false, 1, false)
NAER_GROUP(false, 4, false)
NAER_GROUP(true, 1, true)
NAER_GROUP(true, 4, true)
NAER_GROUP(false, 1, true)
#undef NAER_GROUP

size_t group_smem_bytes(uint32_t own_neurons, uint32_t per_lane, bool rows, bool det) {
    return kGroupList * sizeof(GroupSpike) + kGroupWarps * kGroupQueue * sizeof(DriveWindow) +
           (size_t)own_neurons * (5 + (rows ? 16 : 0)) + own_neurons / (32 * per_lane) * sizeof(uint2) +
           (det ? kGroupSteppers * kDetStarts * sizeof(DetStart) : 0);
}

}  // namespace naer
