// Where networks step: the lines and step-time models by which the engine
// chooses between the forms of k_group (group_kernel.cuh) and the grid kernels
// (k_step, k_det_step, k_run with k_drive).  Host code; the forms give the same
// results.
#pragma once
#include <stdint.h>

#include <algorithm>
#include <cmath>

#include "engine_types.cuh"

namespace naer {

constexpr uint32_t kGroupSingle = 16;  // blocks of a single network's cluster

// Expected activity of a network in a grid step.
struct Activity {
    double neurons = 0, drawn = 0;  // drawn: with Poisson counts
    double spikes = 0, events = 0;
};

struct GroupNeed {
    uint32_t window = 1;    // steps of a window
    bool stdp = false;
    bool det = false;       // deterministic aggregation
    uint32_t chunks = 0;    // of 32 neurons
    uint64_t synapses = 0;
    Activity act;
};

struct GroupForm {
    bool group = false;     // k_group (else the grid kernels)
    bool cluster = false;   // in one cluster of kGroupSingle blocks (else on the grid)
    bool local = false;     // block-local delivery
};

// Block-local delivery (one barrier a step) up to 500k synapses a block: a
// block's share of a step's spikes varies, which costs more than the barrier
// saves once it is bound by its reductions (50k / 400: 6.6 us a step against 8.4
// with the exchange; 200k / 1000: 11.8 against 11.0).
inline bool block_local(uint32_t window, bool stdp, uint64_t synapses, uint32_t blocks) {
    return window == 1 && !stdp && synapses <= 500000ull * blocks;
}

// Form of a single network.  The lines were measured on B200, us per grid step,
// atomic aggregation (n neurons / out-degree); "k_step" includes its k_drive.
//
//   cluster of 16 blocks, 1 neuron a lane: at most one chunk a warp (two with
//     windows of one step, up to 8M synapses).  LIF networks of 5k / 100: 3.5
//     (grid 4.2, k_step 9.5); 12k / 100: 4.4 (4.6, 9.5); 12k / 1000: 6.7 (6.0);
//     plastic 12k / 300: 7.3 (8.4, 10.5); Brunel 5k: 1.44 (1.55, 9.2), 10k: 2.2
//     (1.6, 9.4)
//   grid, 1 neuron a lane up to two chunks a warp, else 4: 20k / 500: 5.1 (4 a
//     lane 6.7, k_step 10.5); 100k / 1000: 9.2 (9.3, 12.0); 400k / 500: 13.9
//     (12.4, 14.5); Brunel 40k: 3.4 (3.9, 10.4)
//   k_step from 500k neurons (700k / 300: 17.0, grid 17.0; 1M / 1000: 27.0,
//     27.4), 250k with plasticity (300k / 300: 14.1, 14.1), unless windows are
//     longer than one step; k_det_step from 250k, 600k with plasticity (600k /
//     100: 30.9, k_det_step 35.3)
//
// Within these lines the events of a step decide: a block delivers about a
// thousand in a microsecond, so the few blocks of a cluster, or those that hold a
// small network's neurons, fall behind the grid when a step has many; and
// k_step, which delivers while it waits at its barriers, gains on k_group's
// exchange.  The form of the lines above stays until k_step is expected to be
// faster, and then the faster of k_step and the exchange on the grid is taken.
// Events a step: us in a cluster with block-local delivery / in a cluster with the
// exchange / on the grid with the exchange / k_step:
//     2k / 1000:   7.6k 5.0 / 5.3 / 6.6 / 9.1, 17k 6.7 / 5.8 / 7.1 / 9.8
//     2k / 4000:   8k 6.2 / 5.1 / 6.5 / 9.0, 30k 10.6 / 6.5 / 7.3 / 10.3, 142k 27.6 /
//                  12.6 / 8.2 / 10.9
//     6.1k / 2000: 12k 6.0 / 5.7 / 7.1 / 9.9, 46k 8.7 / 7.9 / 7.9 / 10.7, 102k 13.2 /
//                  11.8 / 8.2 / 10.9
//   on the grid block-local / with the exchange / k_step:
//     50k / 2000:  99k 8.1 / 8.2 / 10.9, 372k 12.8 / 10.6 / 11.9, 834k 17.8 / 15.2 / 13.8
//     200k / 4000: 784k 21.8 / 15.7 / 14.1, 2,967k 42.5 / 30.8 / 26.2
//     450k / 300:  1,123k 18.0 / 20.5 / 22.7
//   with plasticity, cluster / grid / k_step: 6.1k / 1000: 3.1k 6.3 / 7.9 / 9.7, 13k
//     9.3 / 9.1 / 11.2, 36k 14.9 / 9.9 / 12.3; 12k / 1000: 67k 27.5 / 11.1 / 13.2
//   windows of several steps: 15 steps, 6k / 1000: 50k 3.5 / 2.0 / 9.8, 6k / 4000:
//     459k 15.9 / 4.8 / 13.3; 2 steps, 6k / 4000: 418k 21.3 / 8.2 / 10.5
//   deterministic aggregation, cluster / grid / k_det_step: 6k / 1000: 6.0k 9.6 /
//     10.7 / 17.8, 23k 16.6 / 12.7 / 22.7; 12k / 4000: 180k 117 / 26.0 / 34.7; grid /
//     k_det_step: 100k / 1000: 98k 19.1 / 22.5, 372k 32.7 / 27.6; 160k / 1000: 156k
//     19.8 / 23.1, 591k 51.5 / 33.9; 240k / 100: 200k 26.5 / 20.6; 240k / 1000: 235k
//     25.9 / 23.8 (k_det_step has a third more warps to wait for the events'
//     exchanges); with plasticity 240k / 1000: 489k 47.3 / 49.4, 1,372k 127 / 110
inline GroupForm single_form(const GroupNeed& n, uint32_t sms) {
    constexpr uint32_t step_warps = kGroupStepThreads / 32, cluster_warps = kGroupSingle * step_warps;
    const Activity& a = n.act;
    GroupForm f;
    f.group = true;
    f.cluster = n.chunks <= cluster_warps ||
                (n.window == 1 && n.chunks <= 2 * cluster_warps && n.synapses <= 8000000ull);
    if (n.window == 1 && !n.stdp && !n.det) {
        f.local = block_local(1, false, n.synapses, f.cluster ? kGroupSingle : sms);
        // us that the events add to a step's common time, and the barriers of each form
        auto local_us = [&](uint32_t blocks, double spread, double per_us) {  // the busiest block's
            const double m = a.spikes / std::max(1u, std::min(blocks, (n.chunks + step_warps - 1) / step_warps));
            return (m + spread * std::sqrt(m)) * ((double)n.synapses / a.neurons) / per_us;
        };
        const double exchange = 2.6 + a.events / 130e3;
        const double own = f.cluster ? (n.chunks > cluster_warps ? 0.7 : 0.0) +
                                           (f.local ? local_us(kGroupSingle, 2.2, 1600.0) : 1.4 + a.events / 15e3)
                           : f.local ? 0.5 + local_us(sms, 2.7, 1300.0)
                                     : exchange;
        const double step = 4.5 + std::max(0.0, a.neurons - 200e3) / 100e3 + a.spikes / 2000.0 + a.events / 210e3;
        if (own > step) {
            f.group = exchange <= step;
            f.cluster = f.local = false;
        }
        return f;
    }
    f.cluster = f.cluster && a.events <= (n.det ? 16e3 : n.stdp ? 20e3 : 60e3);
    if (n.det && !f.cluster)
        f.group = n.stdp ? a.events <= 1e6
                         : a.neurons <= 200e3 ? a.events <= 250e3 && a.spikes <= 800.0
                                              : a.events <= 130e3 && a.spikes <= 300.0;
    return f;
}

// Step time (us) of one of several networks in a cluster of c blocks, `per`
// neurons a lane, `rounds` chunks a warp: the LIF's rounds; a chain of 1.3 (2.7
// more with the exchange) or 2.5 (plastic) once a window; and the events at the
// rate a block delivers them or the draws, whichever is longer.  Fitted to 88
// batches (2 to 600 networks of 200 to 50k neurons, out-degrees 30 to 3,000, with
// and without plasticity, even and uneven): 12 % rms.
inline double cluster_us(const GroupNeed& n, uint32_t c, uint32_t per, double rounds) {
    const double lif = per == 1 ? 0.12 + 0.56 * rounds : 0.11 + 1.16 * rounds;
    const double chain = n.stdp ? 2.5 : block_local(n.window, false, n.synapses, c) ? 1.27 : 4.0;
    const double load = n.act.events / (c * (n.stdp ? 178.0 : 1120.0));
    return lif + chain / n.window + std::max(1.6 / n.window + load, n.act.drawn / c / 870.0);
}

// Step time (us) of the grid kernels for the same networks together: a chain of
// 9.6, the neurons, the events at the rate of the reductions (where a network is
// plastic, at that of its post rows' loads), and what of the rings does not stay
// in L2; 7 % rms over the same batches.  A launch with its draws costs 30 us, of
// 64 steps there, of a few in the served form.
inline double grid_us(double neurons, double events, double ring_mb, bool plastic, uint32_t launch_steps) {
    return 9.6 + neurons / 116e3 + events / (plastic ? 24.8e3 : 173e3) +
           41e-6 * events * std::max(0.0, 1.0 - 80.0 / std::max(ring_mb, 1.0)) +
           30.0 * std::max(0.0, 1.0 / launch_steps - 1.0 / 64.0);
}

// Several networks step in clusters.  Measured, clusters / grid (models): 48
// uneven networks of up to 50k neurons 28.7 / 35.1 (27.3 / 30.3), 100 of them 56.9 /
// 78.5 (54.1 / 81.2), 64 of 2k / 200 5.6 / 11.4 (6.0 / 11.0), plastic 8 of 5k / 500
// 8.0 / 11.6 (7.3 / 10.9), but 16 of 50k / 500 30.0 / 19.7 (28.9 / 21.0), 32 of 10k /
// 2000 45.5 / 26.0 (45.5 / 26.1), 100 of 20k with windows of 4 steps 50.2 / 30.3
// (40.2 / 29.1), plastic 16 of 20k / 1000 34.7 / 23.2 (36.4 / 25.1).  With 1.1 the
// choice over the 88 batches costs least, 0.5 % on average.
inline bool clusters_pay(double clusters, double grid) { return clusters <= 1.1 * grid; }

}  // namespace naer
