// mutate_ruleset() (fate_stream.h) by one warp: the same draws in the same order,
// bit-identical results.
//
// A pass makes 174 uniform draws, each compared with a rate, and only where one
// falls below it more draws and a change.  What bounds the pass on one lane is
// latency: a branch, a load and a serial generator step per draw, and 2 us of
// double-precision logarithm and division per change.  Here every lane steps
// the generator (it has no parallel form), lane i keeps the i-th of 32 draws, and
// the warp looks for the first draw below its rate in one ballot.  A change
// takes its draws from the same window; what it adds is worked out afterwards,
// one change per lane.
#pragma once

#include "fate_stream.h"

namespace marl {
namespace fate {

constexpr uint32_t kMutTransport = 24, kMutReaction = 56, kMutEffector = 152, kMutFate = 168, kMutHgt = 172,
                   kMutMeta = 173, kMutDraws = 174;

// A division's stream read by a whole warp; every call by all lanes, every
// result the same on all of them.
struct WarpStream {
    Stream s;
    uint64_t win;  // this lane's draw of the window
    uint32_t cur;  // the window's first draw that is not taken yet

    __device__ __forceinline__ explicit WarpStream(uint64_t key) : s(key), win(0), cur(32) {}
    __device__ __forceinline__ void refill() {
        const int lane = threadIdx.x & 31;
        uint64_t mine = 0;
#pragma unroll 4
        for (int i = 0; i < 32; ++i) {
            mine = i == lane ? s.s[1] : mine;
            s.u64();
        }
        win = Stream::output(mine);
        cur = 0;
    }
    __device__ __forceinline__ uint64_t u64() {
        if (cur == 32) refill();
        return __shfl_sync(0xFFFFFFFFu, win, (int)cur++);
    }
    __device__ __forceinline__ void skip(uint32_t k) {
        for (uint32_t i = 0; i < k; ++i) u64();
    }
    __device__ __forceinline__ uint32_t range(uint32_t lo, uint32_t hi) { return draw_range(*this, lo, hi); }
};

// Draws that redraw a species instead of changing a number.
__device__ __forceinline__ bool mut_structural(uint32_t p) {
    if (p < kMutTransport || p >= kMutEffector) return false;
    return p < kMutReaction ? ((p - kMutTransport) & 3u) >= 2u : (p - kMutReaction) % 6u >= 3u;
}

// The number that draw p changes.
__device__ __forceinline__ float* mut_target(marl_ruleset& rs, uint32_t p) {
    if (p < kMutTransport) {
        marl_receptor_params& r = rs.receptors[p / 3u];
        return p % 3u == 0 ? &r.k_half : (p % 3u == 1 ? &r.n_hill : &r.gain);
    }
    if (p < kMutReaction) {
        marl_transport_params& t = rs.transport[(p - kMutTransport) >> 2];
        return (p - kMutTransport) & 3u ? &t.secrete_rate : &t.uptake_rate;
    }
    if (p < kMutEffector) {
        marl_reaction& x = rs.reactions[(p - kMutReaction) / 6u];
        const uint32_t w = (p - kMutReaction) % 6u;
        return w == 0 ? &x.k_m : (w == 1 ? &x.v_max : &x.k_cat);
    }
    if (p < kMutFate) {
        marl_effector_params& e = rs.effectors[(p - kMutEffector) >> 1];
        return (p - kMutEffector) & 1u ? &e.rate : &e.threshold;
    }
    switch (p) {
        case kMutFate: return &rs.fate.division_energy;
        case kMutFate + 1: return &rs.fate.death_energy;
        case kMutFate + 2: return &rs.fate.quiescence_energy;
        case kMutFate + 3: return &rs.fate.division_prep_ticks;
        case kMutHgt: return &rs.hgt_propensity;
        default: return &rs.mutation_rate;
    }
}

// `rs` in shared memory, written before a __syncwarp(); complete after the next.
__device__ __forceinline__ void mutate_ruleset_warp(marl_ruleset& rs, WarpStream& rng, const marl_sim_params& sim) {
    const uint32_t lane = threadIdx.x & 31u;
    const float rate = rs.mutation_rate;
    const float sd = sim.mutation_stddev;
    const float structural = rate * sim.structural_mutation_rate_mult;
    const unsigned donors = __ballot_sync(
        0xFFFFFFFFu, lane < MARL_R_MAX && fabsf(rs.reactions[lane & 15u].v_max) > sim.active_reaction_threshold);
    const uint32_t n_donors = (uint32_t)__popc(donors);

    // Up to 32 changes that wait for their value, one per lane.
    uint32_t waiting = 0, my_p = 0;
    double my_u = 0.0, my_s2 = 0.0;
    auto apply = [&]() {
        if (lane < waiting) {
            const float d = my_s2 > 0.0 ? polar_normal(my_u, my_s2, sd) : 0.0f;
            float& v = *mut_target(rs, my_p);
            if (my_p == kMutMeta)
                v = clamp_rs(v + d * sim.meta_mutation_rate, sim.meta_mutation_clamp_low, sim.meta_mutation_clamp_high);
            else
                v = fmaxf(v + d, 0.0f);
        }
        waiting = 0;
    };

    for (uint32_t pos = 0; pos < kMutDraws;) {
        if (rng.cur == 32) rng.refill();
        const uint32_t p = pos + lane - rng.cur;
        const float below = p == kMutMeta ? sim.meta_mutation_rate : (mut_structural(p) ? structural : rate);
        const unsigned hits = __ballot_sync(0xFFFFFFFFu, lane >= rng.cur && p < kMutDraws &&
                                                             (float)(rng.win >> 40) * 0x1.0p-24f < below);
        if (hits == 0) {
            const uint32_t seen = min(32u - rng.cur, kMutDraws - pos);
            pos += seen;
            rng.cur += seen;
            continue;
        }
        const uint32_t at = (uint32_t)__ffs((int)hits) - 1u, hit = pos + at - rng.cur;
        rng.cur = at + 1;
        pos = hit + 1;
        if (!mut_structural(hit)) {
            double u = 0.0, s2 = 0.0;
            for (int tries = 0; tries < 64; ++tries) {
                u = (double)(rng.u64() >> 11) * 0x1.0p-52 - 1.0;
                const double v = (double)(rng.u64() >> 11) * 0x1.0p-52 - 1.0;
                const double uu = u * u;
                const double vv = v * v;
                s2 = uu + vv;
                if (s2 < 1.0 && s2 > 0.0) break;
                s2 = 0.0;
            }
            if (lane == waiting) my_p = hit, my_u = u, my_s2 = s2;
            if (++waiting == 32) apply();
        } else if (hit < kMutReaction) {
            marl_transport_params& t = rs.transport[(hit - kMutTransport) >> 2];
            const bool ext = ((hit - kMutTransport) & 3u) == 2u;
            const uint8_t species = (uint8_t)rng.range(0, ext ? MARL_S_EXT : MARL_M_INT);
            if (lane == 0) (ext ? t.ext_species : t.int_species) = species;
        } else {
            const uint32_t i = (hit - kMutReaction) / 6u, slot = (hit - kMutReaction) % 6u - 3u;
            const uint32_t pick = rng.range(0, n_donors > 0 ? n_donors : 1u);
            marl_reaction& x = rs.reactions[i];
            uint8_t* dst = slot == 0 ? &x.substrate : (slot == 1 ? &x.product : &x.catalyst);
            if (pick < n_donors) {
                const uint32_t donor = __fns(donors, 0, (int)pick + 1);  // the pick-th set bit
                const marl_reaction& d = rs.reactions[donor];
                // Lane 0 alone touches the species, in draw order.
                if (lane == 0) *dst = slot == 0 ? d.substrate : (slot == 1 ? d.product : d.catalyst);
            } else {
                const uint8_t species = (uint8_t)rng.range(0, MARL_M_INT);
                if (lane == 0) *dst = species;
            }
        }
    }
    apply();
    __syncwarp();
    if (lane < MARL_S_RECEPTORS) {
        float& h = rs.receptors[lane].n_hill;
        h = clamp_rs(h, sim.hill_exponent_clamp_low, sim.hill_exponent_clamp_high);
    }
    if (lane == 8) rs.fate.division_prep_ticks = fmaxf(rs.fate.division_prep_ticks, 1.0f);
}

}  // namespace fate
}  // namespace marl
