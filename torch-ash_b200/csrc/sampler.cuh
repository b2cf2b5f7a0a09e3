// Ray marching over the hashed block structure, shared by the sampler kernels and the fused ray
// renderer, so that both place every step identically.  Semantics of ash/src/sampler.cu:7-215;
// lengths in cell units; position = fma(t, d, o) per component in float32, block =
// floor(position * (float)(1.0 / grid2cell)).
#pragma once
#include "hashmap.cuh"

namespace ashb {

__device__ __forceinline__ bool block_active(const Table16& t, const float* p, float cell2grid) {
    const int bx = (int)floorf(p[0] * cell2grid);
    const int by = (int)floorf(p[1] * cell2grid);
    const int bz = (int)floorf(p[2] * cell2grid);
    return lookup(t, bx, by, bz, 0) >= 0;
}

__device__ __forceinline__ void ray_at(const float* o, const float* d, float t, float* p) {
    p[0] = __fmaf_rn(t, d[0], o[0]);
    p[1] = __fmaf_rn(t, d[1], o[1]);
    p[2] = __fmaf_rn(t, d[2], o[2]);
}

// A table lookup split in two so that several can be in flight: probe_begin reads the key's home
// slot (when `wanted`), probe_finish walks on from there and says whether the block is active.
struct ProbeStart {
    int k[3];
    uint32_t slot;
    Entry e;
};

__device__ __forceinline__ ProbeStart probe_begin(const Table16& t, const float* p, float cell2grid, bool wanted) {
    ProbeStart ps;
    ps.k[0] = (int)floorf(p[0] * cell2grid);
    ps.k[1] = (int)floorf(p[1] * cell2grid);
    ps.k[2] = (int)floorf(p[2] * cell2grid);
    ps.slot = hash_key(ps.k[0], ps.k[1], ps.k[2], 0) & t.mask;
    ps.e = wanted ? t.read_const(ps.slot) : Entry{0, 0, 0, 0, kEmpty};
    return ps;
}

__device__ __forceinline__ bool probe_finish(const Table16& t, const ProbeStart& ps) {
    Entry e = ps.e;
    uint32_t s = ps.slot;
    for (uint32_t probe = 0; probe <= t.mask; ++probe) {
        if (e.val == kEmpty) return false;
        if (e.val >= 0 && key_match(e, ps.k[0], ps.k[1], ps.k[2], 0)) return true;
        s = (s + 1) & t.mask;
        e = t.read_const(s);
    }
    return false;
}

// First / last occupied stretch of a ray inside the box (ash/src/sampler.cu:7-71): marches in
// half-block steps from t_min; near = -1 when no occupied block is met.
__device__ __forceinline__ void march_near_far(const Table16& t, const float* o, const float* d, const float* lo,
                                               const float* hi, float t_min, float t_max, float grid2cell,
                                               float& near, float& far) {
    const float cell2grid = (float)(1.0 / (double)grid2cell);
    const float step = (float)((double)grid2cell * 0.5);
    near = -1.f;
    far = t_max;
    float tt = t_min;
    // step > 0 is checked by the host, so the march ends after (t_max - t_min) / step rounds.
    // The positions of consecutive steps do not depend on what the probes find, so four steps are
    // taken per round: their first table reads are issued together, then the steps are replayed
    // in order (same sequence of `tt`, same results as one step at a time).
#ifndef ASHB_NEAR_FAR_AHEAD
#define ASHB_NEAR_FAR_AHEAD 4
#endif
    constexpr int kAhead = ASHB_NEAR_FAR_AHEAD;
    auto in_box = [&](const float* p) {
        return p[0] >= lo[0] && p[0] <= hi[0] && p[1] >= lo[1] && p[1] <= hi[1] && p[2] >= lo[2] && p[2] <= hi[2];
    };
    // Along the ray a coordinate only rises or only falls, rounded as it is, so steps between two that are in the box are in
    // it: a round asks for its last step alone, and only where that one is out for each.
    float first[3];
    ray_at(o, d, t_min, first);
    const bool entered = in_box(first);
    bool ended = false;
    while (!ended && tt < t_max) {
        float ts[kAhead], p[kAhead][3];
        bool inside[kAhead];
        ProbeStart ps[kAhead];
        float t_k = tt;
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
            ts[k] = t_k;
            ray_at(o, d, t_k, p[k]);
            t_k += step;
        }
        const bool all = entered && ts[kAhead - 1] < t_max && in_box(p[kAhead - 1]);
#pragma unroll
        for (int k = 0; k < kAhead; ++k) inside[k] = all;
        if (!all) {
#pragma unroll
            for (int k = 0; k < kAhead; ++k) inside[k] = ts[k] < t_max && in_box(p[k]);
        }
        int values = kEmpty;   // all bits set
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
            ps[k] = probe_begin(t, p[k], cell2grid, inside[k]);
            values &= ps[k].e.val;
        }
        tt = t_k;
        if (all && values == kEmpty) continue;   // four home slots that hold nothing
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
            if (ended) break;
            if (!(ts[k] < t_max) || !inside[k]) {
                ended = true;
                break;
            }
            if (probe_finish(t, ps[k])) {
                near = near < 0.f ? ts[k] : fmaxf(near - step, t_min);
                far = fminf(ts[k] + step, t_max);
            }
        }
    }
}

// Step of the interval sampler inside occupied blocks (ash/src/sampler.cu:151): max(0.7, float) is
// a double max whose result is stored as float.
__device__ __forceinline__ float sample_cell_step(float ray_near, float ray_far, int64_t max_samples) {
    return (float)fmax(0.7, (double)((ray_far - ray_near) / (float)max_samples));
}

// The interval sampler's march (ash/src/sampler.cu:123-215) with four probes in flight: from
// `near` to `far`, a cell step inside occupied blocks -- each such step is an interval, reported to
// emit(t_start, t_end) -- and a block step outside.  The next positions are guessed from the kind of
// step taken last, their probes are issued together, and the steps are replayed in order; the
// first step whose outcome differs from the guess ends the round, because the positions after it
// were guessed with the wrong stride.  `tt` goes through exactly the values of the
// one-probe-at-a-time march.
template <class Emit>
__device__ __forceinline__ void march_intervals(const Table16& t, const float* o, const float* d, float ray_near,
                                                float ray_far, float cell_step, float grid_step, float cell2grid,
                                                Emit&& emit) {
    constexpr int kAhead = 4;
    float tt = ray_near, seg_near = ray_near;
    bool guess_active = true;
    while (tt < ray_far) {
        const float stride_guess = guess_active ? cell_step : grid_step;
        float ts[kAhead];
        ProbeStart ps[kAhead];
        float t_k = tt;
#pragma unroll
        for (int a = 0; a < kAhead; ++a) {
            ts[a] = t_k;
            float p[3];
            ray_at(o, d, t_k, p);
            ps[a] = probe_begin(t, p, cell2grid, t_k < ray_far);
            t_k += stride_guess;
        }
#pragma unroll
        for (int a = 0; a < kAhead; ++a) {
            if (!(ts[a] < ray_far)) {
                tt = ts[a];
                break;
            }
            const bool active = probe_finish(t, ps[a]);
            if (active) {
                tt = ts[a] + cell_step;
                emit(seg_near, tt);
                seg_near = tt;
            } else {
                tt = ts[a] + grid_step;
            }
            if (active != guess_active) {
                guess_active = active;
                break;
            }
        }
    }
}

// ---- the same two marches by kGroup lanes of a warp for one ray ----------------------------------
// With a few thousand rays the chip is nearly empty and a march is a chain of round trips, so the lanes of a
// group take consecutive steps side by side and agree on the outcome by votes.  Every lane walks `tt`
// through the same sums in the same order as the marches above, so all positions are theirs.  8192 rays of
// ~160 steps: 82.7 -> 27.6 us.
// All lanes of the warp call these together; `live` lanes have a ray, the same in a group.
constexpr int kGroup = 8;

// Tables of up to this many slots are probed through their occupancy bits in the group marches: a ray mostly meets
// blocks that were never allocated, and 64 KB of bits stay in L1 where the 16-byte slots are an L2 round
// trip away.  A larger map's bits are themselves in L2: one more round trip per hit, nothing saved per
// miss.  The one-thread marches of many rays do not ask them: neighbouring rays find each other's
// slots in L1, and what those marches are short of is instructions (352 us without, 377 with, for 307,200 rays).
constexpr uint32_t kMarchFilterSlots = 1u << 19;

__device__ __forceinline__ bool may_hold(const Table16& t, uint32_t slot) {
    if (t.occupied == nullptr || t.mask >= kMarchFilterSlots) return true;
    return (__ldg(t.occupied + (slot >> 5)) >> (slot & 31)) & 1u;
}

// probe_begin in two: whether the slot is worth reading, and the read.
__device__ __forceinline__ bool probe_key(const Table16& t, const float* p, float cell2grid, bool wanted, ProbeStart& ps) {
    ps = probe_begin(t, p, cell2grid, false);
    return wanted && may_hold(t, ps.slot);
}

__device__ __forceinline__ void probe_read(const Table16& t, bool wanted, ProbeStart& ps) {
    if (wanted) ps.e = t.read_const(ps.slot);
}

// Bits of the calling lane's group out of a warp-wide vote.
__device__ __forceinline__ unsigned group_vote(bool v) {
    return (__ballot_sync(0xffffffffu, v) >> (threadIdx.x & 31 & ~(kGroup - 1))) & ((1u << kGroup) - 1);
}

// The position `n` strides on, by the marches' own sums.
__device__ __forceinline__ float nth_position(float t, float stride, int n) {
    for (int i = 0; i < n; ++i) t += stride;
    return t;
}

__device__ __forceinline__ void group_near_far(const Table16& t, bool live, const float* o, const float* d,
                                               const float* lo, const float* hi, float t_min, float t_max,
                                               float grid2cell, float& near, float& far) {
    constexpr int kAhead = 4;   // steps of a lane per round: 32 of the ray
    const float cell2grid = (float)(1.0 / (double)grid2cell);
    const float step = (float)((double)grid2cell * 0.5);
    const int lane = threadIdx.x & (kGroup - 1);
    near = -1.f;
    far = t_max;
    float tt = t_min;
    bool going = live && tt < t_max;
    while (__any_sync(0xffffffffu, going)) {
        float ts[kAhead];
        bool inside[kAhead], read[kAhead];
        ProbeStart ps[kAhead];
        float t_k = tt;
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
#pragma unroll
            for (int j = 0; j < kGroup; ++j) {
                if (j == lane) ts[k] = t_k;
                t_k += step;
            }
            float p[3];
            ray_at(o, d, ts[k], p);
            inside[k] = going && ts[k] < t_max && p[0] >= lo[0] && p[0] <= hi[0] && p[1] >= lo[1] && p[1] <= hi[1] &&
                        p[2] >= lo[2] && p[2] <= hi[2];
            read[k] = probe_key(t, p, cell2grid, inside[k], ps[k]);
        }
#pragma unroll
        for (int k = 0; k < kAhead; ++k) probe_read(t, read[k], ps[k]);
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
            const unsigned in = group_vote(inside[k]);
            const unsigned before_exit = in & ~(in + 1);             // the steps up to the first outside
            const unsigned hits = group_vote(probe_finish(t, ps[k])) & (going ? before_exit : 0u);
            const float last = __shfl_sync(0xffffffffu, ts[k], hits ? 31 - __clz(hits) : 0, kGroup);
            for (unsigned rest = hits; rest; rest &= rest - 1) {
                if (near < 0.f) near = nth_position(tt, step, k * kGroup + __ffs(rest) - 1);
                else near = fmaxf(near - step, t_min);
            }
            if (hits) far = fminf(last + step, t_max);
            if (in != (1u << kGroup) - 1) going = false;
        }
        tt = t_k;
        going = going && tt < t_max;
    }
}

// emit(k, t_start, t_end) is called once per interval by one lane of the group, k counting the ray's
// intervals; returns their number.
template <class Emit>
__device__ __forceinline__ int group_intervals(const Table16& t, bool live, const float* o, const float* d, float ray_near,
                                               float ray_far, float cell_step, float grid_step, float cell2grid,
                                               Emit&& emit) {
    const int lane = threadIdx.x & (kGroup - 1);
    float tt = ray_near, seg_near = ray_near;
    int count = 0;
    bool guess_active = true, going = live && tt < ray_far;
    while (__any_sync(0xffffffffu, going)) {
        const float stride = guess_active ? cell_step : grid_step;
        float ts = tt, t_k = tt;
#pragma unroll
        for (int j = 0; j < kGroup; ++j) {
            if (j == lane) ts = t_k;
            t_k += stride;
        }
        float p[3];
        ray_at(o, d, ts, p);
        const bool in = going && ts < ray_far;
        ProbeStart ps;
        probe_read(t, probe_key(t, p, cell2grid, in, ps), ps);
        const unsigned ins = group_vote(in), act = group_vote(probe_finish(t, ps));
        if (!going) continue;
        // the steps that went as guessed, and whether one after them did not
        const int n_in = __popc(ins);
        const int run = min(n_in, __ffs(~(guess_active ? act : ~act & ((1u << kGroup) - 1))) - 1);
        const bool surprise = run < n_in;
        const float t_run = nth_position(tt, stride, run);
        if (guess_active) {
            if (lane < run) emit(count + lane, lane == 0 ? seg_near : ts, ts + cell_step);
            count += run;
            if (run > 0) seg_near = t_run;
            tt = surprise ? t_run + grid_step : t_run;
        } else if (surprise) {
            tt = t_run + cell_step;
            if (lane == 0) emit(count, seg_near, tt);
            ++count;
            seg_near = tt;
        } else {
            tt = t_run;
        }
        if (surprise) guess_active = !guess_active;
        going = tt < ray_far;
    }
    return count;
}

}  // namespace ashb
