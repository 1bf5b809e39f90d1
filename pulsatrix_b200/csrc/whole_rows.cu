// Sampling from the whole distribution: no top-k, no top-p, no min-p (src/generation.cpp:123-156 with the filters
// off -- the penalty, the EOS ban and the temperature may be on).  Every token can be drawn, so there is no short
// list of candidates; what the draw needs is the mass of every run of columns, then the columns of one run.
//
//   1. weigh_segments_kernel: a warp takes a segment of 512 columns into registers, finds its two maxima (raw and processed), sums exp() of
//      both in double precision and reports 32 bytes.  The warps of a CTA share a bitmap of the history, nothing else.
//   2. draw_token_kernel, one CTA per row: the segments' masses brought to the row's maximum, their running sum against
//      u times the whole (the inverse-CDF walk of :140-152 in steps of a segment), then the logits of the one segment that
//      holds the crossing, column by column.  (Drawing in the CTA that finishes a row's last segment saves the launch,
//      but costs a fence and an atomic per CTA and runs under the arithmetic of other rows: 5 to 10 % slower from a few rows on.)
//
// Sums are in double precision in a fixed order (the same input gives the same bits); they differ from the
// reference's sequential sums by rounding only, and a draw closer than that to an edge shows in draw_margin.
//
// Bound: 4 bytes per logit from HBM, and two double-precision exponentials per logit (one when the processed row is
// the raw one).  The double-precision pipe (64 lanes per SM) and the issue slots beside it are the longer of the two,
// which is why the exponential is the table one (psx_exp.cuh) and the temperature a product.  A segment is a warp's: 512
// columns keep 16 logits per lane in registers, so that the maximum is known before the first exponential and nothing is
// rescaled, and one row of 50 K columns still gives 98 warps to spread over the SMs.
// 100 rows x 50,021, T = 0.9: 865 us per call when one CTA per row did this in the survivor stage, 20.5 now (17 us for the
// first kernel in two rounds of CTAs, double-precision pipe 43 % and issue slots 53 % busy); 330 rows x 50,257: 32 us.
#include "whole_rows.cuh"

#include <algorithm>

#include "../../include/psx_b200.h"
#include "psx_exp.cuh"

namespace psx {

namespace {

constexpr int kThreads = 128;   // eight CTAs to an SM (64 registers): the loads of some run under the arithmetic of others
constexpr int kWarps = kThreads / 32;
constexpr int kSegmentCols = kSegmentVecs * 4;
constexpr int kVecs = kSegmentVecs / 32;  // float4 per lane
constexpr int kMostPerWarp = 4;           // segments a warp takes one after the other

// The row as aligned float4 vectors: component c of vector v is column 4 v + c - misalign.
struct RowWindow {
    const float4* base;
    int misalign, vectors;
};
__device__ __forceinline__ RowWindow row_window(const WholeRowParams& p, int64_t row) {
    const float* x = p.logits + row * p.row_stride;
    RowWindow w;
    w.misalign = (int)((reinterpret_cast<uintptr_t>(x) >> 2) & 3);
    w.base = reinterpret_cast<const float4*>(x - w.misalign);
    w.vectors = (int)((w.misalign + p.vocab + 3) >> 2);
    return w;
}

// Marks, in a bitmap of `slots` bits that starts at column `first`, the columns that `ids` names (:62: ids outside the
// vocabulary are ignored -- their bits stand for no column of the row).  By the whole block; four ids per thread are
// asked for together, one trip to memory for 512 of them.
__device__ __forceinline__ void mark_columns(const int64_t* ids, int64_t begin, int64_t end, int64_t first, int slots, int64_t vocab,
                                             uint32_t* bits) {
    for (int64_t i = begin + threadIdx.x; i < end; i += 4 * kThreads) {
        int64_t id[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) id[q] = i + q * kThreads < end ? ids[i + q * kThreads] : -1;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint64_t at = (uint64_t)(id[q] - first);
            if (at < (uint64_t)slots && (uint64_t)id[q] < (uint64_t)vocab) atomicOr(&bits[at >> 5], 1u << (at & 31));
        }
    }
}

// The processed logit (:59-79).
__device__ __forceinline__ float processed(float l, bool flagged, bool banned, const WholeRowParams& p) {
    float y = l;
    if (flagged) y = penalize(l, p.penalty);
    if (banned) y = -INFINITY;
    return temper(y, p.apply_temperature != 0, p.temperature);
}

// Running sums over the block in thread order: up to this thread, up to and with it, over all.  A thread's `before` is
// the thread before it's `upto` bit for bit.
struct RunningSum {
    double before, upto, total;
};
__device__ __forceinline__ RunningSum block_running_sum(double v, double* scratch) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double up = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if (lane >= o) v += up;
    }
    double earlier = __shfl_up_sync(0xFFFFFFFFu, v, 1);
    if (lane == 0) earlier = 0.0;
    if (lane == 31) scratch[warp] = v;
    __syncthreads();
    RunningSum r;
    double base = 0.0;
    r.total = 0.0;
#pragma unroll
    for (int i = 0; i < kWarps; ++i) {
        if (i == warp) base = r.total;
        r.total += scratch[i];
    }
    r.before = base + earlier;
    r.upto = base + v;
    return r;
}

// The last thread of the block whose value is positive.
__device__ __forceinline__ int block_last_positive(double v, uint32_t* scratch) {
    const uint32_t votes = __ballot_sync(0xFFFFFFFFu, v > 0.0);
    if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = votes;
    __syncthreads();
    int last = -1;
#pragma unroll
    for (int i = 0; i < kWarps; ++i) {
        if (scratch[i] != 0) last = 32 * i + 31 - __clz(scratch[i]);
    }
    return last;
}

__global__ void __launch_bounds__(kThreads) draw_token_kernel(const __grid_constant__ WholeRowParams p) {
    __shared__ double s_mass[kWarps], s_z[kWarps], s_own[kWarps], s_before;
    __shared__ int s_hit, s_alive;
    __shared__ float s_max[2][kWarps];
    __shared__ uint32_t s_votes[2][kWarps], s_flag[kSegmentCols / 32], s_ban[kSegmentCols / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t row = blockIdx.x;
    grid_dependency_wait();
    grid_dependents_may_launch();
    const SegmentStats* stats = p.stats + row * p.segments;
    // thread t takes a run of segments, so that threads and segments stand in the same order
    const int per = (p.segments + kThreads - 1) / kThreads;
    const int begin = min(tid * per, p.segments), end = min(begin + per, p.segments);
    SegmentStats mine;  // (usually the only one of the thread)
    mine.raw_sum = mine.mass = 0.0;
    mine.raw_max = mine.y_max = -INFINITY;
    mine.alive = mine.nonfinite = 0;
    if (begin < end) mine = stats[begin];
    // (asked for now, needed below)
    const double u = p.uniforms[row];
    int64_t h_begin = 0, h_end = 0;
    if (p.history_ids != nullptr) { h_begin = p.history_offsets[row]; h_end = p.history_offsets[row + 1]; }
    if (tid == 0) s_alive = 0;
    if (tid < kSegmentCols / 32) s_flag[tid] = s_ban[tid] = 0u;
    float raw_max = mine.raw_max, y_max = mine.y_max;
    uint32_t bad = mine.nonfinite;
    for (int s = begin + 1; s < end; ++s) {
        const SegmentStats other = stats[s];
        raw_max = fmaxf(raw_max, other.raw_max);
        y_max = fmaxf(y_max, other.y_max);
        bad |= other.nonfinite;
    }
    raw_max = warp_max(raw_max);
    y_max = warp_max(y_max);
    if (lane == 0) { s_max[0][warp] = raw_max; s_max[1][warp] = y_max; }
    const bool failed = __syncthreads_or((int)bad) != 0;
#pragma unroll
    for (int i = 0; i < kWarps; ++i) { raw_max = fmaxf(raw_max, s_max[0][i]); y_max = fmaxf(y_max, s_max[1][i]); }
    if (failed || !(y_max > -INFINITY)) {
        if (tid == 0) {
            p.row_status[row] = failed ? PSX_ROW_NON_FINITE : PSX_ROW_ALL_REMOVED;  // :128-132, :136-138
            p.tokens[row] = -1;
            p.log_probs[row] = 0.0f;
            if (p.diag) p.diag[row] = psx_row_diag{(int)p.vocab, 0, INFINITY, INFINITY};
        }
        return;
    }
    auto share = [&](double sum, float top, float row_top) { return sum > 0.0 ? sum * exp_below(top, row_top) : 0.0; };
    double mass = 0.0, z = 0.0;
    uint32_t alive = 0;
    for (int s = begin; s < end; ++s) {
        if (s > begin) mine = stats[s];
        mass += share(mine.mass, mine.y_max, y_max);
        z += share(mine.raw_sum, mine.raw_max, raw_max);
        alive += mine.alive;
    }
    z = warp_sum(z);
    if (lane == 0) s_z[warp] = z;
    const RunningSum run = block_running_sum(mass, s_mass);
    if (!(y_max < INFINITY)) {
        // A quotient overflowed: every probability of the reference is NaN then, and its walk (:140-152) ends at the last column.
        if (p.diag) {
            alive = __reduce_add_sync(0xFFFFFFFFu, alive);
            if (lane == 0) atomicAdd(&s_alive, (int)alive);
            __syncthreads();
        }
        if (tid == 0) {
            double z_total = s_z[0];
            for (int i = 1; i < kWarps; ++i) z_total += s_z[i];
            p.row_status[row] = PSX_ROW_OK;
            p.tokens[row] = p.vocab - 1;
            p.log_probs[row] = (float)log(exp((double)p.logits[row * p.row_stride + p.vocab - 1] - (double)raw_max) / z_total);
            if (p.diag) p.diag[row] = psx_row_diag{(int)p.vocab, s_alive, NAN, INFINITY};
        }
        return;
    }
    // (The maximum's own mass is 1, so the total is positive and some thread holds every target from 0 on; a uniform below
    // 0 takes the first token that has mass, one that is not below 1 the last.)
    const double total = run.total, target = u < 0.0 ? 0.0 : u * total;
    // ---- the segment that holds the crossing: the running sum rises above the target there (:140-152); if rounding
    // leaves none, the last that holds mass ----------------------------------------------------------------------------
    bool holds = run.before <= target && target < run.upto;
    if (!(target < total)) holds = tid == block_last_positive(mass, s_votes[0]);
    if (holds) {
        double at = run.before, before = at;
        int found = begin;
        for (int s = begin; s < end; ++s) {
            if (end - begin > 1) mine = stats[s];
            const double here = end - begin > 1 ? share(mine.mass, mine.y_max, y_max) : mass;
            if (here > 0.0) { found = s; before = at; }
            at += here;
            if (here > 0.0 && at > target) break;
        }
        s_hit = found;
        s_before = before;
    }
    __syncthreads();
    // ---- its columns, in order: thread t has vector t of the segment ------------------------------------------------------
    const int segment = s_hit;
    const RowWindow w = row_window(p, row);
    const int64_t first_col = (int64_t)segment * kSegmentCols - w.misalign;
    static_assert(kSegmentVecs == kThreads, "one vector per thread");
    float l[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
    if (segment * kSegmentVecs + tid < w.vectors) {
        const float4 d = w.base[segment * kSegmentVecs + tid];
        l[0] = d.x; l[1] = d.y; l[2] = d.z; l[3] = d.w;
    }
    if (p.history_ids != nullptr) mark_columns(p.history_ids, h_begin, h_end, first_col, kSegmentCols, p.vocab, s_flag);
    mark_columns(p.banned_ids, 0, p.num_banned, first_col, kSegmentCols, p.vocab, s_ban);
    if (p.diag) {
        alive = __reduce_add_sync(0xFFFFFFFFu, alive);
        if (lane == 0) atomicAdd(&s_alive, (int)alive);
    }
    __syncthreads();
    const uint32_t flag4 = s_flag[tid >> 3] >> ((tid & 7) * 4), ban4 = s_ban[tid >> 3] >> ((tid & 7) * 4);
    double e[4], own = 0.0;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const bool here = (uint64_t)(first_col + 4 * tid + c) < (uint64_t)p.vocab;
        e[c] = here ? exp_below(processed(l[c], (flag4 >> c) & 1u, (ban4 >> c) & 1u, p), y_max) : 0.0;
        own += e[c];
    }
    const RunningSum cols = block_running_sum(own, s_own);
    // the target within the segment; its columns' sum may fall short of it by the rounding of the segment's
    const double rest = target - s_before;
    holds = cols.before <= rest && rest < cols.upto;
    if (!(rest < cols.total)) holds = tid == block_last_positive(own, s_votes[1]);
    if (holds) {
        double at = cols.before, before = at, upto = at;
        int chosen = -1;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (e[c] > 0.0 && !(chosen >= 0 && upto > rest)) {
                before = at;
                upto = at + e[c];
                chosen = c;
            }
            at += e[c];
        }
        double z_total = s_z[0];
#pragma unroll
        for (int i = 1; i < kWarps; ++i) z_total += s_z[i];
        const float x = chosen == 0 ? l[0] : chosen == 1 ? l[1] : chosen == 2 ? l[2] : l[3];
        p.row_status[row] = PSX_ROW_OK;
        p.tokens[row] = first_col + 4 * tid + chosen;
        // the unprocessed log-softmax (:133,156)
        p.log_probs[row] = (float)log(exp((double)x - (double)raw_max) / z_total);
        if (p.diag) {
            const double lo = (s_before + before) / total, hi = (s_before + upto) / total;
            p.diag[row] = psx_row_diag{(int)p.vocab, s_alive, lo <= 0.0 ? fabs(u - hi) : fmin(fabs(u - lo), fabs(u - hi)), INFINITY};
        }
    }
}

// x / T as the float divide rounds it (:78), from the reciprocal in double precision: the product is off by 2^-52 of
// the quotient at most, and the quotient of two floats is never closer than 2^-49 of itself to a point halfway between two
// floats (that point times T is an integer of at most 49 bits in units that x is a whole number of, and never x itself),
// so rounding the product to 24 bits -- Dekker's splitting with 2^29 + 1, two additions and a product -- gives the same.
// (Quotients below 2^-126 keep more bits than a float has: no exponential notices.)
__device__ __forceinline__ double tempered(double x, double reciprocal) {
    const double q = __dmul_rn(x, reciprocal), c = __dmul_rn(q, 536870913.0);  // (never contracted)
    return __dsub_rn(c, __dsub_rn(c, q));
}

// kProcessed: penalty, ban or temperature make the processed row another than the raw one.  kFlags: a penalty or a ban.
template <bool kProcessed, bool kFlags>
__global__ void __launch_bounds__(kThreads, 8) weigh_segments_kernel(const __grid_constant__ WholeRowParams p) {
    __shared__ uint32_t s_flag[kMostPerWarp * kWarps * kSegmentCols / 32], s_ban[kMostPerWarp * kWarps * kSegmentCols / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t row = (int64_t)blockIdx.z * 65535 + blockIdx.y;
    // (see ScanParams::wait_before_writes: the last CTA of the grid keeps the kernel from finishing early)
    const bool ends_the_grid = p.inputs_ready && blockIdx.x == gridDim.x - 1 && blockIdx.y == gridDim.y - 1 && blockIdx.z == gridDim.z - 1;
    grid_dependents_may_launch();
    if (!p.inputs_ready) grid_dependency_wait();
    if (row >= p.rows) {
        if (ends_the_grid) grid_dependency_wait();
        return;
    }
    const RowWindow w = row_window(p, row);
    const int per_warp = p.segments_per_warp, first_segment = blockIdx.x * kWarps * per_warp;
    float4 d[kVecs];
    auto load = [&](int segment) {
#pragma unroll
        for (int k = 0; k < kVecs; ++k) {
            const int v = segment * kSegmentVecs + k * 32 + lane;
            d[k] = v < w.vectors ? w.base[v] : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
        }
    };
    load(first_segment + warp);  // (lands under the bitmap)
    const int64_t first_col = (int64_t)first_segment * kSegmentCols - w.misalign;
    if (kFlags) {
        const int slots = per_warp * kWarps * kSegmentCols;
        for (int i = threadIdx.x; i < slots / 32; i += kThreads) s_flag[i] = s_ban[i] = 0u;
        __syncthreads();
        if (p.history_ids != nullptr) {
            mark_columns(p.history_ids, p.history_offsets[row], p.history_offsets[row + 1], first_col, slots, p.vocab, s_flag);
        }
        mark_columns(p.banned_ids, 0, p.num_banned, first_col, slots, p.vocab, s_ban);
        __syncthreads();
    }
    const double power = exp_power_of_lane();
    const double reciprocal = p.apply_temperature ? 1.0 / (double)p.temperature : 1.0;
#pragma unroll 1
    for (int turn = 0; turn < per_warp; ++turn) {
        const int local = turn * kWarps + warp, segment = first_segment + local;
        if (segment >= p.segments) break;
        if (turn > 0) load(segment);
        const int lane_col = (segment * kSegmentVecs + lane) * 4 - w.misalign;  // the column of d[0].x; d[k] lies 128 k further
        float l[kVecs * 4];
        uint32_t marked = 0, banned = 0;  // bit 4 k + c: component c of d[k]
#pragma unroll
        for (int k = 0; k < kVecs; ++k) {
            l[4 * k] = d[k].x; l[4 * k + 1] = d[k].y; l[4 * k + 2] = d[k].z; l[4 * k + 3] = d[k].w;
            if (kFlags) {
                const int v = local * kSegmentVecs + k * 32 + lane, shift = (v & 7) * 4;
                banned |= ((s_ban[v >> 3] >> shift) & 15u) << (4 * k);
                marked |= ((s_flag[v >> 3] >> shift) & 15u) << (4 * k);
            }
        }
        marked |= banned;
        // The first and the last vector of a row may reach past it.
        uint32_t here = 0xFFFFu;
        const bool edge = segment == 0 || segment * kSegmentVecs + kSegmentVecs >= w.vectors;
        if (edge) {
#pragma unroll
            for (int i = 0; i < kVecs * 4; ++i) {
                const int col = lane_col + (i >> 2) * 128 + (i & 3);
                if (!((uint32_t)col < (uint32_t)p.vocab)) {
                    here &= ~(1u << i);
                    l[i] = -FLT_MAX;  // (finite; never the maximum)
                }
            }
        }
        bool finite = true;
        float raw_max = -INFINITY, raw_min = INFINITY, clear_max = -INFINITY;  // clear: neither penalised nor banned
#pragma unroll
        for (int i = 0; i < kVecs * 4; i += 2) {
            finite = finite && fabsf(l[i]) < INFINITY && fabsf(l[i + 1]) < INFINITY;
            raw_max = fmax3(raw_max, l[i], l[i + 1]);
            if (kFlags) clear_max = fmax3(clear_max, ((marked >> i) & 1u) ? -FLT_MAX : l[i], ((marked >> i) & 2u) ? -FLT_MAX : l[i + 1]);
        }
        raw_max = warp_max(raw_max);
        if (kFlags) clear_max = warp_max(clear_max);
        if (!__any_sync(0xFFFFFFFFu, here != 0)) raw_max = -INFINITY;  // (past the end of the row)
        // What is not there weighs next to nothing: exp(-690), in the raw sum exp(-690 T) if T < 1, in the other one exp(-690 / T) if T > 1.
        // 511 slots of exp(-60) are 5e-24; where it could be more (very low or high temperatures, maxima so large that 690
        // rounds away), and in a segment that is not there at all, the sums leave the slots out one by one.
        bool absent_weighs = false;
        if (edge) {
            const float nothing = __fmaf_rn(-690.0f, fminf(1.0f, p.apply_temperature ? p.temperature : 1.0f), raw_max), gap = raw_max - nothing;
            // (with flags the other sum leaves them out anyway)
            absent_weighs = !(gap >= 60.0f && (kFlags || !p.apply_temperature || gap >= 60.0f * p.temperature));
#pragma unroll
            for (int i = 0; i < kVecs * 4; ++i) l[i] = ((here >> i) & 1u) ? l[i] : nothing;
        }
#pragma unroll
        for (int i = 0; i < kVecs * 4; i += 2) raw_min = fmin3(raw_min, l[i], l[i + 1]);
        raw_min = -warp_max(-raw_min);
        if (kFlags && !__any_sync(0xFFFFFFFFu, (here & ~marked) != 0)) clear_max = -INFINITY;
        // the processed value of a marked logit, which is read again from the row (a lane usually has none)
        auto marked_value = [&](int i) {
            const int col = lane_col + (i >> 2) * 128 + (i & 3);
            return processed(p.logits[row * p.row_stride + col], true, (banned >> i) & 1u, p);
        };
        float y_max = raw_max;
        if (kProcessed) y_max = temper(kFlags ? clear_max : raw_max, p.apply_temperature != 0, p.temperature);
        if (kFlags) {
            float most = -INFINITY;
            for (uint32_t bits = marked & here; bits; bits &= bits - 1) most = fmaxf(most, marked_value(__ffs(bits) - 1));
            y_max = fmaxf(y_max, warp_max(most));
        }
        double raw_sum = 0.0, mass = 0.0;
        uint32_t gone = banned;  // not alive
        const bool within = !absent_weighs && raw_max - raw_min <= 700.0f && (!kProcessed || y_max - temper(raw_min, p.apply_temperature != 0, p.temperature) <= 700.0f);
        if (within) {  // no exponential needs looking after
            const double raw_top = (double)raw_max, y_top = (double)y_max;
            const uint32_t apart = marked | ~here;  // marked logits are added below, absent ones (they may lie above y_top) never
#pragma unroll
            for (int i = 0; i < kVecs * 4; ++i) {
                const double x = (double)l[i];
                raw_sum += exp_of_gap(x - raw_top, power);
                if (kProcessed) {
                    const double e = exp_of_gap(tempered(x, reciprocal) - y_top, power);
                    // (what is left of a term without its upper half is next to nothing)
                    mass += kFlags ? __hiloint2double(((apart >> i) & 1u) ? 0 : __double2hiint(e), __double2loint(e)) : e;
                }
            }
        } else {  // logits further apart than an exponential reaches; ends of a row whose absent slots would weigh
#pragma unroll 1
            for (int i = 0; i < kVecs * 4; ++i) {
                if (!((here >> i) & 1u)) continue;
                const float x = p.logits[row * p.row_stride + lane_col + (i >> 2) * 128 + (i & 3)];
                raw_sum += exp_below(x, raw_max);
                if (kProcessed && !((marked >> i) & 1u)) {
                    const float y = temper(x, p.apply_temperature != 0, p.temperature);
                    mass += exp_below(y, y_max);
                    if (!(y > -INFINITY)) gone |= 1u << i;  // (a quotient that overflowed)
                }
            }
        }
        if (kFlags) {
            for (uint32_t bits = marked & here; bits; bits &= bits - 1) {
                const int i = __ffs(bits) - 1;
                const float y = marked_value(i);
                if (y > -INFINITY) mass += exp_below(y, y_max); else gone |= 1u << i;
            }
        }
        raw_sum = warp_sum(raw_sum);
        mass = kProcessed ? warp_sum(mass) : raw_sum;
        const uint32_t alive = __reduce_add_sync(0xFFFFFFFFu, (uint32_t)__popc(here & ~gone));
        const bool all_finite = __all_sync(0xFFFFFFFFu, finite);
        if (lane == 0) {
            SegmentStats s;
            s.raw_sum = raw_sum;  // (a segment past the end of its row: maxima of -inf, sums of nothing)
            s.mass = mass;
            s.raw_max = raw_max;
            s.y_max = y_max;
            s.alive = alive;
            s.nonfinite = all_finite ? 0u : 1u;
            p.stats[row * p.segments + segment] = s;
        }
    }
    if (ends_the_grid) grid_dependency_wait();
}

}  // namespace

cudaError_t launch_whole_rows(const WholeRowParams& p, cudaStream_t stream) {
    if (p.rows <= 0) return cudaSuccess;
    if (p.rows > 65535ll * 65535ll || p.rows > 0x7FFFFFFFll) return cudaErrorInvalidConfiguration;
    // One segment per warp up to 24,000 segments (some five rounds of the 148 SMs x 32 warps that are resident); from there on up to
    // four, one after the other, which share a CTA's bitmap.
    WholeRowParams q = p;
    q.segments_per_warp = (int)std::max<int64_t>(1, std::min<int64_t>(kMostPerWarp, p.rows * p.segments / 12000));
    const int64_t per_cta = (int64_t)kWarps * q.segments_per_warp;
    const dim3 grid((unsigned)((p.segments + per_cta - 1) / per_cta), (unsigned)std::min<int64_t>(p.rows, 65535),
                    (unsigned)((p.rows + 65534) / 65535));
    const bool flags = p.history_ids != nullptr || p.num_banned > 0;
    const auto kernel = flags ? weigh_segments_kernel<true, true> : p.apply_temperature ? weigh_segments_kernel<true, false> : weigh_segments_kernel<false, false>;
    const cudaError_t e = launch_overlapping(kernel, grid, dim3(kThreads), 0, stream, q);
    if (e != cudaSuccess) return e;
    return launch_overlapping(draw_token_kernel, dim3((unsigned)p.rows), dim3(kThreads), 0, stream, q);
}

}  // namespace psx
