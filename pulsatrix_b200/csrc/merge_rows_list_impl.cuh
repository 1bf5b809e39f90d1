// One row of the survivor stage by a block of kMergeThreads threads, the usual way: no sort and no serial walk.  Rows that this way
// does not hold, or whose decision comes too close to its level, are replayed in the reference's own order by merge_row.
//
// A decision of the reference (src/generation.cpp:80-152) compares a running sum with a level: the top-p walk (value ascending,
// then column ascending) with 1 - top_p, the draw's walk (column ascending) with u.  Where an entry stands in such a walk, the sum up
// to it is the sum over the entries that come before it.  list_top_k has a list of little more than k entries: every entry
// forms its own sum by looking at all the others.  list_nucleus may have thousands: a histogram of the mass over 256 ranges of
// the value (then of the column) gives the sums at the edges of the ranges, and only the entries of the one range that the level
// falls into look at one another.  The sums are made of integers, units of a power of two of the largest term, so they are
// the same in any order; they differ from the reference's sequential sums by rounding only (n units), and a decision that comes
// closer to its level than that allows is not taken here.
//
// Latency bound: a few KB per row out of L2, then dependent steps by one block (one row of 49,152 under a top-k of 50: the whole
// call 19.6 us with sorts and serial walks, 10.9 now; 256 nucleus rows of 128,256: 104 and 64.7 us).  What counts is the number of instructions one
// after another: candidates are fetched together with their counts, chunk by chunk over all lists (the same chunk of
// every list first, so that the warps share the slots that are in use), and nothing but a comparison, a bin and a float
// exponential is done for a candidate before the cut; double-precision exponentials, divides and the logarithm are for what is left.
#pragma once

#include "merge_rows_impl.cuh"
#include "psx_exp.cuh"

namespace psx {
namespace survivor {

constexpr int kListWarps = kMergeThreads / 32;
constexpr int kListCap = 512;        // entries that look at one another
constexpr int kWideLeast = 2048;     // room for candidates at or above the threshold, before the cut (top-k): at least
constexpr int kNucleusCap = 4096;    // the same without a top-k
constexpr double kDoubt = 1e-11;     // of the whole mass: well above 512 units of 2^-52
constexpr double kNucleusDoubt = 4e-9;  // the same for kNucleusCap units of 2^-40
constexpr uint32_t kRemoved = 0x80000000u;
constexpr int kTopKArena = kListCap * (16 + 8 + 4) + kWideLeast * 12;
constexpr int kNucleusArena = kListCap * (16 + 4) + kNucleusCap * 20 + 4 * 256 * 4;

// Where one row's inputs lie and where its results go.
struct RowView {
    const char *stats, *counts, *lists;
    int64_t stats_stride, count_stride, list_stride;  // from part to part
    int32_t cap;                                      // slots of a part's list
    const double* u;
    int64_t* token;
    float* log_prob;
    int32_t* status;
    psx_row_diag* diag;
};

__device__ __forceinline__ RowView view_of_row(const MergeParams& p, const int64_t row) {
    RowView v;
    v.stats = static_cast<const char*>(p.stats) + row * p.stats_row_stride;
    v.counts = static_cast<const char*>(p.part_counts) + row * p.count_row_stride;
    v.lists = static_cast<const char*>(p.candidates) + row * p.cand_row_stride;
    v.stats_stride = p.stats_part_stride;
    v.count_stride = p.count_part_stride;
    v.list_stride = p.cand_part_stride;
    v.cap = p.part_cap;
    v.u = p.uniforms ? p.uniforms + row : nullptr;
    v.token = p.tokens + row;
    v.log_prob = p.log_probs + row;
    v.status = p.row_status + row;
    v.diag = p.diag ? p.diag + row : nullptr;
    return v;
}

// What every warp knows of the row's parts; lane L keeps part L's record.
struct PartsJoined {
    float raw_max, y_max, thr;
    uint32_t bad, tail_alive, count, longest;
    PartStats mine;
};

// The row's candidates, four chunks of 32 per warp at a time.
struct ChunkWalk {
    const char* lists;
    int64_t stride;
    int parts, cap, lane, part, chunk, step_part, step_chunk;

    __device__ __forceinline__ ChunkWalk(const MergeParams& p, const RowView& v)
        : lists(v.lists), stride(v.list_stride), parts(p.parts), cap(v.cap), lane(threadIdx.x & 31) {
        const uint32_t warp = threadIdx.x >> 5, per_part = (0x10000u + parts - 1) / (uint32_t)parts;  // (x * per_part) >> 16 == x / parts for x <= 8
        chunk = (int)((warp * per_part) >> 16);
        part = (int)warp - chunk * parts;
        step_chunk = (int)((kListWarps * per_part) >> 16);
        step_part = kListWarps - step_chunk * parts;
    }
    // where[q]: part | first slot << 8 (slots beyond the list's count are fetched as well, and not looked at)
    __device__ __forceinline__ void fetch(uint2 (&c)[4], uint32_t (&where)[4]) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int slot = chunk * 32 + lane;
            where[q] = (uint32_t)part | ((uint32_t)(chunk * 32) << 8);
            c[q] = slot < cap ? reinterpret_cast<const uint2*>(lists + part * stride)[slot] : make_uint2(0, 0);
            part += step_part;
            chunk += step_chunk;
            if (part >= parts) { part -= parts; ++chunk; }
        }
    }
    __device__ __forceinline__ bool beyond(uint32_t longest) const { return (uint32_t)(chunk * 32) >= longest; }
};

__device__ __forceinline__ void load_parts(const MergeParams& p, const RowView& v, PartsJoined& j) {
    const int lane = threadIdx.x & 31;
    j.mine.raw_tail = 0.0; j.mine.proc_tail = 0.0;
    j.mine.raw_max = -FLT_MAX; j.mine.y_max = -INFINITY; j.mine.thr = -INFINITY;
    j.mine.nonfinite = 0; j.mine.alive_tail = 0; j.mine.overflow = 0;
    j.count = 0;
    if (lane < p.parts) {
        j.mine = *reinterpret_cast<const PartStats*>(v.stats + lane * v.stats_stride);
        j.count = *reinterpret_cast<const uint32_t*>(v.counts + lane * v.count_stride);
    }
}

// false: the row is not for this way (a list that ran out of slots).  A part that lies below the threshold of another as a whole, and so
// far below the row's maxima that all its logits together weigh less than 1e-38 of them, is left aside instead: the parts of a row in
// which all but a few logits are masked by a number (one row of 50,000 with 50 left, top-k 1: 484 us decided from the row, 10 so).
__device__ __forceinline__ bool join_parts(const MergeParams& p, const RowView& v, PartsJoined& j) {
    j.count = min(j.count, (uint32_t)v.cap);
    j.raw_max = warp_max(j.mine.raw_max);
    j.y_max = warp_max(j.mine.y_max);
    j.thr = warp_max(j.mine.thr);
    j.bad = __reduce_or_sync(0xFFFFFFFFu, (j.mine.nonfinite & 3u) | (j.mine.overflow ? 4u : 0u));
    if ((j.bad & 4u) != 0) {
        const bool apply_t = p.apply_temperature != 0;
        const bool aside = j.mine.raw_max < j.raw_max - 100.0f && j.mine.y_max < relax_threshold(j.thr, apply_t, p.temperature) &&
                           temper(j.mine.y_max, apply_t, p.temperature) < temper(j.y_max, apply_t, p.temperature) - 100.0f;
        if (j.mine.overflow && aside) {
            j.count = 0;
            j.mine.alive_tail = 1;  // (some of it is outside the lists, however many)
        }
        j.bad = (j.bad & 3u) | (__any_sync(0xFFFFFFFFu, j.mine.overflow && !aside) ? 4u : 0u);
    }
    j.tail_alive = __reduce_add_sync(0xFFFFFFFFu, j.mine.alive_tail);
    j.longest = __reduce_max_sync(0xFFFFFFFFu, j.count);
    return (j.bad & 4u) == 0;
}

__device__ __forceinline__ void report_bad_row(const RowView& v, const PartsJoined& j) {  // (by one thread)
    *v.token = -1;
    *v.log_prob = 0.0f;
    *v.status = (j.bad & 2u) ? PSX_ROW_DEVICE_TIMEOUT : (j.bad & 1u) ? PSX_ROW_NON_FINITE : PSX_ROW_ALL_REMOVED;
    if (v.diag) *v.diag = psx_row_diag{0, 0, INFINITY, INFINITY};
}

// true: the row has a non-finite logit, a copy that did not arrive, or nothing left (top: its largest processed value; -inf
// also when every quotient by the temperature overflows); its status is written
__device__ __forceinline__ bool settle_bad_row(const RowView& v, const PartsJoined& j, const float top) {
    if (j.bad == 0 && top > -INFINITY) return false;
    if (threadIdx.x == 0) report_bad_row(v, j);
    return true;
}

// sum over the warp of integers below 2^59, by two of the 32-bit reductions
__device__ __forceinline__ u64 warp_sum_units(u64 v) {
    const uint32_t lo = __reduce_add_sync(0xFFFFFFFFu, (uint32_t)v & 0x7FFFFFFu), hi = __reduce_add_sync(0xFFFFFFFFu, (uint32_t)(v >> 27));
    return (u64)lo + ((u64)hi << 27);
}

// The raw sum-exp: what the row pass left behind (the parts' tails, joined by one warp), and float exponentials of the candidates
// below the cut, taken as the row pass takes its own (against the rounded exponent of the maximum, the rounding put back
// once); candidates above it are taken in double.
struct RawSum {
    static constexpr float kLog2e = 1.4426950408889634f;
    float c_l2, c_res, low = 0.0f;
    double high = 0.0;
    __device__ __forceinline__ explicit RawSum(float raw_max) {
        c_l2 = __fmul_rn(raw_max, kLog2e);
        c_res = __fmaf_rn(raw_max, kLog2e, -c_l2);
    }
    __device__ __forceinline__ void add_low(float l) { low += ex2_approx(__fmaf_rn(l, kLog2e, -c_l2)); }
    // The warp's sum, in units of 2^-40 of the largest term: integer reductions, a fraction of the time of five additions in double
    // one after another.  (A lane has up to 128 terms of at most one, 256 where a warp has a row of eight full lists to itself, as a rule a few: their
    // float sum differs from another order's by a rounding of the float log-probability, the units stay below 2^49.)
    __device__ __forceinline__ u64 of_warp() const { return warp_sum_units((u64)__double2ull_rn((high + (double)low * exp2_of_minus_small(c_res)) * 0x1p40)); }
};

__device__ __forceinline__ double tails_of_parts(const PartsJoined& j) {  // by one warp; the sum in every lane
    double tail = 0.0;
    if (j.mine.raw_tail > 0.0) tail = j.mine.raw_tail * exp((double)j.mine.raw_max - (double)j.raw_max);
    return warp_sum(tail);
}

// exp(v - top), by the whole warp
__device__ __forceinline__ double exp_to(float v, float top, bool there, double power) {
    const bool small = !there || v - top < kExpFloor;
    const double e = exp_of_gap(small ? -1.0 : (double)v - (double)top, power);
    return small ? 0.0 : e;
}

// The sum over the lanes before this one, and over all, by a whole warp.
__device__ __forceinline__ u64 lanes_before(u64 v, int lane, u64& all) {
    u64 incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const u64 up = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += up;
    }
    all = __shfl_sync(0xFFFFFFFFu, incl, 31);
    return incl - v;
}

// ---- greedy ----------------------------------------------------------------------------------------------------------------
template <class Ready>
__device__ __forceinline__ bool list_greedy(const MergeParams& p, const RowView& v, Ready ready) {
    __shared__ u64 s_z[kListWarps], s_best[kListWarps];
    __shared__ double s_tails;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    PartsJoined j;
    uint2 c[4];
    uint32_t where[4];
    ChunkWalk walk(p, v);
    ready();
    load_parts(p, v, j);
    walk.fetch(c, where);
    if (!join_parts(p, v, j)) return false;
    if (settle_bad_row(v, j, j.y_max)) return true;
    PSX_MERGE_STAGE(3);
    const float keep_from = fmaxf(j.y_max, -FLT_MAX);
    RawSum z(j.raw_max);
    u64 best = 0;  // the maximum's lowest column, as ~column above the raw logit
    for (;;) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t here = __shfl_sync(0xFFFFFFFFu, j.count, where[q] & 255u);
            if ((where[q] >> 8) + lane < here) {
                const float l = __uint_as_float(c[q].x);
                if (processed_before_temperature(l, c[q].y, p.penalty) >= keep_from) {
                    z.high += exp_below(l, j.raw_max);
                    const u64 key = ((u64)~(c[q].y & kColumnMask) << 32) | c[q].x;
                    best = key > best ? key : best;
                } else {
                    z.add_low(l);
                }
            }
        }
        if (walk.beyond(j.longest)) break;
        walk.fetch(c, where);
    }
    const u64 of_warp = z.of_warp();
    if (warp == kListWarps - 1) {
        const double tails = tails_of_parts(j);
        if (lane == 0) s_tails = tails;
    }
    const uint32_t top = __reduce_max_sync(0xFFFFFFFFu, (uint32_t)(best >> 32));
    if ((uint32_t)(best >> 32) == top && (top != 0 || lane == 0)) s_best[warp] = best;  // (columns differ: one lane)
    if (lane == 0) s_z[warp] = of_warp;
    __syncthreads();
    PSX_MERGE_STAGE(4);
    if (threadIdx.x == 0) {
        best = s_best[0];
        u64 sum = s_z[0];
#pragma unroll
        for (int w = 1; w < kListWarps; ++w) {
            best = s_best[w] > best ? s_best[w] : best;
            sum += s_z[w];
        }
        *v.status = PSX_ROW_OK;
        *v.token = (int64_t)(uint32_t)~(uint32_t)(best >> 32);
        *v.log_prob = (float)(((double)__uint_as_float((uint32_t)best) - (double)j.raw_max) - log((double)sum * 0x1p-40 + s_tails));  // src/generation.cpp:156
        if (v.diag) *v.diag = psx_row_diag{1, 1, INFINITY, INFINITY};
    }
    PSX_MERGE_STAGE(9);
    return true;
}

// The same by one warp, for many rows: a greedy row has a handful of candidates, and what a block does for it is mostly to meet.
__device__ __forceinline__ bool list_greedy_by_warp(const MergeParams& p, const RowView& v) {
    const int lane = threadIdx.x & 31;
    PartsJoined j;
    uint2 c[4];
    // 32 slots of four parts' lists at a time (slots beyond a list's count are fetched as well, and not looked at)
    auto fetch = [&](uint32_t slot, int part) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            c[q] = part + q < p.parts && slot < (uint32_t)v.cap ? reinterpret_cast<const uint2*>(v.lists + (part + q) * v.list_stride)[slot] : make_uint2(0, 0);
        }
    };
    load_parts(p, v, j);
    fetch(lane, 0);
    if (!join_parts(p, v, j)) return false;
    if (j.bad != 0 || !(j.y_max > -INFINITY)) {
        if (lane == 0) report_bad_row(v, j);
        return true;
    }
    const float keep_from = fmaxf(j.y_max, -FLT_MAX);
    RawSum z(j.raw_max);
    u64 best = 0;  // the maximum's lowest column, as ~column above the raw logit
    for (uint32_t first = 0; first < j.longest; first += 32) {
        for (int part = 0; part < p.parts; part += 4) {
            if (first + (uint32_t)part > 0) fetch(first + lane, part);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint32_t here = __shfl_sync(0xFFFFFFFFu, j.count, (part + q) & 31);
                if (part + q >= p.parts || first + lane >= here) continue;
                const float l = __uint_as_float(c[q].x);
                if (processed_before_temperature(l, c[q].y, p.penalty) >= keep_from) {
                    z.high += exp_below(l, j.raw_max);
                    const u64 key = ((u64)~(c[q].y & kColumnMask) << 32) | c[q].x;
                    best = key > best ? key : best;
                } else {
                    z.add_low(l);
                }
            }
            __syncwarp();
        }
    }
    const double tails = tails_of_parts(j);
    const u64 sum = z.of_warp();
    const uint32_t top = __reduce_max_sync(0xFFFFFFFFu, (uint32_t)(best >> 32));
    if ((uint32_t)(best >> 32) == top && (top != 0 || lane == 0)) {  // (columns differ: one lane)
        *v.status = PSX_ROW_OK;
        *v.token = (int64_t)(uint32_t)~top;
        *v.log_prob = (float)(((double)__uint_as_float((uint32_t)best) - (double)j.raw_max) - log((double)sum * 0x1p-40 + tails));  // src/generation.cpp:156
        if (v.diag) *v.diag = psx_row_diag{1, 1, INFINITY, INFINITY};
    }
    return true;
}

// ---- sampling under a top-k ------------------------------------------------------------------------------------------------
template <class Ready>
__device__ __forceinline__ bool list_top_k(const MergeParams& p, const int64_t row, const RowView& v, u64* dyn, Ready ready) {
    ulonglong2* const s_list = reinterpret_cast<ulonglong2*>(dyn);       // (ordered value << 32) | column; units of 2^-52
    uint32_t* const s_by_value = reinterpret_cast<uint32_t*>(s_list + kListCap);  // place by column << 16 | entry
    uint32_t* const s_by_column = s_by_value + kListCap;                          // entry, kRemoved
    float* const s_raw = reinterpret_cast<float*>(s_by_column + kListCap);
    u64* const s_wide = reinterpret_cast<u64*>(s_raw + kListCap);        // raw logit, column | flags
    // as many candidates as the launch has shared memory for: 3670 and more (64 rows of 151,936, top-k 200: 80 us with 2048, 58 so)
    const int wide_cap = (p.dyn_bytes - kListCap * (16 + 8 + 4)) / 12;
    float* const s_wide_y = reinterpret_cast<float*>(s_wide + wide_cap);
    __shared__ uint32_t s_hist[32];
    __shared__ u64 s_z[kListWarps];
    __shared__ double s_log_z;
    __shared__ int s_wide_n, s_n, s_doubt, s_won, s_survivors;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t below = (1u << lane) - 1u;
    const bool apply_t = p.apply_temperature != 0;
    PartsJoined j;
    uint2 c[4];
    uint32_t where[4];
    ChunkWalk walk(p, v);
    const double power = exp_power_of_lane();
    if (tid < 32) s_hist[tid] = 0;
    if (tid == 0) { s_wide_n = 0; s_n = 0; s_doubt = 0; s_won = 0; s_survivors = 0; }
    ready();
    load_parts(p, v, j);
    walk.fetch(c, where);
    const double u = v.u ? *v.u : 0.5;
    __syncthreads();
    if (!join_parts(p, v, j)) return false;
    const float x_max = temper(j.y_max, apply_t, p.temperature);
    if (settle_bad_row(v, j, x_max)) return true;
    PSX_MERGE_STAGE(3);
    // ---- 1. what reaches the largest part threshold (that part alone has k logits which reach it), and its histogram -------
    const float keep_from = relax_threshold(j.thr, apply_t, p.temperature);
    // (Any map from value to bin that never decreases as the value falls would do.  Without a threshold -- a row that was handed on whole --
    // four bins per octave of the distance, from 1/16 on, the last one for all the rest: 2000 rows of 600, top-k 50: 136 us with one bin for
    // all of them, which no list holds.)
    const bool whole = j.thr == -INFINITY;
    float bin_scale = 0.0f;
    if (j.y_max - keep_from > 0.0f && j.y_max - keep_from < INFINITY) bin_scale = __fdividef(31.5f, j.y_max - keep_from);
    auto bin_of = [&](float y) {
        const float d = fmaxf(__fsub_rn(j.y_max, y), 0.0f);
        const int bin = whole ? (int)(__float_as_uint(d) >> 21) - (0x3D800000 >> 21) + 1 : (int)__fmul_rn(d, bin_scale);
        return min(31, max(0, bin));
    };
    RawSum z(j.raw_max);
    for (;;) {
        float y[4];
        uint32_t votes[4];
        int all = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t here = __shfl_sync(0xFFFFFFFFu, j.count, where[q] & 255u);
            const bool there = (where[q] >> 8) + lane < here;
            const float l = __uint_as_float(c[q].x);
            y[q] = there ? l : -INFINITY;
            if (there && (c[q].y & ~kColumnMask) != 0) y[q] = processed_before_temperature(l, c[q].y, p.penalty);
            const bool on = y[q] >= keep_from;
            if (there && !on) z.add_low(l);
            if (on) atomicAdd(&s_hist[bin_of(y[q])], 1u);
            votes[q] = __ballot_sync(0xFFFFFFFFu, on);
            all += __popc(votes[q]);
        }
        if (all != 0) {
            int at = 0;
            if (lane == 0) at = atomicAdd(&s_wide_n, all);
            at = __shfl_sync(0xFFFFFFFFu, at, 0);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int mine = at + __popc(votes[q] & below);
                if (((votes[q] >> lane) & 1u) && mine < wide_cap) {
                    s_wide[mine] = ((u64)c[q].x << 32) | c[q].y;
                    s_wide_y[mine] = y[q];
                }
                at += __popc(votes[q]);
            }
        }
        if (walk.beyond(j.longest)) break;
        walk.fetch(c, where);
    }
    __syncthreads();
    PSX_MERGE_STAGE(4);
    const int wide = s_wide_n;
    if (wide > wide_cap) return false;
    // ---- 2. the list: down to the bin in which the count reaches k.  The place in the histogram is by the value before the
    // temperature; a candidate is listed by the bin of its value raised by what the divide can merge (twice
    // relax_threshold's margin), so one that is not listed lies below k others after the divide as well -------------------------
    int cut = 31;
    {
        uint32_t incl = s_hist[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t up = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o) incl += up;
        }
        const uint32_t reached = __ballot_sync(0xFFFFFFFFu, (int64_t)incl >= p.top_k);
        if (reached != 0) cut = __ffs(reached) - 1;
    }
    if (!(fabsf(x_max) < INFINITY)) return false;  // (quotients that overflow tie: merge_row's business)
    for (int first = warp * 32; first < wide; first += kMergeThreads) {
        const int e = first + lane;
        const u64 cand = e < wide ? s_wide[e] : 0;
        const float l = __uint_as_float((uint32_t)(cand >> 32)), y = e < wide ? s_wide_y[e] : -INFINITY;
        const float up = apply_t ? __fadd_rn(y, __fmaf_rn(fabsf(y), 0x1p-20f, __fmul_rn(p.temperature, 0x1p-146f))) : y;
        const float x = temper(y, apply_t, p.temperature);
        const bool on = e < wide && bin_of(up) <= cut && x > -INFINITY;  // (a quotient that overflowed is removed)
        if (e < wide && !on) z.add_low(l);
        const uint32_t takers = __ballot_sync(0xFFFFFFFFu, on);
        if (takers == 0) continue;
        int at = 0;
        if (lane == 0) at = atomicAdd(&s_n, __popc(takers));
        const u64 units = (u64)__double2ull_rn(exp_to(x, x_max, on, power) * 0x1p52);
        z.high += exp_to(l, j.raw_max, on, power);
        at = __shfl_sync(0xFFFFFFFFu, at, 0) + __popc(takers & below);
        if (on && at < kListCap) {
            s_list[at] = make_ulonglong2(((u64)ordered_key(x) << 32) | (uint32_t)(cand & kColumnMask), units);
            s_raw[at] = l;
        }
    }
    {
        const u64 sum = z.of_warp();
        if (lane == 0) s_z[warp] = sum;
    }
    __syncthreads();
    PSX_MERGE_STAGE(5);
    const int n = s_n;
    if (n > kListCap || n == 0) return false;
    // ---- 3. every entry's place by value and by column: it looks at all the others; T neighbouring threads share one ------------
    {
        int n_pad = 8;
        while (n_pad < n && n_pad < kMergeThreads) n_pad <<= 1;
        const int shift = 8 - (31 - __clz(n_pad)), T = 1 << shift, slice = tid & (T - 1);
        for (int e0 = 0; e0 < n; e0 += n_pad) {
            const int e = e0 + (tid >> shift);
            const u64 me = e < n ? s_list[e].x : 0;
            uint32_t places = 0;  // by value, descending (equal values: the higher column first); by column, above it
#pragma unroll 4
            for (int i = slice; i < n; i += T) {
                const u64 other = s_list[i].x;
                places += other > me ? 1u : 0u;
                places += (uint32_t)other < (uint32_t)me ? 0x10000u : 0u;
            }
            for (int o = T >> 1; o > 0; o >>= 1) places += __shfl_xor_sync(0xFFFFFFFFu, places, o);
            if (slice == 0 && e < n) s_by_value[places & 0xFFFFu] = (places & 0xFFFF0000u) | (uint32_t)e;
        }
    }
    __syncthreads();
    PSX_MERGE_STAGE(6);
    bool won = false, doubt = false;
    int won_entry = 0, survivors = 0;
    double won_margin = 0.0, top_p_margin = INFINITY;
    if (warp == kListWarps - 1) {
        // the logarithm for the log-probability, meanwhile
        u64 sum = 0;
#pragma unroll
        for (int w = 0; w < kListWarps; ++w) sum += s_z[w];
        const double log_z = log(tails_of_parts(j) + (double)sum * 0x1p-40);
        if (lane == 0) s_log_z = log_z;
    } else if (warp == 0) {
        // ---- 4. who stays, by one warp: a lane takes `each` entries one after another in the order of the values ------------------
        const int each = (n + 31) >> 5, begin = lane * each, end = min(begin + each, n);
        const uint32_t kth = n >= p.top_k ? (uint32_t)(s_list[s_by_value[p.top_k - 1] & 0xFFFFu].x >> 32) : 0u;
        u64 sum = 0;
        for (int i = begin; i < end; ++i) {
            const ulonglong2 it = s_list[s_by_value[i] & 0xFFFFu];
            sum += (uint32_t)(it.x >> 32) >= kth ? it.y : 0;  // :80-88: the k-th value and its ties stay
        }
        u64 all, after = lanes_before(sum, lane, all);
        const double limit = 1.0 - (double)p.top_p, whole = (double)all * 0x1p-52, min_p = (double)p.min_p;
        for (int i = begin; i < end; ++i) {
            const uint32_t at = s_by_value[i];
            const ulonglong2 it = s_list[at & 0xFFFFu];
            bool stays = (uint32_t)(it.x >> 32) >= kth;
            if (stays && p.top_p < 1.0f && after != 0) {  // :89-103; the last of the walk always stays
                const double beyond = (double)(all - after) * 0x1p-52 - limit * whole;
                stays = beyond > 0.0;
                doubt = doubt || fabs(beyond) < kDoubt * whole;
                top_p_margin = fmin(top_p_margin, fabs(beyond));
            }
            after += it.y;
            if (stays && min_p > 0.0 && it.y < (1ull << 52)) {  // :104-111, against the first maximum's exp(0)
                const double mass = (double)it.y * 0x1p-52;
                stays = mass >= min_p;
                doubt = doubt || fabs(mass - min_p) < kDoubt;
            }
            s_by_column[at >> 16] = (at & 0xFFFFu) | (stays ? 0u : kRemoved);
            survivors += stays ? 1 : 0;
        }
        doubt = __any_sync(0xFFFFFFFFu, doubt);
        __syncwarp();
        PSX_MERGE_STAGE(7);
        // ---- 5. the draw (:140-152): the entry whose share of the running sum, by ascending column, holds u -----------------------
        sum = 0;
        for (int i = begin; i < end; ++i) {
            const uint32_t at = s_by_column[i];
            sum += (at & kRemoved) ? 0 : s_list[at].y;
        }
        u64 before = lanes_before(sum, lane, all);
        const double target = u * (double)all;
        for (int i = begin; i < end && !doubt; ++i) {
            const uint32_t at = s_by_column[i];
            if (at & kRemoved) continue;
            const u64 mass = s_list[at].y;
            const double lo = target - (double)before, hi = (double)(before + mass) - target;
            if (lo >= 0.0 && hi > 0.0) {
                won_margin = before == 0 ? hi : fmin(lo, hi);
                won_entry = (int)at;
                won = won_margin >= kDoubt * (double)all;  // (nobody takes it otherwise: replayed)
            }
            before += mass;
        }
        if (won) s_won = 1;
        if (doubt && lane == 0) s_doubt = 1;
        if (v.diag) {
            won_margin /= (double)all;
            top_p_margin /= whole;
            survivors = (int)__reduce_add_sync(0xFFFFFFFFu, (uint32_t)survivors);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) top_p_margin = fmin(top_p_margin, __shfl_xor_sync(0xFFFFFFFFu, top_p_margin, o));
        }
    }
    __syncthreads();
    PSX_MERGE_STAGE(8);
    if (p.survivor_cols != nullptr) {  // the surviving set itself (ProcessLogits)
        if (s_doubt != 0 || n > p.survivor_cap) return false;
        for (int i = tid; i < n; i += kMergeThreads) {
            const uint32_t e = s_by_column[i];
            if (e & kRemoved) continue;
            const int64_t at = row * p.survivor_cap + atomicAdd(&s_survivors, 1);
            p.survivor_cols[at] = (uint32_t)s_list[e].x;
            p.survivor_vals[at] = from_ordered_key((uint32_t)(s_list[e].x >> 32));
        }
        __syncthreads();
        if (tid == 0) {
            p.survivor_counts[row] = (uint32_t)s_survivors;
            *v.status = PSX_ROW_OK;
        }
        return true;
    }
    if (won) {
        *v.status = PSX_ROW_OK;
        *v.token = (int64_t)(uint32_t)s_list[won_entry].x;
        *v.log_prob = (float)(((double)s_raw[won_entry] - (double)j.raw_max) - s_log_z);  // :133,156
        if (v.diag) *v.diag = psx_row_diag{n, survivors, won_margin, top_p_margin};
    }
    PSX_MERGE_STAGE(9);
    return s_won != 0;
}

// ---- sampling without a top-k ----------------------------------------------------------------------------------------------
// Masses by range: 256 sums of units of 2^-40, as 20 low and 21 high bits in two words.  (4096 of either fit 32 bits, but for 4096 entries that all weigh
// 2^40: their sum reads zero, no range is found and the row is replayed.)
__device__ __forceinline__ void add_units(uint32_t* hist, uint32_t bin, u64 units) {
    atomicAdd(&hist[bin], (uint32_t)units & 0xFFFFFu);
    atomicAdd(&hist[256 + bin], (uint32_t)(units >> 20));
}
// The running sums over the ranges, by a whole warp; lane L holds ranges 8L to 8L + 7.
struct RangeSums {
    u64 run[8], lead, all;
    int lane;
    __device__ __forceinline__ explicit RangeSums(const uint32_t* hist) : lane(threadIdx.x & 31) {
        u64 sum = 0;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const uint4 lo = reinterpret_cast<const uint4*>(hist)[2 * lane + half], hi = reinterpret_cast<const uint4*>(hist + 256)[2 * lane + half];
            run[4 * half + 0] = sum += lo.x + ((u64)hi.x << 20);
            run[4 * half + 1] = sum += lo.y + ((u64)hi.y << 20);
            run[4 * half + 2] = sum += lo.z + ((u64)hi.z << 20);
            run[4 * half + 3] = sum += lo.w + ((u64)hi.w << 20);
        }
        lead = lanes_before(sum, lane, all);
    }
    // The first range whose running sum reaches `level` (kBeyond: goes past it), 256 when none does; the sum before it.
    template <bool kBeyond>
    __device__ __forceinline__ uint32_t find(double level, u64& before) const {
        uint32_t short_of = 0;
        u64 last = lead;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const double reach = (double)(lead + run[q]);
            if (!(kBeyond ? reach > level : reach >= level)) { ++short_of; last = lead + run[q]; }
        }
        const uint32_t lanes = __ballot_sync(0xFFFFFFFFu, short_of < 8);
        if (lanes == 0) { before = all; return 256u; }
        const int src = __ffs(lanes) - 1;
        before = __shfl_sync(0xFFFFFFFFu, last, src);
        return 8u * src + __shfl_sync(0xFFFFFFFFu, short_of, src);
    }
};

template <class Ready>
__device__ __forceinline__ bool list_nucleus(const MergeParams& p, const int64_t row, const RowView& v, u64* dyn, Ready ready) {
    ulonglong2* const s_list = reinterpret_cast<ulonglong2*>(dyn);
    float* const s_raw = reinterpret_cast<float*>(s_list + kListCap);
    uint32_t* const s_by_value = reinterpret_cast<uint32_t*>(s_raw + kListCap);  // masses over 256 ranges of the value
    uint32_t* const s_by_column = s_by_value + 512;                              // ... and of the column
    u64* const s_unit = reinterpret_cast<u64*>(s_by_column + 512);               // a candidate's mass in units of 2^-40 of the largest
    float* const s_l = reinterpret_cast<float*>(s_unit + kNucleusCap);
    float* const s_x = s_l + kNucleusCap;
    uint32_t* const s_col = reinterpret_cast<uint32_t*>(s_x + kNucleusCap);
    __shared__ u64 s_z[kListWarps], s_rest[kListWarps];
    __shared__ double s_tails, s_proc_tails;
    __shared__ u64 s_cut_key, s_margin;
    __shared__ uint32_t s_dropped[kListWarps];
    __shared__ int s_n, s_cut_n, s_draw_n, s_decided, s_survivors, s_doubt;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t below = (1u << lane) - 1u;
    const bool apply_t = p.apply_temperature != 0;
    PartsJoined j;
    uint2 c[4];
    uint32_t where[4];
    ChunkWalk walk(p, v);
    const double power = exp_power_of_lane();
    reinterpret_cast<uint4*>(s_by_value)[tid] = make_uint4(0, 0, 0, 0);  // both histograms
    if (tid == 0) { s_n = 0; s_cut_n = 0; s_draw_n = 0; s_decided = 0; s_survivors = 0; s_doubt = 0; s_cut_key = ~0ull; s_margin = ~0ull; }
    ready();
    load_parts(p, v, j);
    walk.fetch(c, where);
    const double u = v.u ? *v.u : 0.5;
    __syncthreads();
    if (!join_parts(p, v, j)) return false;
    const float x_max = temper(j.y_max, apply_t, p.temperature);
    if (settle_bad_row(v, j, x_max)) return true;
    PSX_MERGE_STAGE(3);
    // ---- 1. candidates at or above the largest part threshold into shared memory, their masses by value; what lies below it
    // belongs to the rest of the vocabulary, which the candidates do not cover ---------------------------------------------------
    if (!(fabsf(x_max) < INFINITY)) return false;  // (quotients that overflow tie: merge_row's business)
    const float keep_from = relax_threshold(j.thr, apply_t, p.temperature);
    const float x_low = temper(keep_from, apply_t, p.temperature);
    float bin_scale = 0.0f;
    if (j.thr == -INFINITY) bin_scale = 8.0f;  // (no threshold, i.e. the row was handed on whole: an eighth of a unit per range, the last one for the rest)
    else if (x_max - x_low > 0.0f && x_max - x_low < INFINITY) bin_scale = __fdiv_rn(255.0f, x_max - x_low);
    auto bin_of = [&](float x) { return (uint32_t)max(0, min(255, (int)__fmul_rn(__fsub_rn(x_max, x), bin_scale))); };
    RawSum z(j.raw_max);
    double rest = 0.0;
    uint32_t dropped = 0;
    for (;;) {
        uint2 next[4];
        uint32_t where_next[4];
        const bool last = walk.beyond(j.longest);
        if (!last) walk.fetch(next, where_next);
        // (four candidates in straight line: their chains of dependent operations run side by side)
        float x[4];
        u64 units[4];
        uint32_t votes[4], there = 0;
        int all = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t here = __shfl_sync(0xFFFFFFFFu, j.count, where[q] & 255u);
            const bool in = (where[q] >> 8) + lane < here;
            there |= in ? 1u << q : 0u;
            x[q] = in ? __uint_as_float(c[q].x) : -INFINITY;
            if (in && (c[q].y & ~kColumnMask) != 0) x[q] = processed_before_temperature(x[q], c[q].y, p.penalty);
            votes[q] = __ballot_sync(0xFFFFFFFFu, x[q] >= keep_from);
            all += __popc(votes[q]);
        }
        if (apply_t) {
#pragma unroll
            for (int q = 0; q < 4; ++q) x[q] = __fdiv_rn(x[q], p.temperature);
        }
        double mass[4], raw[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) mass[q] = exp_to(x[q], x_max, x[q] > -INFINITY, power);
#pragma unroll
        for (int q = 0; q < 4; ++q) raw[q] = exp_to(__uint_as_float(c[q].x), j.raw_max, (votes[q] >> lane) & 1u, power);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const bool on = (votes[q] >> lane) & 1u, in = (there >> q) & 1u;
            units[q] = (u64)__double2ull_rn(mass[q] * 0x1p40);
            z.high += raw[q];  // (zero unless listed)
            if (on) add_units(s_by_value, bin_of(x[q]), units[q]);
            rest += on ? 0.0 : mass[q];
            dropped += !on && x[q] > -INFINITY ? 1u : 0u;
            if (in && !on) z.add_low(__uint_as_float(c[q].x));
        }
        if (all != 0) {
            int at = 0;
            if (lane == 0) at = atomicAdd(&s_n, all);
            at = __shfl_sync(0xFFFFFFFFu, at, 0);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int mine = at + __popc(votes[q] & below);
                if (((votes[q] >> lane) & 1u) && mine < kNucleusCap) {
                    s_unit[mine] = units[q];
                    s_l[mine] = __uint_as_float(c[q].x);
                    s_x[mine] = x[q];
                    s_col[mine] = c[q].y & kColumnMask;
                }
                at += __popc(votes[q]);
            }
        }
        if (last) break;
#pragma unroll
        for (int q = 0; q < 4; ++q) { c[q] = next[q]; where[q] = where_next[q]; }
    }
    {
        const u64 sum = z.of_warp(), rest_of_warp = warp_sum_units((u64)__double2ull_rn(rest * 0x1p40));
        if (warp == kListWarps - 1) {
            const double tails = tails_of_parts(j);
            if (lane == 0) s_tails = tails;
        } else if (warp == kListWarps - 2) {
            double tails = 0.0;
            if (j.mine.y_max > -INFINITY && j.mine.proc_tail > 0.0) {
                tails = j.mine.proc_tail * exp((double)temper(j.mine.y_max, apply_t, p.temperature) - (double)x_max);
            }
            tails = warp_sum(tails);
            if (lane == 0) s_proc_tails = tails;
        }
        dropped = __reduce_add_sync(0xFFFFFFFFu, dropped);
        if (lane == 0) { s_z[warp] = sum; s_rest[warp] = rest_of_warp; s_dropped[warp] = dropped; }
    }
    __syncthreads();
    PSX_MERGE_STAGE(4);
    const int n = s_n;
    if (n > kNucleusCap || n == 0) return false;
    u64 rest_units = 0, sum_units = 0, outside = j.tail_alive;
#pragma unroll
    for (int w = 0; w < kListWarps; ++w) { rest_units += s_rest[w]; sum_units += s_z[w]; outside += s_dropped[w]; }
    rest = (double)rest_units * 0x1p-40 + s_proc_tails;
    // ---- 2. the top-p (:89-103): the range that its level falls into ---------------------------------------------------------
    const double limit = 1.0 - (double)p.top_p, min_p = (double)p.min_p;
    const bool top_p_on = p.top_p < 1.0f, rest_alive = outside != 0;
    uint32_t cut_bin = 256u;
    double top_p_margin = INFINITY;
    u64 cut_key = 0;
    if (top_p_on) {
        u64 before;
        const RangeSums ranges(s_by_value);
        const double listed = (double)ranges.all * 0x1p-40, whole = listed + (rest_alive ? rest : 0.0);
        const double need = (whole - limit * whole) * 0x1p40;  // an entry stays while what comes after it is less
        // Everything outside the list leads the ascending walk and has to fall as a whole.
        if (rest_alive) {
            if (!(rest <= (limit - kNucleusDoubt) * whole)) return false;
            top_p_margin = fabs(rest / whole - limit);
        }
        cut_bin = ranges.find<false>(need, before);
        if (cut_bin > 255u) return false;
        // ---- 3. its entries look at one another ---------------------------------------------------------------------------------
        for (int first = warp * 32; first < n; first += kMergeThreads) {
            const int e = first + lane;
            const bool on = e < n && bin_of(s_x[e]) == cut_bin;
            const uint32_t takers = __ballot_sync(0xFFFFFFFFu, on);
            if (takers == 0) continue;
            int at = 0;
            if (lane == 0) at = atomicAdd(&s_cut_n, __popc(takers));
            at = __shfl_sync(0xFFFFFFFFu, at, 0) + __popc(takers & below);
            if (on && at < kListCap) s_list[at] = make_ulonglong2(((u64)ordered_key(s_x[e]) << 32) | s_col[e], s_unit[e]);
        }
        __syncthreads();
        PSX_MERGE_STAGE(5);
        const int cut_n = s_cut_n;
        if (cut_n > kListCap) return false;
        for (int e = tid; e < cut_n; e += kMergeThreads) {
            const ulonglong2 me = s_list[e];
            u64 after = before;
#pragma unroll 4
            for (int i = 0; i < cut_n; ++i) {
                const ulonglong2 other = s_list[i];
                after += other.x > me.x ? other.y : 0;
            }
            // the last one down that stays (the last of the walk always does)
            if (((double)after < need || after == 0) && (double)(after + me.y) >= need) {
                const double above = after == 0 ? INFINITY : need - (double)after, under = (double)(after + me.y) - need;
                const double margin = fmin(above, under) * 0x1p-40;
                if (margin >= kNucleusDoubt * whole) {
                    s_cut_key = me.x;
                    s_margin = (u64)__double_as_longlong(margin / whole);
                }
            }
        }
        __syncthreads();
        PSX_MERGE_STAGE(6);
        cut_key = s_cut_key;
        if (cut_key == ~0ull) return false;
        top_p_margin = fmin(top_p_margin, __longlong_as_double((long long)s_margin));
    } else if (rest_alive) {  // what is outside has to fall to the min-p
        if (!(min_p > 0.0 && exp((double)x_low - (double)x_max) < min_p - kDoubt)) return false;
    }
    // ---- 4. the masses of those that stay, by column --------------------------------------------------------------------------
    const int col_shift = max(0, 24 - __clz((uint32_t)(p.vocab - 1)));
    auto stays = [&](int e) {  // (s_doubt where the min-p cannot tell)
        if (top_p_on) {
            const float x = s_x[e];
            const uint32_t b = bin_of(x);
            if (b > cut_bin || (b == cut_bin && (((u64)ordered_key(x) << 32) | s_col[e]) < cut_key)) return false;
        }
        if (min_p > 0.0 && s_unit[e] < (1ull << 40)) {  // :104-111, against the first maximum's exp(0)
            const double mass = (double)s_unit[e] * 0x1p-40;
            if (fabs(mass - min_p) < kDoubt) s_doubt = 1;
            return mass >= min_p;
        }
        return true;
    };
    for (int e = tid; e < n; e += kMergeThreads) {
        if (!stays(e)) continue;
        if (p.survivor_cols != nullptr) {
            const int at = atomicAdd(&s_survivors, 1);
            if (at < p.survivor_cap) {
                p.survivor_cols[row * p.survivor_cap + at] = s_col[e];
                p.survivor_vals[row * p.survivor_cap + at] = s_x[e];
            }
        } else {
            add_units(s_by_column, s_col[e] >> col_shift, s_unit[e]);
            if (v.diag) atomicAdd(&s_survivors, 1);
        }
    }
    __syncthreads();
    PSX_MERGE_STAGE(7);
    if (s_doubt != 0) return false;
    if (p.survivor_cols != nullptr) {  // the surviving set itself (ProcessLogits)
        if (s_survivors > p.survivor_cap) return false;
        if (tid == 0) {
            p.survivor_counts[row] = (uint32_t)s_survivors;
            *v.status = PSX_ROW_OK;
        }
        return true;
    }
    // ---- 5. the draw (:140-152): the range of columns that holds u, then its entries one by one --------------------------------
    u64 before;
    const RangeSums columns(s_by_column);
    const double total = (double)columns.all, target = u * total;
    const uint32_t range = columns.find<true>(target, before);
    if (range > 255u) return false;
    for (int e = tid; e < n; e += kMergeThreads) {
        if ((s_col[e] >> col_shift) != range || !stays(e)) continue;
        const int at = atomicAdd(&s_draw_n, 1);
        if (at < kListCap) {
            s_list[at] = make_ulonglong2(s_col[e], s_unit[e]);
            s_raw[at] = s_l[e];
        }
    }
    __syncthreads();
    PSX_MERGE_STAGE(8);
    const int draw_n = s_draw_n;
    if (draw_n > kListCap) return false;
    for (int e = tid; e < draw_n; e += kMergeThreads) {
        const ulonglong2 me = s_list[e];
        u64 mine = before;
#pragma unroll 4
        for (int i = 0; i < draw_n; ++i) {
            const ulonglong2 other = s_list[i];
            mine += other.x < me.x ? other.y : 0;
        }
        const double lo = target - (double)mine, hi = (double)(mine + me.y) - target;
        if (lo < 0.0 || hi <= 0.0) continue;
        const double margin = mine == 0 ? hi : fmin(lo, hi);
        if (margin < kNucleusDoubt * total) continue;  // (nobody takes it: replayed)
        *v.status = PSX_ROW_OK;
        *v.token = (int64_t)me.x;
        *v.log_prob = (float)(((double)s_raw[e] - (double)j.raw_max) - log((double)sum_units * 0x1p-40 + s_tails));  // :133,156
        if (v.diag) *v.diag = psx_row_diag{n, s_survivors, margin / total, top_p_margin};
        s_decided = 1;
    }
    __syncthreads();
    PSX_MERGE_STAGE(9);
    return s_decided != 0;
}

enum ListKind { kListGreedy, kListTopK, kListNucleus };

// ready(): waits until the row's inputs are complete; what does not need them is done before.
template <int kKind, class Ready>
__device__ __forceinline__ bool list_row(const MergeParams& p, const int64_t row, const RowView& v, u64* dyn, Ready ready) {
    const int arena = kKind == kListTopK ? kTopKArena : kKind == kListNucleus ? kNucleusArena : 0;
    if (p.parts > 32 || p.dyn_bytes < arena || (kKind == kListGreedy && p.survivor_cols != nullptr)) {  // (a record per lane)
        ready();
        return false;
    }
    if (kKind == kListGreedy) return list_greedy(p, v, ready);
    if (kKind == kListTopK) return list_top_k(p, row, v, dyn, ready);
    return list_nucleus(p, row, v, dyn, ready);
}

}  // namespace survivor
}  // namespace psx
