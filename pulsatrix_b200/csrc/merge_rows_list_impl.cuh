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
// Latency bound: a few KB per row out of L2, then dependent steps by one block.  What counts is the number of instructions one
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
constexpr int kWideCap = 2048;       // candidates at or above the threshold, before the cut (top-k)
constexpr int kNucleusCap = 4096;    // the same without a top-k
constexpr double kDoubt = 1e-11;     // of the whole mass: well above 512 units of 2^-52
constexpr double kNucleusDoubt = 4e-9;  // the same for kNucleusCap units of 2^-40
constexpr int kTopKArena = kListCap * (16 + 8 + 4) + kWideCap * 12;
constexpr int kNucleusArena = kListCap * (16 + 4) + kNucleusCap * 12 + 4 * 256 * 4;

// sum over the warp of integers below 2^59, by two of the 32-bit reductions
__device__ __forceinline__ u64 warp_sum_units(u64 v) {
    const uint32_t lo = __reduce_add_sync(0xFFFFFFFFu, (uint32_t)v & 0x7FFFFFFu), hi = __reduce_add_sync(0xFFFFFFFFu, (uint32_t)(v >> 27));
    return (u64)lo + ((u64)hi << 27);
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

    __device__ __forceinline__ ChunkWalk(const MergeParams& p, const int64_t row)
        : lists(static_cast<const char*>(p.candidates) + row * p.cand_row_stride), stride(p.cand_part_stride), parts(p.parts), cap(p.part_cap),
          lane(threadIdx.x & 31) {
        const int warp = threadIdx.x >> 5;
        chunk = warp / parts;
        part = warp - chunk * parts;
        step_chunk = kListWarps / parts;
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

__device__ __forceinline__ void load_parts(const MergeParams& p, const int64_t row, PartsJoined& j) {
    const int lane = threadIdx.x & 31;
    j.mine.raw_tail = 0.0; j.mine.proc_tail = 0.0;
    j.mine.raw_max = -FLT_MAX; j.mine.y_max = -INFINITY; j.mine.thr = -INFINITY;
    j.mine.nonfinite = 0; j.mine.alive_tail = 0; j.mine.overflow = 0;
    j.count = 0;
    if (lane < p.parts) {
        j.mine = *reinterpret_cast<const PartStats*>(static_cast<const char*>(p.stats) + row * p.stats_row_stride + lane * p.stats_part_stride);
        j.count = *reinterpret_cast<const uint32_t*>(static_cast<const char*>(p.part_counts) + row * p.count_row_stride + lane * p.count_part_stride);
    }
}

// false: the row is not for this way (a list that ran out of slots)
__device__ __forceinline__ bool join_parts(const MergeParams& p, PartsJoined& j) {
    j.count = min(j.count, (uint32_t)p.part_cap);
    j.raw_max = warp_max(j.mine.raw_max);
    j.y_max = warp_max(j.mine.y_max);
    j.thr = warp_max(j.mine.thr);
    j.bad = __reduce_or_sync(0xFFFFFFFFu, (j.mine.nonfinite & 3u) | (j.mine.overflow ? 4u : 0u));
    j.tail_alive = __reduce_add_sync(0xFFFFFFFFu, j.mine.alive_tail);
    j.longest = __reduce_max_sync(0xFFFFFFFFu, j.count);
    return (j.bad & 4u) == 0;
}

// true: the row has a non-finite logit, a copy that did not arrive, or nothing left; its status is written
__device__ __forceinline__ bool settle_bad_row(const MergeParams& p, const int64_t row, const PartsJoined& j) {
    if (j.bad == 0 && j.y_max > -INFINITY) return false;
    if (threadIdx.x == 0) {
        p.tokens[row] = -1;
        p.log_probs[row] = 0.0f;
        p.row_status[row] = (j.bad & 2u) ? PSX_ROW_DEVICE_TIMEOUT : (j.bad & 1u) ? PSX_ROW_NON_FINITE : PSX_ROW_ALL_REMOVED;
        if (p.diag) p.diag[row] = psx_row_diag{0, 0, INFINITY, INFINITY};
    }
    return true;
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
    __device__ __forceinline__ double of_warp() const { return warp_sum(high + (double)low * exp2_of_minus_small(c_res)); }
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

__device__ __forceinline__ void barrier_of_half() { asm volatile("bar.sync 1, 128;" ::: "memory"); }  // the first four warps

// ---- greedy ----------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ bool list_greedy(const MergeParams& p, const int64_t row) {
    __shared__ double s_z[kListWarps];
    __shared__ u64 s_best[kListWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    PartsJoined j;
    uint2 c[4];
    uint32_t where[4];
    ChunkWalk walk(p, row);
    load_parts(p, row, j);
    walk.fetch(c, where);
    if (!join_parts(p, j)) return false;
    if (settle_bad_row(p, row, j)) return true;
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
    double sum = z.of_warp();
    if (warp == 0) sum += tails_of_parts(j);
    const uint32_t top = __reduce_max_sync(0xFFFFFFFFu, (uint32_t)(best >> 32));
    if ((uint32_t)(best >> 32) == top && (top != 0 || lane == 0)) s_best[warp] = best;  // (columns differ: one lane)
    if (lane == 0) s_z[warp] = sum;
    __syncthreads();
    PSX_MERGE_STAGE(4);
    if (threadIdx.x == 0) {
        best = s_best[0];
        sum = s_z[0];
#pragma unroll
        for (int w = 1; w < kListWarps; ++w) {
            best = s_best[w] > best ? s_best[w] : best;
            sum += s_z[w];
        }
        p.row_status[row] = PSX_ROW_OK;
        p.tokens[row] = (int64_t)(uint32_t)~(uint32_t)(best >> 32);
        p.log_probs[row] = (float)(((double)__uint_as_float((uint32_t)best) - (double)j.raw_max) - log(sum));  // src/generation.cpp:156
        if (p.diag) p.diag[row] = psx_row_diag{1, 1, INFINITY, INFINITY};
    }
    PSX_MERGE_STAGE(9);
    return true;
}

// ---- sampling under a top-k ------------------------------------------------------------------------------------------------
__device__ __forceinline__ bool list_top_k(const MergeParams& p, const int64_t row, u64* dyn) {
    ulonglong2* const s_list = reinterpret_cast<ulonglong2*>(dyn);       // (ordered value << 32) | column; units of 2^-52
    u64* const s_after = reinterpret_cast<u64*>(s_list + kListCap);
    float* const s_raw = reinterpret_cast<float*>(s_after + kListCap);
    u64* const s_wide = reinterpret_cast<u64*>(s_raw + kListCap);        // raw logit, column | flags
    float* const s_wide_y = reinterpret_cast<float*>(s_wide + kWideCap);
    __shared__ uint32_t s_hist[32];
    __shared__ double s_z[kListWarps], s_log_z;
    __shared__ u64 s_part[4], s_margin;
    __shared__ int s_wide_n, s_n, s_doubt, s_won, s_survivors;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t below = (1u << lane) - 1u;
    const bool apply_t = p.apply_temperature != 0;
    PartsJoined j;
    uint2 c[4];
    uint32_t where[4];
    ChunkWalk walk(p, row);
    load_parts(p, row, j);
    walk.fetch(c, where);
    const double u = p.uniforms ? p.uniforms[row] : 0.5;
    if (tid < 32) s_hist[tid] = 0;
    if (tid == 0) { s_wide_n = 0; s_n = 0; s_doubt = 0; s_won = 0; s_survivors = 0; s_margin = ~0ull; }
    const double power = exp_power_of_lane();
    __syncthreads();
    if (!join_parts(p, j)) return false;
    if (settle_bad_row(p, row, j)) return true;
    PSX_MERGE_STAGE(3);
    // ---- 1. what reaches the largest part threshold (that part alone has k logits which reach it), and its histogram -------
    const float keep_from = relax_threshold(j.thr, apply_t, p.temperature);
    float bin_scale = 0.0f;  // (any map from value to bin that never decreases as the value falls would do)
    if (j.y_max - keep_from > 0.0f && j.y_max - keep_from < INFINITY) bin_scale = __fdividef(31.5f, j.y_max - keep_from);
    auto bin_of = [&](float y) { return min(31, max(0, (int)__fmul_rn(__fsub_rn(j.y_max, y), bin_scale))); };
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
                if (((votes[q] >> lane) & 1u) && mine < kWideCap) {
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
    if (wide > kWideCap) return false;
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
    const float x_max = temper(j.y_max, apply_t, p.temperature);
    if (!(fabsf(x_max) < INFINITY)) return false;  // (quotients that overflow tie: merge_row's business)
    for (int first = warp * 32; first < wide; first += kMergeThreads) {
        const int e = first + lane;
        const u64 cand = e < wide ? s_wide[e] : 0;
        const float l = __uint_as_float((uint32_t)(cand >> 32)), y = e < wide ? s_wide_y[e] : -INFINITY;
        const float up = apply_t ? __fadd_rn(y, __fmaf_rn(fabsf(y), 0x1p-20f, __fmul_rn(p.temperature, 0x1p-146f))) : y;
        const bool on = e < wide && bin_of(up) <= cut;
        if (e < wide && !on) z.add_low(l);
        const uint32_t takers = __ballot_sync(0xFFFFFFFFu, on);
        if (takers == 0) continue;
        int at = 0;
        if (lane == 0) at = atomicAdd(&s_n, __popc(takers));
        const float x = temper(y, apply_t, p.temperature);
        const u64 units = (u64)__double2ull_rn(exp_to(x, x_max, on, power) * 0x1p52);
        z.high += exp_to(l, j.raw_max, on, power);
        at = __shfl_sync(0xFFFFFFFFu, at, 0) + __popc(takers & below);
        if (on && at < kListCap) {
            s_list[at] = make_ulonglong2(((u64)ordered_key(x) << 32) | (uint32_t)(cand & kColumnMask), units);
            s_raw[at] = l;
        }
    }
    {
        const double sum = z.of_warp();
        if (lane == 0) s_z[warp] = sum;
    }
    __syncthreads();
    PSX_MERGE_STAGE(5);
    const int n = s_n;
    if (n > kListCap || n == 0) return false;
    bool won = false;
    int won_entry = 0;
    double won_margin = 0.0;
    if (warp == kListWarps - 1) {
        // the logarithm for the log-probability, meanwhile
        double sum = tails_of_parts(j);
#pragma unroll
        for (int w = 0; w < kListWarps; ++w) sum += s_z[w];
        if (lane == 0) s_log_z = log(sum);
    } else if (warp < 4) {
        // ---- 3. every entry against all the others; T neighbouring threads share one -----------------------------------------
        int n_pad = 8;
        while (n_pad < n && n_pad < 128) n_pad <<= 1;
        const int shift = 7 - (31 - __clz(n_pad)), T = 1 << shift, slice = tid & (T - 1);
        u64 sum = 0;
        for (int e0 = 0; e0 < n; e0 += n_pad) {
            const int e = e0 + (tid >> shift);
            const ulonglong2 me = e < n ? s_list[e] : make_ulonglong2(~0ull, 0);
            uint32_t greater = 0;
            u64 after = 0;
#pragma unroll 4
            for (int i = slice; i < n; i += T) {
                const ulonglong2 other = s_list[i];
                greater += (uint32_t)(other.x >> 32) > (uint32_t)(me.x >> 32) ? 1u : 0u;
                after += other.x > me.x ? other.y : 0;  // later in the top-p walk: a larger value, or the same at a higher column
            }
            for (int o = T >> 1; o > 0; o >>= 1) {
                greater += __shfl_xor_sync(0xFFFFFFFFu, greater, o);
                after += __shfl_xor_sync(0xFFFFFFFFu, after, o);
            }
            const bool stays = e < n && (int64_t)greater < p.top_k;  // :80-88: the k-th value and its ties stay
            if (slice == 0 && e < n) {
                s_after[e] = stays ? after : ~0ull;
                sum += stays ? me.y : 0;
            }
        }
        sum = warp_sum_units(sum);
        if (lane == 0) s_part[warp] = sum;
        barrier_of_half();
        PSX_MERGE_STAGE(6);
        sum = s_part[0] + s_part[1] + s_part[2] + s_part[3];
        const double limit = 1.0 - (double)p.top_p, whole = (double)sum * 0x1p-52, min_p = (double)p.min_p;
        bool doubt = false;
        for (int e = tid; e < n; e += 128) {
            const u64 after = s_after[e], unit = s_list[e].y;
            bool stays = after != ~0ull;
            if (stays && p.top_p < 1.0f && after != 0) {  // :89-103; the last of the walk always stays
                const double beyond = (double)(sum - after) * 0x1p-52 - limit * whole;
                stays = beyond > 0.0;
                doubt = doubt || fabs(beyond) < kDoubt * whole;
                if (p.diag) atomicMin(&s_margin, (u64)__double_as_longlong(fabs(beyond) / whole));
            }
            if (stays && min_p > 0.0 && unit < (1ull << 52)) {  // :104-111, against the first maximum's exp(0)
                const double mass = (double)unit * 0x1p-52;
                stays = mass >= min_p;
                doubt = doubt || fabs(mass - min_p) < kDoubt;
            }
            s_after[e] = stays ? 1 : 0;
            if (p.diag && p.survivor_cols == nullptr && stays) atomicAdd(&s_survivors, 1);
        }
        if (doubt) s_doubt = 1;
        barrier_of_half();
        PSX_MERGE_STAGE(7);
        // ---- 4. the draw (:140-152): the entry whose share of the running sum, by ascending column, holds u --------------------
        if (p.survivor_cols == nullptr && s_doubt == 0) {
            for (int e0 = 0; e0 < n; e0 += n_pad) {
                const int e = e0 + (tid >> shift);
                const ulonglong2 me = e < n ? s_list[e] : make_ulonglong2(~0ull, 0);
                u64 before = 0, total = 0;
#pragma unroll 4
                for (int i = slice; i < n; i += T) {
                    const ulonglong2 other = s_list[i];
                    const u64 mass = s_after[i] != 0 ? other.y : 0;
                    total += mass;
                    before += (uint32_t)other.x < (uint32_t)me.x ? mass : 0;
                }
                for (int o = T >> 1; o > 0; o >>= 1) {
                    total += __shfl_xor_sync(0xFFFFFFFFu, total, o);
                    before += __shfl_xor_sync(0xFFFFFFFFu, before, o);
                }
                const double target = u * (double)total, lo = target - (double)before, hi = (double)(before + me.y) - target;
                if (e < n && slice == 0 && s_after[e] != 0 && lo >= 0.0 && hi > 0.0) {
                    const double margin = before == 0 ? hi : fmin(lo, hi);
                    if (margin >= kDoubt * (double)total) {  // (nobody takes it otherwise: replayed)
                        won = true;
                        won_entry = e;
                        won_margin = margin / (double)total;
                        s_won = 1;
                    }
                }
            }
        }
    }
    __syncthreads();
    PSX_MERGE_STAGE(8);
    if (p.survivor_cols != nullptr) {  // the surviving set itself (ProcessLogits)
        if (s_doubt != 0 || n > p.survivor_cap) return false;
        for (int e = tid; e < n; e += kMergeThreads) {
            if (s_after[e] == 0) continue;
            const int64_t at = row * p.survivor_cap + atomicAdd(&s_survivors, 1);
            p.survivor_cols[at] = (uint32_t)s_list[e].x;
            p.survivor_vals[at] = from_ordered_key((uint32_t)(s_list[e].x >> 32));
        }
        __syncthreads();
        if (tid == 0) {
            p.survivor_counts[row] = (uint32_t)s_survivors;
            p.row_status[row] = PSX_ROW_OK;
        }
        return true;
    }
    if (won) {
        p.row_status[row] = PSX_ROW_OK;
        p.tokens[row] = (int64_t)(uint32_t)s_list[won_entry].x;
        p.log_probs[row] = (float)(((double)s_raw[won_entry] - (double)j.raw_max) - s_log_z);  // :133,156
        if (p.diag) {
            const double top_p_margin = s_margin == ~0ull ? (double)INFINITY : __longlong_as_double((long long)s_margin);
            p.diag[row] = psx_row_diag{n, s_survivors, won_margin, top_p_margin};
        }
    }
    PSX_MERGE_STAGE(9);
    return s_won != 0;
}

// ---- sampling without a top-k ----------------------------------------------------------------------------------------------
// Masses by range: 256 sums of units of 2^-40, as 20 low and 21 high bits in two words (4096 of either fit 32 bits).
__device__ __forceinline__ void add_units(uint32_t* hist, uint32_t bin, u64 units) {
    atomicAdd(&hist[bin], (uint32_t)units & 0xFFFFFu);
    atomicAdd(&hist[256 + bin], (uint32_t)(units >> 20));
}
// The range in which the running sum over the ranges reaches `level` (a level of 0 and below: the first), by a whole warp: its
// index (256: none does), the sum before it and with it; and the sum of all.
__device__ __forceinline__ uint32_t find_range(const uint32_t* hist, double level, bool beyond, u64& before, u64& upto, u64& all) {
    const int lane = threadIdx.x & 31;
    u64 run[8], sum = 0;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const uint4 lo = reinterpret_cast<const uint4*>(hist)[2 * lane + half], hi = reinterpret_cast<const uint4*>(hist + 256)[2 * lane + half];
        run[4 * half + 0] = sum += lo.x + ((u64)hi.x << 20);
        run[4 * half + 1] = sum += lo.y + ((u64)hi.y << 20);
        run[4 * half + 2] = sum += lo.z + ((u64)hi.z << 20);
        run[4 * half + 3] = sum += lo.w + ((u64)hi.w << 20);
    }
    u64 incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const u64 up = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += up;
    }
    all = __shfl_sync(0xFFFFFFFFu, incl, 31);
    const u64 lead = incl - sum;
    uint32_t short_of = 0;
    u64 last = lead, hit = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const double reach = (double)(lead + run[q]);
        const bool reached = beyond ? reach > level : reach >= level;  // (`beyond`: has to go past it)
        if (!reached) { ++short_of; last = lead + run[q]; }
        if (reached && hit == 0) hit = lead + run[q] + 1;
    }
    const uint32_t lanes = __ballot_sync(0xFFFFFFFFu, short_of < 8);
    if (lanes == 0) { before = upto = all; return 256u; }
    const int src = __ffs(lanes) - 1;
    before = __shfl_sync(0xFFFFFFFFu, last, src);
    upto = __shfl_sync(0xFFFFFFFFu, hit, src) - 1;
    return 8u * src + __shfl_sync(0xFFFFFFFFu, short_of, src);
}

__device__ __forceinline__ bool list_nucleus(const MergeParams& p, const int64_t row, u64* dyn) {
    ulonglong2* const s_list = reinterpret_cast<ulonglong2*>(dyn);
    float* const s_raw = reinterpret_cast<float*>(s_list + kListCap);
    uint32_t* const s_by_value = reinterpret_cast<uint32_t*>(s_raw + kListCap);  // masses over 256 ranges of the value
    uint32_t* const s_by_column = s_by_value + 512;                              // ... and of the column
    float* const s_l = reinterpret_cast<float*>(s_by_column + 512);
    float* const s_x = s_l + kNucleusCap;
    uint32_t* const s_col = reinterpret_cast<uint32_t*>(s_x + kNucleusCap);
    __shared__ double s_z[kListWarps], s_rest[kListWarps];
    __shared__ u64 s_cut_key, s_margin;
    __shared__ uint32_t s_dropped[kListWarps];
    __shared__ int s_n, s_cut_n, s_draw_n, s_decided, s_survivors, s_doubt;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t below = (1u << lane) - 1u;
    const bool apply_t = p.apply_temperature != 0;
    PartsJoined j;
    uint2 c[4];
    uint32_t where[4];
    ChunkWalk walk(p, row);
    load_parts(p, row, j);
    walk.fetch(c, where);
    const double u = p.uniforms ? p.uniforms[row] : 0.5;
    reinterpret_cast<uint4*>(s_by_value)[tid] = make_uint4(0, 0, 0, 0);  // both histograms
    if (tid == 0) { s_n = 0; s_cut_n = 0; s_draw_n = 0; s_decided = 0; s_survivors = 0; s_doubt = 0; s_cut_key = ~0ull; s_margin = ~0ull; }
    const double power = exp_power_of_lane();
    __syncthreads();
    if (!join_parts(p, j)) return false;
    if (settle_bad_row(p, row, j)) return true;
    PSX_MERGE_STAGE(3);
    // ---- 1. candidates at or above the largest part threshold into shared memory, their masses by value; what lies below it
    // belongs to the rest of the vocabulary, which the candidates do not cover ---------------------------------------------------
    const float x_max = temper(j.y_max, apply_t, p.temperature);
    if (!(fabsf(x_max) < INFINITY)) return false;  // (quotients that overflow tie: merge_row's business)
    const float keep_from = relax_threshold(j.thr, apply_t, p.temperature);
    const float x_low = temper(keep_from, apply_t, p.temperature);
    float bin_scale = 0.0f;
    if (x_max - x_low > 0.0f && x_max - x_low < INFINITY) bin_scale = __fdiv_rn(255.0f, x_max - x_low);
    auto bin_of = [&](float x) { return (uint32_t)max(0, min(255, (int)__fmul_rn(__fsub_rn(x_max, x), bin_scale))); };
    RawSum z(j.raw_max);
    double rest = 0.0;
    uint32_t dropped = 0;
    for (;;) {
        uint2 next[4];
        uint32_t where_next[4];
        const bool last = walk.beyond(j.longest);
        if (!last) walk.fetch(next, where_next);
        float x[4];
        uint32_t votes[4];
        int all = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t here = __shfl_sync(0xFFFFFFFFu, j.count, where[q] & 255u);
            const bool there = (where[q] >> 8) + lane < here;
            const float l = __uint_as_float(c[q].x);
            float y = there ? l : -INFINITY;
            if (there && (c[q].y & ~kColumnMask) != 0) y = processed_before_temperature(l, c[q].y, p.penalty);
            x[q] = temper(y, apply_t, p.temperature);
            const bool on = y >= keep_from;
            votes[q] = __ballot_sync(0xFFFFFFFFu, on);
            if (!__any_sync(0xFFFFFFFFu, there)) continue;
            const double mass = exp_to(x[q], x_max, y > -INFINITY, power);
            if (there && !on) {
                z.add_low(l);
                rest += mass;
                dropped += y > -INFINITY ? 1u : 0u;
            }
            if (votes[q] == 0) continue;
            z.high += exp_to(l, j.raw_max, on, power);
            if (on) add_units(s_by_value, bin_of(x[q]), (u64)__double2ull_rn(mass * 0x1p40));
            all += __popc(votes[q]);
        }
        if (all != 0) {
            int at = 0;
            if (lane == 0) at = atomicAdd(&s_n, all);
            at = __shfl_sync(0xFFFFFFFFu, at, 0);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int mine = at + __popc(votes[q] & below);
                if (((votes[q] >> lane) & 1u) && mine < kNucleusCap) {
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
        double sum = z.of_warp();
        if (warp == 0) {
            sum += tails_of_parts(j);
            if (j.mine.y_max > -INFINITY && j.mine.proc_tail > 0.0) {
                rest += j.mine.proc_tail * exp((double)temper(j.mine.y_max, apply_t, p.temperature) - (double)x_max);
            }
        }
        rest = warp_sum(rest);
        dropped = __reduce_add_sync(0xFFFFFFFFu, dropped);
        if (lane == 0) { s_z[warp] = sum; s_rest[warp] = rest; s_dropped[warp] = dropped; }
    }
    __syncthreads();
    PSX_MERGE_STAGE(4);
    const int n = s_n;
    if (n > kNucleusCap || n == 0) return false;
    rest = s_rest[0];
    double sum_exp = s_z[0];
    u64 outside = j.tail_alive + s_dropped[0];
#pragma unroll
    for (int w = 1; w < kListWarps; ++w) { rest += s_rest[w]; outside += s_dropped[w]; sum_exp += s_z[w]; }
    // ---- 2. the top-p (:89-103): the range that its level falls into ---------------------------------------------------------
    const double limit = 1.0 - (double)p.top_p, min_p = (double)p.min_p;
    const bool top_p_on = p.top_p < 1.0f, rest_alive = outside != 0;
    uint32_t cut_bin = 256u;
    double top_p_margin = INFINITY;
    u64 cut_key = 0;
    if (top_p_on) {
        u64 before, upto, all = 0;
        for (int i = lane; i < 256; i += 32) all += s_by_value[i] + ((u64)s_by_value[256 + i] << 20);
        all = warp_sum_units(all);
        const double listed = (double)all * 0x1p-40, whole = listed + (rest_alive ? rest : 0.0);
        const double need = (whole - limit * whole) * 0x1p40;  // an entry stays while what comes after it is less
        // Everything outside the list leads the ascending walk and has to fall as a whole.
        if (rest_alive) {
            if (!(rest <= (limit - kNucleusDoubt) * whole)) return false;
            top_p_margin = fabs(rest / whole - limit);
        }
        cut_bin = find_range(s_by_value, need, false, before, upto, all);
        if (cut_bin > 255u) return false;
        // ---- 3. its entries look at one another ---------------------------------------------------------------------------------
        for (int first = warp * 32; first < n; first += kMergeThreads) {
            const int e = first + lane;
            const bool on = e < n && bin_of(s_x[e]) == cut_bin;
            const uint32_t takers = __ballot_sync(0xFFFFFFFFu, on);
            if (takers == 0) continue;
            int at = 0;
            if (lane == 0) at = atomicAdd(&s_cut_n, __popc(takers));
            const float x = on ? s_x[e] : 0.0f;
            const u64 units = (u64)__double2ull_rn(exp_to(x, x_max, on, power) * 0x1p40);
            at = __shfl_sync(0xFFFFFFFFu, at, 0) + __popc(takers & below);
            if (on && at < kListCap) s_list[at] = make_ulonglong2(((u64)ordered_key(x) << 32) | s_col[e], units);
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
    auto stays_of = [&](int e, u64& units) {  // by a whole warp; s_doubt where the min-p cannot tell
        const float x = e < n ? s_x[e] : -INFINITY;
        bool stays = e < n;
        if (top_p_on && stays) {
            const uint32_t b = bin_of(x);
            stays = b < cut_bin || (b == cut_bin && (((u64)ordered_key(x) << 32) | s_col[e]) >= cut_key);
        }
        const double mass = exp_to(x, x_max, stays, power);
        if (min_p > 0.0 && stays && x < x_max) {  // :104-111, against the first maximum's exp(0)
            if (fabs(mass - min_p) < kDoubt) s_doubt = 1;
            stays = mass >= min_p;
        }
        units = stays ? (u64)__double2ull_rn(mass * 0x1p40) : 0;
        return stays;
    };
    for (int first = warp * 32; first < n; first += kMergeThreads) {
        const int e = first + lane;
        u64 units;
        const bool stays = stays_of(e, units);
        if (p.survivor_cols != nullptr) {
            if (stays) {
                const int at = atomicAdd(&s_survivors, 1);
                if (at < p.survivor_cap) {
                    p.survivor_cols[row * p.survivor_cap + at] = s_col[e];
                    p.survivor_vals[row * p.survivor_cap + at] = s_x[e];
                }
            }
        } else {
            if (units != 0) add_units(s_by_column, s_col[e] >> col_shift, units);
            if (p.diag && stays) atomicAdd(&s_survivors, 1);
        }
    }
    __syncthreads();
    PSX_MERGE_STAGE(7);
    if (s_doubt != 0) return false;
    if (p.survivor_cols != nullptr) {  // the surviving set itself (ProcessLogits)
        if (s_survivors > p.survivor_cap) return false;
        if (tid == 0) {
            p.survivor_counts[row] = (uint32_t)s_survivors;
            p.row_status[row] = PSX_ROW_OK;
        }
        return true;
    }
    // ---- 5. the draw (:140-152): the range of columns that holds u, then its entries one by one --------------------------------
    u64 before, upto, total = 0;
    for (int i = lane; i < 256; i += 32) total += s_by_column[i] + ((u64)s_by_column[256 + i] << 20);
    total = warp_sum_units(total);
    const double target = u * (double)total;
    const uint32_t range = find_range(s_by_column, target, true, before, upto, total);
    if (range > 255u) return false;
    for (int first = warp * 32; first < n; first += kMergeThreads) {
        const int e = first + lane;
        const bool near = e < n && (s_col[e] >> col_shift) == range;
        if (!__any_sync(0xFFFFFFFFu, near)) continue;
        u64 units;
        const bool stays = stays_of(near ? e : n, units);
        const uint32_t takers = __ballot_sync(0xFFFFFFFFu, stays);
        if (takers == 0) continue;
        int at = 0;
        if (lane == 0) at = atomicAdd(&s_draw_n, __popc(takers));
        at = __shfl_sync(0xFFFFFFFFu, at, 0) + __popc(takers & below);
        if (stays && at < kListCap) {
            s_list[at] = make_ulonglong2(s_col[e], units);
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
        if (margin < kNucleusDoubt * (double)total) continue;  // (nobody takes it: replayed)
        p.row_status[row] = PSX_ROW_OK;
        p.tokens[row] = (int64_t)me.x;
        p.log_probs[row] = (float)(((double)s_raw[e] - (double)j.raw_max) - log(sum_exp));  // :133,156
        if (p.diag) p.diag[row] = psx_row_diag{n, s_survivors, margin / (double)total, top_p_margin};
        s_decided = 1;
    }
    __syncthreads();
    PSX_MERGE_STAGE(9);
    return s_decided != 0;
}

enum ListKind { kListGreedy, kListTopK, kListNucleus };

template <int kKind>
__device__ __forceinline__ bool list_row(const MergeParams& p, const int64_t row, u64* dyn) {
    if (p.parts > 32) return false;  // (a record per lane)
    if (kKind == kListGreedy) return p.survivor_cols == nullptr && list_greedy(p, row);
    if (kKind == kListTopK) return p.dyn_bytes >= kTopKArena && list_top_k(p, row, dyn);
    return p.dyn_bytes >= kNucleusArena && list_nucleus(p, row, dyn);
}

}  // namespace survivor
}  // namespace psx
