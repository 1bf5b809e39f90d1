// Sampling from the whole distribution: no top-k, no top-p, no min-p (src/generation.cpp:123-156 with the filters
// off -- the penalty, the EOS ban and the temperature may be on).  Every token can be drawn, so there is no short
// list of candidates; what the draw needs is the mass of every run of columns, then the columns of one run.
//
//   1. weigh_segments_kernel reads every logit once.  A warp takes a segment of 512 columns into registers, finds its
//      two maxima (raw and processed) and sums exp() of both in double precision; it reports 32 bytes.  The warps of a
//      CTA share a bitmap of the history and a table of powers, nothing else.
//   2. draw_token_kernel, one CTA per row: the segments' masses brought to the row's maximum, their running sum
//      against u times the whole (the inverse-CDF walk of :140-152 in steps of a segment), then the logits of the one
//      segment that holds the crossing, column by column.
//
// Sums are in double precision in a fixed order (the same input gives the same bits); they differ from the
// reference's sequential sums by rounding only, and a draw closer than that to an edge shows in draw_margin.
//
// Bound: 4 bytes per logit from HBM, and two double-precision exponentials per logit (one when the processed row is
// the raw one).  The double-precision pipe (64 lanes per SM) is the longer of the two -- about 17 operations per logit
// against 4 bytes are 1.35 : 1 -- which is why the exponential is the table one (psx_exp.cuh).  A segment is a warp's:
// 512 columns keep 16 logits per lane in registers, so that the maximum is known before the first exponential and
// nothing is rescaled, and one row of 50 K columns still gives 98 warps to spread over the SMs.
#include "whole_rows.cuh"

#include <algorithm>

#include "../../include/psx_b200.h"
#include "psx_exp.cuh"

namespace psx {

namespace {

constexpr int kThreads = 256;
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
// vocabulary are ignored -- their bits stand for no column of the row).  By the whole block.
__device__ __forceinline__ void mark_columns(const int64_t* ids, int64_t begin, int64_t end, int64_t first, int slots, int64_t vocab,
                                             uint32_t* bits) {
    for (int64_t i = begin + threadIdx.x; i < end; i += kThreads) {
        const int64_t id = ids[i];
        const uint64_t at = (uint64_t)(id - first);
        if (at < (uint64_t)slots && (uint64_t)id < (uint64_t)vocab) atomicOr(&bits[at >> 5], 1u << (at & 31));
    }
}

// The processed logit (:59-79).
__device__ __forceinline__ float processed(float l, bool flagged, bool banned, const WholeRowParams& p) {
    float y = l;
    if (flagged) y = penalize(l, p.penalty);
    if (banned) y = -INFINITY;
    return temper(y, p.apply_temperature != 0, p.temperature);
}

// kPlain: the processed row is the raw row (no penalty, no ban, no temperature).
template <bool kPlain>
__global__ void __launch_bounds__(kThreads) weigh_segments_kernel(const WholeRowParams p) {
    __shared__ double s_table[kExpTable];
    __shared__ uint32_t s_flag[kMostPerWarp * kWarps * kSegmentCols / 32], s_ban[kMostPerWarp * kWarps * kSegmentCols / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t row = (int64_t)blockIdx.z * 65535 + blockIdx.y;
    const bool ends_the_grid = !p.wait_before_writes && blockIdx.x == gridDim.x - 1 && blockIdx.y == gridDim.y - 1 && blockIdx.z == gridDim.z - 1;
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
    load(first_segment + warp);  // (under the table and the bitmap)
    load_exp_table(s_table);
    const bool penalise = !kPlain && p.history_ids != nullptr, flags = penalise || (!kPlain && p.num_banned > 0);
    const int64_t first_col = (int64_t)first_segment * kSegmentCols - w.misalign;
    const int slots = per_warp * kWarps * kSegmentCols;
    if (flags) {
        for (int i = threadIdx.x; i < slots / 32; i += kThreads) s_flag[i] = s_ban[i] = 0u;
        __syncthreads();
        if (penalise) mark_columns(p.history_ids, p.history_offsets[row], p.history_offsets[row + 1], first_col, slots, p.vocab, s_flag);
        mark_columns(p.banned_ids, 0, p.num_banned, first_col, slots, p.vocab, s_ban);
    }
    __syncthreads();
    if (p.inputs_ready && p.wait_before_writes) grid_dependency_wait();
#pragma unroll 1
    for (int turn = 0; turn < per_warp; ++turn) {
        const int local = turn * kWarps + warp, segment = first_segment + local;
        if (segment >= p.segments) break;
        if (turn > 0) load(segment);
        float raw_max = -INFINITY, y_max = -INFINITY;
        bool bad = false;
        uint32_t alive = 0;
        float l[kVecs * 4], y[kVecs * 4];
#pragma unroll
        for (int k = 0; k < kVecs; ++k) {
            const float c4[4] = {d[k].x, d[k].y, d[k].z, d[k].w};
            const int v = k * 32 + lane;  // within the segment
            uint32_t flag4 = 0, ban4 = 0;
            if (flags) {
                const int word = (local * kSegmentVecs + v) >> 3, shift = (v & 7) * 4;
                flag4 = s_flag[word] >> shift;
                ban4 = s_ban[word] >> shift;
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int col = (segment * kSegmentVecs + v) * 4 + c - w.misalign;
                const bool here = (uint32_t)col < (uint32_t)p.vocab;
                bad = bad || (here && !(fabsf(c4[c]) < INFINITY));
                l[4 * k + c] = here ? c4[c] : -INFINITY;
                raw_max = fmaxf(raw_max, l[4 * k + c]);
                if (!kPlain) {
                    y[4 * k + c] = processed(l[4 * k + c], (flag4 >> c) & 1u, (ban4 >> c) & 1u, p);
                    y_max = fmaxf(y_max, y[4 * k + c]);
                    alive += y[4 * k + c] > -INFINITY ? 1u : 0u;
                } else {
                    alive += here ? 1u : 0u;
                }
            }
        }
        raw_max = warp_max(raw_max);
        y_max = kPlain ? raw_max : warp_max(y_max);
        const double raw_top = double_of_float(raw_max), y_top = double_of_float(y_max);
        double raw_sum = 0.0, mass = 0.0;
#pragma unroll
        for (int i = 0; i < kVecs * 4; ++i) {
            raw_sum += exp_below(l[i], double_of_float(l[i]), raw_max, raw_top, s_table);
            if (!kPlain) mass += exp_below(y[i], double_of_float(y[i]), y_max, y_top, s_table);
        }
        raw_sum = warp_sum(raw_sum);
        mass = kPlain ? raw_sum : warp_sum(mass);
        alive = __reduce_add_sync(0xFFFFFFFFu, alive);
        const bool any_bad = __any_sync(0xFFFFFFFFu, bad);
        if (lane == 0) {
            SegmentStats s;
            s.raw_sum = raw_sum;  // (a segment past the end of its row: maxima of -inf, sums of nothing)
            s.mass = mass;
            s.raw_max = raw_max;
            s.y_max = y_max;
            s.alive = alive;
            s.nonfinite = any_bad ? 1u : 0u;
            p.stats[row * p.segments + segment] = s;
        }
    }
    if (ends_the_grid) grid_dependency_wait();
}

// Inclusive running sum over the block in thread order; `total` is the whole.
__device__ __forceinline__ double block_running_sum(double v, double* scratch, double& total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double up = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if (lane >= o) v += up;
    }
    __syncthreads();
    if (lane == 31) scratch[warp] = v;
    __syncthreads();
    double before = 0.0;
    total = 0.0;
#pragma unroll
    for (int i = 0; i < kWarps; ++i) {
        if (i < warp) before += scratch[i];
        total += scratch[i];
    }
    return before + v;
}

__global__ void __launch_bounds__(kThreads) draw_token_kernel(const WholeRowParams p) {
    __shared__ double s_table[kExpTable], s_scratch[kWarps];
    __shared__ double s_before;
    __shared__ int s_segment, s_last, s_chosen, s_hit, s_any_alive;
    __shared__ float s_max[2][kWarps];
    __shared__ uint32_t s_flag[kSegmentCols / 32], s_ban[kSegmentCols / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t row = blockIdx.x;
    load_exp_table(s_table);
    if (tid == 0) { s_segment = 0x7FFFFFFF; s_last = -1; s_chosen = 0x7FFFFFFF; s_hit = -1; }
    if (tid < kSegmentCols / 32) s_flag[tid] = s_ban[tid] = 0u;
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
    float raw_max = mine.raw_max, y_max = mine.y_max;
    uint32_t bad = mine.nonfinite;
    for (int s = begin + 1; s < end; ++s) {
        raw_max = fmaxf(raw_max, stats[s].raw_max);
        y_max = fmaxf(y_max, stats[s].y_max);
        bad |= stats[s].nonfinite;
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
    const double y_top = double_of_float(y_max), raw_top = double_of_float(raw_max);
    auto share = [&](double sum, float top, float row_top, double row_top_d) {
        return sum > 0.0 ? sum * exp_below(top, double_of_float(top), row_top, row_top_d, s_table) : 0.0;
    };
    double mass = 0.0, z = 0.0;
    int alive = 0;
    for (int s = begin; s < end; ++s) {
        if (s > begin) mine = stats[s];
        mass += share(mine.mass, mine.y_max, y_max, y_top);
        z += share(mine.raw_sum, mine.raw_max, raw_max, raw_top);
        alive += (int)mine.alive;
    }
    double total, z_total;
    const double upto = block_running_sum(mass, s_scratch, total);
    block_running_sum(z, s_scratch, z_total);
    const double u = p.uniforms[row], target = u * total;
    // ---- the segment that holds the crossing: the first whose running sum rises above the target (:140-152); if
    // rounding leaves none, the last that holds mass -----------------------------------------------------------------
    if (mass > 0.0) {
        if (upto > target) atomicMin(&s_segment, begin);
        atomicMax(&s_last, begin);
    }
    __syncthreads();
    const int owner_begin = s_segment != 0x7FFFFFFF ? s_segment : s_last;
    if (begin == owner_begin && mass > 0.0) {
        double at = upto - mass, before = at;
        int found = begin;
        for (int s = begin; s < end; ++s) {
            if (end - begin > 1) mine = stats[s];
            const double share_of = end - begin > 1 ? share(mine.mass, mine.y_max, y_max, y_top) : mass;
            if (share_of > 0.0) { found = s; before = at; }
            at += share_of;
            if (share_of > 0.0 && at > target) break;
        }
        s_hit = found;
        s_before = before;
    }
    __syncthreads();
    const int segment = s_hit;
    const double before_segment = s_before;
    // ---- its columns, in order: thread t has columns 2t and 2t + 1 of the segment --------------------------------------
    const RowWindow w = row_window(p, row);
    const int64_t first_col = (int64_t)segment * kSegmentCols - w.misalign;
    static_assert(kSegmentCols == 2 * kThreads, "two columns per thread");
    float l[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const int64_t col = first_col + 2 * tid + c;
        l[c] = col >= 0 && col < p.vocab ? p.logits[row * p.row_stride + col] : -INFINITY;
    }
    if (p.history_ids != nullptr) {
        mark_columns(p.history_ids, p.history_offsets[row], p.history_offsets[row + 1], first_col, kSegmentCols, p.vocab, s_flag);
    }
    mark_columns(p.banned_ids, 0, p.num_banned, first_col, kSegmentCols, p.vocab, s_ban);
    __syncthreads();
    double e[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const int at = 2 * tid + c;
        const float y = processed(l[c], (s_flag[at >> 5] >> (at & 31)) & 1u, (s_ban[at >> 5] >> (at & 31)) & 1u, p);
        e[c] = y > -INFINITY ? exp_below(y, double_of_float(y), y_max, y_top, s_table) : 0.0;
    }
    double unused;
    const double run = before_segment + block_running_sum(e[0] + e[1], s_scratch, unused);
    const double run_first = run - e[1];  // up to this thread's first column
    if (tid == 0) s_last = -1;
    __syncthreads();
    if (e[1] > 0.0) {
        if (run > target) atomicMin(&s_chosen, 2 * tid + 1);
        atomicMax(&s_last, 2 * tid + 1);
    }
    if (e[0] > 0.0) {
        if (run_first > target) atomicMin(&s_chosen, 2 * tid);
        atomicMax(&s_last, 2 * tid);
    }
    __syncthreads();
    const int chosen = s_chosen != 0x7FFFFFFF ? s_chosen : s_last;
    if (p.diag) {
        alive = (int)__reduce_add_sync(0xFFFFFFFFu, (uint32_t)alive);
        __syncthreads();
        if (tid == 0) s_any_alive = 0;
        __syncthreads();
        if (lane == 0) atomicAdd(&s_any_alive, alive);
        __syncthreads();
    }
    if (chosen >> 1 == tid) {
        const int c = chosen & 1;
        p.row_status[row] = PSX_ROW_OK;
        p.tokens[row] = first_col + chosen;
        // the unprocessed log-softmax (:133,156)
        p.log_probs[row] = (float)log(exp((double)l[c] - (double)raw_max) / z_total);
        if (p.diag) {
            const double hi = (c ? run : run_first) / total, lo = ((c ? run_first : run_first - e[0])) / total;
            const double margin = lo <= 0.0 ? fabs(u - hi) : fmin(fabs(u - lo), fabs(u - hi));
            p.diag[row] = psx_row_diag{(int)p.vocab, s_any_alive, margin, INFINITY};
        }
    }
}

}  // namespace

cudaError_t launch_whole_rows(const WholeRowParams& p, cudaStream_t stream) {
    if (p.rows <= 0) return cudaSuccess;
    if (p.rows > 65535ll * 65535ll || p.rows > 0x7FFFFFFFll) return cudaErrorInvalidConfiguration;
    // One segment per warp while that leaves the GPU short of warps; up to four, which share a CTA's table and
    // bitmap, once there are some six thousand warps' worth (148 SMs x 40 warps).
    const int64_t warps = p.rows * p.segments;
    WholeRowParams q = p;
    q.segments_per_warp = (int)std::max<int64_t>(1, std::min<int64_t>(kMostPerWarp, warps / 6000));
    const int64_t per_cta = (int64_t)kWarps * q.segments_per_warp;
    const dim3 grid((unsigned)((p.segments + per_cta - 1) / per_cta), (unsigned)std::min<int64_t>(p.rows, 65535),
                    (unsigned)((p.rows + 65534) / 65535));
    const bool plain = p.history_ids == nullptr && p.num_banned == 0 && !p.apply_temperature;
    const cudaError_t e = launch_overlapping(plain ? weigh_segments_kernel<true> : weigh_segments_kernel<false>, grid, dim3(kThreads), 0,
                                           stream, q);
    if (e != cudaSuccess) return e;
    return launch_overlapping(draw_token_kernel, dim3((unsigned)p.rows), dim3(kThreads), 0, stream, q);
}

}  // namespace psx
