// top_k_rows: the k best entries of every row in rank order, with their columns as floats.
//
// A row belongs to a thread-block cluster of 1, 2, 4 or 8 CTAs (by its length), a slice of the
// row per CTA.  Entries are compared as order-preserving keys: NaN above every number,
// -0.0 == +0.0, `largest == 0` mirrors the order.
//
// The short way (k <= 256): two sweeps over the slice as floats, out of shared memory where a slice of
// up to 16,384 entries fits (bulk copies; longer ones are read from global memory twice, the second time out of L2).
// Bound by instructions more than by HBM: 4096 x 16,384, k 64: 79.7 us with 256 threads reading twice from global memory,
// 67.9 now; 8192 x 4096, k 16: 63.5 -> 34.8 us.  Sweep one notes every thread's best entry; the smallest over the warps of
// the kp-th best of those (kp = ceil(k / 8)) is a bound that k entries of the slice reach.  Sweep
// two lists what reaches the bound, usually k and a few; the list is put in rank order by
// counting (a long one by sorting), and with several CTAs per row the best k of each meet in the first CTA's shared memory
// (distributed shared memory, two cluster barriers), where each finds its place in the others' lists by bisection.
//
// The long way (larger k, or a list that overflowed: thousands of ties): the slice becomes keys in
// shared memory (or is swept where the short way holds it, or from global memory when it does not fit), and
//   1. a 4 x 8-bit radix select finds the k-th key: every CTA counts its slice's digits into a
//      histogram of its own, the cluster meets, and every CTA adds the cluster's histograms up
//      through distributed shared memory for itself;
//   2. when more entries tie with the k-th key than are wanted, a second radix select, over the
//      columns of the tying entries, finds the column up to which they are taken (the reference
//      keeps the lowest columns, src/top_k_math.hpp:19-47);
//   3. the entries above the k-th key and the chosen ties are collected in the first CTA's shared
//      memory (remote atomics and stores) and sorted there by (key, ~column) -- rank order, equal
//      values by ascending column.
// The values written are copied from the input, so that their bits (the sign of zero, NaN
// payloads) are the input's.  Pure selection: nothing is computed, so the result equals the host
// reference bit for bit.
#include <cooperative_groups.h>

#include "psx_async.cuh"
#include "scan_rows.cuh"
#include "topk_rows.cuh"

namespace cg = cooperative_groups;

namespace psx {

namespace {

using u64 = unsigned long long;
constexpr int kWidest = 256;  // threads of a CTA at most
constexpr int kSliceMax = 48 * 1024;  // keys one CTA keeps in shared memory (192 KB)
// A list from which sorting it takes fewer steps than looking at all the others for each entry (4096 x 500, k 128: 175 us counted, 149
// sorted; 1000 x 300, k 65: 25 and 39).
constexpr uint32_t kSortedFrom = 448;
constexpr uint32_t kHeldMax = 16 * 1024;  // entries the short way keeps in shared memory: 64 KB, three CTAs per SM
constexpr uint32_t kHeldCopies = 4, kHeldChunk = kHeldMax / 4 / kHeldCopies;  // bulk copies, vectors of each

__device__ __forceinline__ uint32_t rank_key(float x, bool largest) {
    const uint32_t k = (x != x) ? 0xFFFFFFFFu : ordered_key(x);
    return largest ? k : ~k;
}

// Three-input maximum / minimum in one instruction (sm_100); the .NaN forms return NaN when any
// operand is NaN, the plain forms pass NaN operands by.
__device__ __forceinline__ float max3_nan(float a, float b, float c) {
    float r;
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// A key that at least kp (1-based, kp <= 32) of the 32 lanes' keys reach, the kp-th largest or up to 31 below it: for small kp the
// maximum is taken away kp - 1 times, the low five bits of a key giving way to its lane so that all are distinct; else a
// bitonic sort across the lanes.
__device__ __forceinline__ uint32_t warp_kth_largest_key(uint32_t key, int kp, int lane) {
    if (kp <= 10) {
        key = (key & ~31u) | (uint32_t)lane;
        uint32_t top = __reduce_max_sync(0xFFFFFFFFu, key);
        for (int i = 1; i < kp; ++i) {
            key = key == top ? 0u : key;
            top = __reduce_max_sync(0xFFFFFFFFu, key);
        }
        return top & ~31u;
    }
#pragma unroll
    for (int k = 2; k <= 32; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            const uint32_t other = __shfl_xor_sync(0xFFFFFFFFu, key, j);
            const bool descending_block = (lane & k) == 0, lower_lane = (lane & j) == 0;
            key = (lower_lane == descending_block) ? max(key, other) : min(key, other);
        }
    }
    return __shfl_sync(0xFFFFFFFFu, key, kp - 1);
}

struct TopKParams {
    const float* in;
    float* values;
    float* indices;
    size_t cols;
    size_t k;
    int largest;
    int cluster;     // CTAs per row
    uint32_t slice;  // entries per CTA (a multiple of 4)
    int in_shared;   // the slice's keys are kept in shared memory
    uint32_t k_pad;  // power of two >= k: slots of the collecting array
    uint32_t list_cap;  // entries of a CTA's short list (0: no lists)
    unsigned long long wait_limit_ns;  // longest wait for a copy in flight
};

// The cluster's histograms of one pass, added up and scanned from the top by warp 0 of every CTA:
// the digit at which the count from the top reaches `remaining`, the count above that digit, and
// the count in it.  hist points at this CTA's 256 counters of the pass (the same address in every
// CTA of the cluster); the histograms of CTAs first_rank .. first_rank + ranks - 1 are added up.
struct Found {
    uint32_t digit, above, inside;
};
__device__ __forceinline__ Found find_digit(cg::cluster_group& cluster, uint32_t* hist, int first_rank, int ranks,
                                            uint32_t remaining, int lane) {
    // lane L owns digits 255-8L down to 248-8L
    uint32_t bins[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int r = first_rank; r < first_rank + ranks; ++r) {
        const uint4* remote = reinterpret_cast<const uint4*>(cluster.map_shared_rank(hist, r));
        const uint4 lo = remote[62 - 2 * lane], hi = remote[63 - 2 * lane];
        bins[0] += hi.w; bins[1] += hi.z; bins[2] += hi.y; bins[3] += hi.x;
        bins[4] += lo.w; bins[5] += lo.z; bins[6] += lo.y; bins[7] += lo.x;
    }
    uint32_t local = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) local += bins[q];
    uint32_t incl = local;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t up = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += up;
    }
    const uint32_t excl = incl - local;
    const bool here = excl < remaining && remaining <= incl;
    uint32_t above = excl, inside = bins[0];
    int q_found = 0;
    if (here) {
#pragma unroll
        for (int q = 0; q < 7; ++q) {
            if (q_found == q && above + bins[q] < remaining) {
                above += bins[q];
                q_found = q + 1;
                inside = bins[q + 1];
            }
        }
    }
    const int src = max(0, __ffs(__ballot_sync(0xFFFFFFFFu, here)) - 1);  // exactly one lane while remaining <= total
    Found f;
    f.digit = __shfl_sync(0xFFFFFFFFu, (uint32_t)(255 - 8 * lane - q_found), src);
    f.above = __shfl_sync(0xFFFFFFFFu, above, src);
    f.inside = __shfl_sync(0xFFFFFFFFu, inside, src);
    return f;
}

// The long way (k > 256, or a list that overflowed: ties in the thousands), by the whole cluster over its slices.
// held4: the slice from its first 16-byte boundary on as floats in shared memory, or null.
template <bool kLargest, bool kHeld, int kThreads>
__device__ __forceinline__ void select_row(const TopKParams& p, u64* collected, uint32_t* keys, const float4* held4) {
    // histograms, used in turn by the passes; a pass clears the one before it once the cluster has met again (nobody reads it any more)
    __shared__ __align__(16) uint32_t s_hist[2][256];
    __shared__ uint32_t s_prefix, s_remaining, s_inside, s_collected;
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank(), ranks = p.cluster;
    const size_t row_index = blockIdx.x / (unsigned)p.cluster;
    constexpr bool largest = kLargest;
    const float* row = p.in + row_index * p.cols;
    const int tid = threadIdx.x, lane = tid & 31;
    const uint32_t n = (uint32_t)p.cols;
    const uint32_t begin = min(n, (uint32_t)rank * p.slice), mine = min(n, begin + p.slice) - begin;
    const bool in_shared = p.in_shared != 0;
    const float* src = row + begin;
    const uint32_t head = min(mine, (uint32_t)((4 - ((reinterpret_cast<uintptr_t>(src) >> 2) & 3)) & 3));
    const uint32_t vectors = (mine - head) / 4;
    const float4* src4 = reinterpret_cast<const float4*>(src + head);
    float* out_v = p.values + row_index * p.k;
    float* out_i = p.indices + row_index * p.k;
    // The cluster's barrier costs about a microsecond; one CTA on its own meets with the block barrier.
    auto meet = [&]() {
        if (ranks > 1) cluster.sync(); else __syncthreads();
    };
    for (int i = tid; i < 2 * 256; i += kThreads) (&s_hist[0][0])[i] = 0;
    if (tid == 0) s_collected = 0;

    // ---- 0. the slice as keys in shared memory, where it fits ------------------------------------------------
    if (in_shared) {
        // keys[head] on a 16-byte boundary, like src[head]: the array starts up to three words in
        keys = reinterpret_cast<uint32_t*>((reinterpret_cast<uintptr_t>(keys) + 15) & ~uintptr_t(15)) + ((4 - head) & 3);
        for (uint32_t i = tid; i < head; i += kThreads) keys[i] = rank_key(src[i], largest);
        uint4* keys4 = reinterpret_cast<uint4*>(keys + head);
        constexpr int kBatch = 8;  // loads in flight per thread
        for (uint32_t v0 = tid; v0 < vectors; v0 += kBatch * kThreads) {
            float4 d[kBatch];
#pragma unroll
            for (int q = 0; q < kBatch; ++q) {
                const uint32_t v = v0 + q * kThreads;
                d[q] = v < vectors ? __ldg(src4 + v) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
#pragma unroll
            for (int q = 0; q < kBatch; ++q) {
                const uint32_t v = v0 + q * kThreads;
                if (v < vectors) {
                    keys4[v] = make_uint4(rank_key(d[q].x, largest), rank_key(d[q].y, largest), rank_key(d[q].z, largest),
                                          rank_key(d[q].w, largest));
                }
            }
        }
        for (uint32_t i = head + 4 * vectors + tid; i < mine; i += kThreads) keys[i] = rank_key(src[i], largest);
    }
    __syncthreads();
    auto slice_key = [&](uint32_t i) { return in_shared ? keys[i] : rank_key(src[i], largest); };

    // visit(key, column) for every entry of the slice: four at a time where the slice lies in shared memory
    auto each_entry = [&](auto visit) {
        if (kHeld && held4 != nullptr) {
            for (uint32_t i = tid; i < head; i += kThreads) visit(rank_key(src[i], largest), begin + i);
            for (uint32_t v = tid; v < vectors; v += kThreads) {
                const float4 d = held4[v];
                const uint32_t col = begin + head + 4 * v;
                visit(rank_key(d.x, largest), col);
                visit(rank_key(d.y, largest), col + 1);
                visit(rank_key(d.z, largest), col + 2);
                visit(rank_key(d.w, largest), col + 3);
            }
            for (uint32_t i = head + 4 * vectors + tid; i < mine; i += kThreads) visit(rank_key(src[i], largest), begin + i);
        } else {
            for (uint32_t i = tid; i < mine; i += kThreads) visit(slice_key(i), begin + i);
        }
    };
    const int first_rank = 0;

    // ---- 1. radix select of the k-th key ---------------------------------------------------------------
    uint32_t prefix = 0, mask = 0, remaining = (uint32_t)p.k, inside = 0;
    for (int pass = 0; pass < 4; ++pass) {
        const int shift = 24 - 8 * pass;
        uint32_t* hist = s_hist[pass & 1];
        each_entry([&](uint32_t key, uint32_t) {
            if ((key & mask) == prefix) atomicAdd(&hist[(key >> shift) & 255u], 1u);
        });
        meet();
        if (pass > 0) {
            for (int i = tid; i < 256; i += kThreads) s_hist[(pass - 1) & 1][i] = 0;
        }
        if (tid < 32) {
            const Found f = find_digit(cluster, hist, first_rank, ranks, remaining, lane);
            if (lane == 0) {
                s_prefix = prefix | (f.digit << shift);
                s_remaining = remaining - f.above;
                s_inside = f.inside;
            }
        }
        __syncthreads();
        prefix = s_prefix;
        remaining = s_remaining;
        inside = s_inside;
        mask |= 255u << shift;
    }
    const uint32_t kth = prefix;
    const uint32_t ties_wanted = remaining;  // entries equal to the k-th key to take; `inside` entries equal it

    // ---- 2. more ties than wanted: the column up to which they are taken ------------------------------------
    uint32_t last_tie_column = 0xFFFFFFFFu;
    if (inside > ties_wanted) {  // uniform over the cluster
        uint32_t cprefix = 0, cmask = 0, cremaining = ties_wanted;
        for (int pass = 0; pass < 3; ++pass) {
            const int shift = 16 - 8 * pass;
            uint32_t* hist = s_hist[pass & 1];  // the key's four passes left [0] cleared and [1] to clear
            each_entry([&](uint32_t key, uint32_t col) {
                const uint32_t inverted = ~col & 0x00FFFFFFu;  // lower columns rank higher; columns are below 2^24
                if (key == kth && (inverted & cmask) == cprefix) atomicAdd(&hist[(inverted >> shift) & 255u], 1u);
            });
            meet();
            for (int i = tid; i < 256; i += kThreads) s_hist[(pass + 1) & 1][i] = 0;
            if (tid < 32) {
                const Found f = find_digit(cluster, hist, first_rank, ranks, cremaining, lane);
                if (lane == 0) {
                    s_prefix = cprefix | (f.digit << shift);
                    s_remaining = cremaining - f.above;
                }
            }
            __syncthreads();
            cprefix = s_prefix;
            cremaining = s_remaining;
            cmask |= 255u << shift;
        }
        last_tie_column = ~cprefix & 0x00FFFFFFu;
    }

    // ---- 3. collect in the first CTA, sort there, write -------------------------------------------------------
    {
        uint32_t* count0 = cluster.map_shared_rank(&s_collected, first_rank);
        u64* collected0 = cluster.map_shared_rank(collected, first_rank);
        each_entry([&](uint32_t key, uint32_t col) {
            if (key > kth || (key == kth && col <= last_tie_column)) {
                const uint32_t slot = atomicAdd(count0, 1u);
                if (slot < p.k_pad) collected0[slot] = ((u64)key << 32) | (uint32_t)~col;
            }
        });
    }
    meet();  // nobody touches another CTA's shared memory after this
    if (rank != 0) return;
    const uint32_t taken = min(s_collected, (uint32_t)p.k);  // == k
    for (uint32_t i = taken + tid; i < p.k_pad; i += kThreads) collected[i] = 0;
    __syncthreads();
    if (p.k_pad > 1) block_bitonic_sort(collected, (int)p.k_pad, /*descending=*/true);
    for (uint32_t j = tid; j < taken; j += kThreads) {
        const uint32_t col = ~(uint32_t)collected[j];
        out_v[j] = row[col];
        out_i[j] = (float)col;
    }
}

// The same as a call, so that the short way of a held slice has the registers to itself (4096 x 16,384, k 64: 77.8 us with the long way
// in line, 73.7 so); without a held slice the long way is the usual one and stays in line (k 256: 483 us, called 784).
template <bool kLargest, int kThreads>
__device__ __noinline__ void select_held_row(const TopKParams& p, u64* collected, uint32_t* keys, const float4* held4) {
    select_row<kLargest, true, kThreads>(p, collected, keys, held4);
}

// kHeld: the short way keeps its slice (at most kHeldMax entries) in shared memory, where four bulk copies bring it, each on a barrier of its
// own; the sweeps read it from there.
// kThreads: most of a CTA's instructions are a warp's own (its bound, its entries, their places), whatever its share of the
// slice: few warps where each still has at most 32 vectors per lane and k is at most half of the threads.
// kSorts: lists may be long (k above 64, where a list holds 512 entries and more) and are sorted then; a kernel of its own, since the code
// for it costs the others 2.5 %.
template <bool kLargest, bool kHeld, int kThreads, bool kSorts>
__global__ void __launch_bounds__(kThreads, 1024 / kThreads) topk_rows_kernel(const __grid_constant__ TopKParams p) {
    extern __shared__ __align__(16) unsigned char dyn[];
    // layout: [k_pad collected entries][list_cap listed entries][cluster * k_pad gathered entries], 8 bytes
    //         each, then [slice keys, 4 bytes each (when in_shared)]
    u64* collected = reinterpret_cast<u64*>(dyn);
    u64* list = collected + p.k_pad;
    uint32_t* list_key = reinterpret_cast<uint32_t*>(list + p.list_cap);  // the listed entries' keys by themselves
    uint32_t* claimed = list_key + p.list_cap;                            // entries that found themselves at a place
    u64* gathered = reinterpret_cast<u64*>(claimed + p.list_cap);
    uint32_t* keys = reinterpret_cast<uint32_t*>(gathered + (size_t)p.k_pad * (p.cluster > 1 && p.list_cap != 0 ? p.cluster : 0));
    __shared__ uint32_t s_listed, s_overflow;

    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank();
    int ranks = p.cluster;  // CTAs that take part in the steps below (1 once the lists are in the first CTA)
    const size_t row_index = blockIdx.x / (unsigned)p.cluster;
    constexpr bool largest = kLargest;
    const float* row = p.in + row_index * p.cols;
    const int tid = threadIdx.x, lane = tid & 31;
    const uint32_t n = (uint32_t)p.cols;
    const uint32_t begin = min(n, (uint32_t)rank * p.slice), end = min(n, begin + p.slice);
    const uint32_t mine = end - begin;
    // the slice from its first 16-byte boundary on, as vectors; up to three entries before them and after them
    const float* src = row + begin;
    const uint32_t head = min(mine, (uint32_t)((4 - ((reinterpret_cast<uintptr_t>(src) >> 2) & 3)) & 3));
    const uint32_t vectors = (mine - head) / 4;
    const float4* src4 = reinterpret_cast<const float4*>(src + head);
    float4* held4 = reinterpret_cast<float4*>((reinterpret_cast<uintptr_t>(keys) + 15) & ~uintptr_t(15));
    __shared__ __align__(8) uint64_t s_bar[kHeldCopies];
    if (kHeld && tid < kHeldCopies) {
        const uint32_t first = tid * kHeldChunk;
        if (first < vectors) {
            const uint32_t bytes = min(vectors - first, kHeldChunk) * 16;
            barrier_init(&s_bar[tid], 1);
            barrier_init_fence();
            barrier_expect_bytes(&s_bar[tid], bytes);
            bulk_copy_to_shared(held4 + first, src4 + first, bytes, &s_bar[tid]);
        }
    }
    // The held slice is padded to whole trips of the block with what nothing ranks below, so that the sweeps need no bounds.
    const uint32_t trips = (vectors + kThreads - 1) / kThreads;
    if (kHeld && vectors != trips * kThreads && (trips - 1) * kThreads + tid >= vectors) {
        const float worst = kLargest ? -INFINITY : INFINITY;
        held4[(trips - 1) * kThreads + tid] = make_float4(worst, worst, worst, worst);
    }
    for (uint32_t i = tid; i < p.list_cap / 2; i += kThreads) reinterpret_cast<uint4*>(list_key)[i] = make_uint4(0, 0, 0, 0);  // (claimed, too)
    if (tid == 0) {
        s_listed = 0;
        s_overflow = 0;
    }
    __syncthreads();
    float* out_v = p.values + row_index * p.k;
    float* out_i = p.indices + row_index * p.k;

    bool held_here = false;  // the slice lies in shared memory as floats
    // ---- 0. the short way (k <= 256): two sweeps over the slice as floats, the second one out of L2.
    //      Sweep one notes every thread's best entry; a bound that k of those reach is a lower bound of
    //      the slice's k-th best.  Sweep two lists what reaches the bound, usually k and a few; the list
    //      is put in rank order, and the best k of every CTA meet in the first CTA. ----------
    if (p.list_cap != 0) {  // uniform over the cluster
        __shared__ uint32_t s_warp_bound[kThreads / 32];
        constexpr int kBatch = 8;  // loads in flight per thread
        bool landed = true;
        // sweep one: the extreme entry this thread sees.  With the largest wanted a NaN is the best
        // there is, and the maximum that returns NaN for a NaN operand finds it; with the smallest
        // wanted a NaN is the worst, and the plain minimum passes it by.
        float extreme = largest ? -INFINITY : INFINITY;
        auto note = [&](float x) { extreme = largest ? max3_nan(extreme, x, x) : fminf(extreme, x); };
        auto note4 = [&](const float4& d) {
            extreme = largest ? max3_nan(max3_nan(d.x, d.y, d.z), d.w, extreme) : min3(min3(d.x, d.y, d.z), d.w, extreme);
        };
        for (uint32_t i = tid; i < head; i += kThreads) note(src[i]);
        if (kHeld) {
            constexpr uint32_t kTripsOfChunk = kHeldChunk / kThreads;
            for (uint32_t c = 0; c * kHeldChunk < vectors; ++c) {
                landed = barrier_wait_bounded(&s_bar[c], 0, p.wait_limit_ns) && landed;
                const float4* const mine4 = held4 + c * kHeldChunk + tid;
                if ((c + 1) * kTripsOfChunk <= trips) {
#pragma unroll
                    for (uint32_t q = 0; q < kTripsOfChunk; ++q) note4(mine4[q * kThreads]);
                } else {
                    for (uint32_t q = 0; c * kTripsOfChunk + q < trips; ++q) note4(mine4[q * kThreads]);
                }
            }
        } else {
            for (uint32_t v0 = tid; v0 < vectors; v0 += kBatch * kThreads) {
                float4 d[kBatch];
#pragma unroll
                for (int q = 0; q < kBatch; ++q) {
                    const uint32_t v = v0 + q * kThreads;
                    d[q] = v < vectors ? __ldg(src4 + v) : make_float4(extreme, extreme, extreme, extreme);
                }
#pragma unroll
                for (int q = 0; q < kBatch; ++q) note4(d[q]);
            }
        }
        for (uint32_t i = head + 4 * vectors + tid; i < mine; i += kThreads) note(src[i]);
        // The thread's best key, never overstated: a thread that saw nothing offers 0, and so does one
        // whose minimum is still +inf when the smallest are wanted (it may have seen nothing but NaN).
        const bool saw_any = (uint32_t)tid < head || (uint32_t)tid < vectors || head + 4 * vectors + tid < mine;
        uint32_t thread_max = saw_any ? rank_key(extreme, largest) : 0u;
        if (!largest && extreme == INFINITY) thread_max = 0;

        uint32_t bound = 0;
        if (mine > p.k) {  // else everything is listed
            // every warp's kp-th largest thread maximum, kp = ceil(k / 8): the smallest of the eight is
            // reached by 8 * kp >= k thread maxima (mine > k and k <= 256: enough threads hold an entry)
            const int kp = ((int)p.k + kThreads / 32 - 1) / (kThreads / 32);
            const uint32_t warp_bound = warp_kth_largest_key(thread_max, kp, lane);
            if (lane == 0) s_warp_bound[tid >> 5] = warp_bound;
            __syncthreads();
            bound = s_warp_bound[0];
#pragma unroll
            for (int w = 1; w < kThreads / 32; ++w) bound = min(bound, s_warp_bound[w]);
        }
        // sweep two: key >= bound, decided on the float itself: with the largest wanted, x is NaN or
        // x >= the bound's float; with the smallest wanted, x <= the mirrored bound's float.  A bound of
        // 0 lists everything; a bound that only NaN reaches is left to the long way.
        if (kHeld && __syncthreads_or(landed ? 0 : 1) != 0) {
            // a copy did not arrive in time: one more bounded wait (nothing may land after the CTA has left), then the long way
            for (uint32_t c = 0; c * kHeldChunk < vectors; ++c) barrier_wait_bounded(&s_bar[c], 0, p.wait_limit_ns);
            landed = false;
        }
        held_here = kHeld && landed;
        const float edge = largest ? from_ordered_key(bound) : from_ordered_key(~bound);
        const bool everything = bound == 0 && landed, only_nan = edge != edge || !landed;  // (or only what no number lies below)
        auto reaches = [&](float x) { return largest ? !(x < edge) : x <= edge; };
        auto put = [&](float x, uint32_t col) {
            const uint32_t slot = atomicAdd(&s_listed, 1u);
            if (slot < p.list_cap) {
                const uint32_t key = rank_key(x, largest);
                list[slot] = ((u64)key << 32) | (uint32_t)~col;
                list_key[slot] = key;
            }
        };
        if (everything) {
            if (mine <= p.list_cap) {
                for (uint32_t i = tid; i < mine; i += kThreads) put(src[i], begin + i);
            } else if (tid == 0) {
                s_listed = p.list_cap + 1;  // does not fit
            }
        } else if (only_nan) {
            if (tid == 0) s_listed = p.list_cap + 1;
        } else {
            for (uint32_t i = tid; i < head; i += kThreads) {
                if (reaches(src[i])) put(src[i], begin + i);
            }
            if (kHeld) {
                // branch-free over the vectors, one bit for each that reaches the bound
                uint32_t noted = 0;
                const float4* const mine4 = held4 + tid;
#pragma unroll 8
                for (uint32_t t = 0; t < trips; ++t) {
                    const float4 d = mine4[t * kThreads];
                    const float best4 = largest ? max3_nan(max3_nan(d.x, d.y, d.z), d.w, d.w) : min3(min3(d.x, d.y, d.z), d.w, d.w);
                    if (reaches(best4)) noted |= 1u << t;
                }
                if (trips * kThreads - kThreads + tid >= vectors) noted &= ~(1u << ((trips - 1) & 31));  // padding
                for (uint32_t m = noted; m != 0; m &= m - 1) {
                    const uint32_t v = (__ffs(m) - 1) * kThreads + tid, col = begin + head + 4 * v;
                    const float4 d = held4[v];
                    if (reaches(d.x)) put(d.x, col);
                    if (reaches(d.y)) put(d.y, col + 1);
                    if (reaches(d.z)) put(d.z, col + 2);
                    if (reaches(d.w)) put(d.w, col + 3);
                }
            } else
            for (uint32_t v0 = tid; v0 < vectors; v0 += kBatch * kThreads) {
                float4 d[kBatch];
#pragma unroll
                for (int q = 0; q < kBatch; ++q) {
                    const uint32_t v = v0 + q * kThreads;
                    // beyond the slice: a value that does not reach the bound
                    d[q] = v < vectors ? __ldg(src4 + v) : (largest ? make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY)
                                                                   : make_float4(INFINITY, INFINITY, INFINITY, INFINITY));
                }
#pragma unroll
                for (int q = 0; q < kBatch; ++q) {
                    // (a NaN among the four makes best4 NaN when the largest are wanted, and NaN reaches)
                    const float best4 = largest ? max3_nan(max3_nan(d[q].x, d[q].y, d[q].z), d[q].w, d[q].w)
                                                : min3(min3(d[q].x, d[q].y, d[q].z), d[q].w, d[q].w);
                    if (reaches(best4) && v0 + q * kThreads < vectors) {  // rare
                        const uint32_t col = begin + head + 4 * (v0 + q * kThreads);
                        if (reaches(d[q].x)) put(d[q].x, col);
                        if (reaches(d[q].y)) put(d[q].y, col + 1);
                        if (reaches(d[q].z)) put(d[q].z, col + 2);
                        if (reaches(d[q].w)) put(d[q].w, col + 3);
                    }
                }
            }
            for (uint32_t i = head + 4 * vectors + tid; i < mine; i += kThreads) {
                if (reaches(src[i])) put(src[i], begin + i);
            }
        }
        __syncthreads();
        const uint32_t on_list = s_listed;
        // (A list of the whole slice is a row of equal values, as a rule: the radix selection is faster than telling them apart.  16,384
        // constant rows of 200, k 8: 310 us, 163 so.)
        const bool fits = on_list <= p.list_cap && (everything || on_list < mine);
        const uint32_t best = min(on_list, (uint32_t)p.k);  // entries of this CTA that can be among the row's k best
        // Where the best entries go: straight out (one CTA), or into this CTA's k_pad slots of the
        // first CTA's array.  An entry's place is the number of entries that rank before it.
        u64* gathered0 = ranks > 1 ? cluster.map_shared_rank(gathered, 0) + (size_t)rank * p.k_pad : nullptr;
        if (fits) {
            auto place_entry = [&](u64 entry, uint32_t place) {
                if (place >= best) return;
                if (ranks == 1) {
                    const uint32_t col = ~(uint32_t)entry, at = col - begin - head;
                    out_v[place] = kHeld && at < 4 * vectors ? reinterpret_cast<const float*>(held4)[at] : row[col];
                    out_i[place] = (float)col;
                } else {
                    gathered0[place] = entry;
                }
            };
            if (kSorts && on_list > kSortedFrom) {
                uint32_t n_pad = 512;
                while (n_pad < on_list) n_pad <<= 1;
                for (uint32_t i = on_list + tid; i < n_pad; i += kThreads) list[i] = 0;
                __syncthreads();
                block_bitonic_sort(list, (int)n_pad, /*descending=*/true);
                for (uint32_t i = tid; i < best; i += kThreads) place_entry(list[i], i);
            } else {
                // An entry's place by looking at all the others' keys, four at a time; neighbouring threads share an entry when there are
                // threads left over.  Entries with equal keys find themselves at the same place: then (rare) the columns are looked at too.
                uint32_t n_pad = 8;
                while (n_pad < on_list && n_pad < (uint32_t)kThreads) n_pad <<= 1;
                const uint32_t share = (uint32_t)kThreads / n_pad < 32u ? (uint32_t)kThreads / n_pad : 32u, slice = tid & (share - 1);
                const uint32_t quads = (on_list + 3) / 4, per_round = (uint32_t)kThreads / share;  // (zeros behind the list)
                bool tied = false;
                for (uint32_t first = 0; first < on_list; first += per_round) {
                    const uint32_t i = first + (uint32_t)tid / share;
                    if (first + (uint32_t)(tid & ~31) / share >= on_list) break;  // (nothing for this warp)
                    const uint32_t key = i < on_list ? list_key[i] : ~0u;
                    uint32_t place = 0;
#pragma unroll 4
                    for (uint32_t j = slice; j < quads; j += share) {
                        const uint4 other = reinterpret_cast<const uint4*>(list_key)[j];
                        place += (other.x > key ? 1u : 0u) + (other.y > key ? 1u : 0u) + (other.z > key ? 1u : 0u) + (other.w > key ? 1u : 0u);
                    }
                    for (uint32_t o = share >> 1; o > 0; o >>= 1) place += __shfl_xor_sync(0xFFFFFFFFu, place, o);
                    if (slice == 0 && i < on_list && place < best) {
                        if (atomicAdd(&claimed[place], 1u) != 0) tied = true;
                        place_entry(list[i], place);
                    }
                }
                if (__syncthreads_or(tied ? 1 : 0) != 0) {
                    for (uint32_t i = tid; i < on_list; i += kThreads) {
                        const u64 entry = list[i];
                        uint32_t place = 0;
                        for (uint32_t j = 0; j < on_list; ++j) place += list[j] > entry ? 1u : 0u;
                        place_entry(entry, place);
                    }
                }
            }
            if (ranks == 1) return;
            for (uint32_t j = best + tid; j < p.k_pad; j += kThreads) gathered0[j] = 0;
        }
        if (ranks > 1) {
            if (tid == 0) s_overflow = fits ? 0u : 1u;
            cluster.sync();
            uint32_t overflow = 0;
            for (int r = 0; r < ranks; ++r) overflow |= *cluster.map_shared_rank(&s_overflow, r);
            if (overflow == 0) {  // uniform over the cluster
                cluster.sync();   // everybody has read everybody's verdict: CTAs may leave
                if (rank != 0) return;
                // The CTAs' lists are in rank order (zeros fill them up): an entry's place is its place in its own list and, by
                // bisection, the number of entries of each other list that rank before it.
                for (uint32_t i = tid; i < p.k_pad * (uint32_t)ranks; i += kThreads) {
                    const u64 entry = gathered[i];
                    const uint32_t own = i / p.k_pad;
                    uint32_t place = i - own * p.k_pad;
                    if (entry == 0 || place >= (uint32_t)p.k) continue;
                    for (uint32_t r = 0; r < (uint32_t)ranks; ++r) {
                        if (r == own) continue;
                        const u64* other = gathered + r * p.k_pad;
                        uint32_t before = 0;
                        for (uint32_t step = p.k_pad; step > 0; step >>= 1) {
                            if (before + step <= p.k_pad && other[before + step - 1] > entry) before += step;
                        }
                        place += before;
                    }
                    if (place < (uint32_t)p.k) {
                        const uint32_t col = ~(uint32_t)entry;
                        out_v[place] = row[col];
                        out_i[place] = (float)col;
                    }
                }
                return;
            }
        }
        // (s_listed stays as it is: a warp that is late has yet to read it, and all have to come to the same verdict)
    }
    if (kHeld) select_held_row<kLargest, kThreads>(p, collected, keys, held_here ? held4 : nullptr);
    else select_row<kLargest, false, kThreads>(p, collected, keys, nullptr);
}

// ---- k beyond what one CTA's shared memory sorts: the whole row is sorted in global memory -----------
// One CTA of 1024 threads per row: the row becomes 64-bit keys (rank key, ~column), padded to a power
// of two with keys below every real one, in scratch memory; a bitonic network sorts them, descending --
// steps that reach across more than 4096 keys run over global memory, all the others over one tile of
// 4096 keys at a time in shared memory --, and the first k keys are the answer, in rank order: equal
// values keep the lower column first because ~column is part of the key.
constexpr int kSortThreads = 1024;
constexpr int kSortTile = 4096;

__device__ __forceinline__ void tile_steps(u64* tile, uint32_t tile_base, uint32_t k2, uint32_t j_from) {
    for (uint32_t j = j_from; j > 0; j >>= 1) {
        for (uint32_t q = threadIdx.x; q < kSortTile / 2; q += kSortThreads) {
            const uint32_t i = ((q & ~(j - 1)) << 1) | (q & (j - 1)), l = i | j;
            const bool descending = ((tile_base + i) & k2) == 0;
            const u64 a = tile[i], b = tile[l];
            if (descending ? a < b : a > b) {
                tile[i] = b;
                tile[l] = a;
            }
        }
        __syncthreads();
    }
}

template <bool kLargest>
__global__ void __launch_bounds__(kSortThreads) sort_rows_kernel(const float* __restrict__ in, float* values, float* indices,
                                                                 u64* scratch, size_t cols, size_t k, uint32_t n_pad,
                                                                 size_t first_row) {
    __shared__ u64 tile[kSortTile];
    const size_t row = first_row + blockIdx.x;
    const float* x = in + row * cols;
    u64* keys = scratch + (size_t)blockIdx.x * n_pad;
    const uint32_t tile_len = min((uint32_t)kSortTile, n_pad);
    // every tile on its own: keys from the row, all steps up to the tile's length
    for (uint32_t base = 0; base < n_pad; base += kSortTile) {
        for (uint32_t t = threadIdx.x; t < tile_len; t += kSortThreads) {
            const size_t i = (size_t)base + t;
            tile[t] = i < cols ? (((u64)rank_key(x[i], kLargest) << 32) | (uint32_t)~(uint32_t)i) : 0ull;
        }
        __syncthreads();
        for (uint32_t k2 = 2; k2 <= tile_len; k2 <<= 1) {
            for (uint32_t j = k2 >> 1; j > 0; j >>= 1) {
                for (uint32_t q = threadIdx.x; q < tile_len / 2; q += kSortThreads) {
                    const uint32_t i = ((q & ~(j - 1)) << 1) | (q & (j - 1)), l = i | j;
                    const bool descending = ((base + i) & k2) == 0;
                    const u64 a = tile[i], b = tile[l];
                    if (descending ? a < b : a > b) {
                        tile[i] = b;
                        tile[l] = a;
                    }
                }
                __syncthreads();
            }
        }
        for (uint32_t t = threadIdx.x; t < tile_len; t += kSortThreads) keys[base + t] = tile[t];
        __syncthreads();
    }
    // the longer steps over global memory, the rest of each merge over the tiles again
    for (uint32_t k2 = 2 * kSortTile; k2 <= n_pad && k2 != 0; k2 <<= 1) {
        for (uint32_t j = k2 >> 1; j >= (uint32_t)kSortTile; j >>= 1) {
            for (uint32_t q = threadIdx.x; q < n_pad / 2; q += kSortThreads) {
                const uint32_t i = ((q & ~(j - 1)) << 1) | (q & (j - 1)), l = i | j;
                const bool descending = (i & k2) == 0;
                const u64 a = keys[i], b = keys[l];
                if (descending ? a < b : a > b) {
                    keys[i] = b;
                    keys[l] = a;
                }
            }
            __syncthreads();  // (orders this block's global writes before its next reads)
        }
        for (uint32_t base = 0; base < n_pad; base += kSortTile) {
            for (uint32_t t = threadIdx.x; t < kSortTile; t += kSortThreads) tile[t] = keys[base + t];
            __syncthreads();
            tile_steps(tile, base, k2, kSortTile / 2);
            for (uint32_t t = threadIdx.x; t < kSortTile; t += kSortThreads) keys[base + t] = tile[t];
            __syncthreads();
        }
    }
    for (size_t jj = threadIdx.x; jj < k; jj += kSortThreads) {
        const uint32_t col = ~(uint32_t)keys[jj];
        values[row * k + jj] = x[col];
        indices[row * k + jj] = (float)col;
    }
}

}  // namespace

size_t sort_rows_scratch_bytes(size_t rows, size_t cols, size_t* rows_per_launch) {
    size_t n_pad = 1;
    while (n_pad < cols) n_pad <<= 1;
    const size_t budget = (size_t)256 << 20;  // scratch of one launch
    size_t batch = budget / (n_pad * 8);
    batch = batch < 1 ? 1 : batch > rows ? rows : batch;
    if (rows_per_launch) *rows_per_launch = batch;
    return batch * n_pad * 8;
}

cudaError_t launch_sort_rows(const float* in, float* values, float* indices, size_t rows, size_t cols, size_t k, bool largest,
                             void* scratch, cudaStream_t stream) {
    if (rows == 0) return cudaSuccess;
    size_t batch = 0;
    sort_rows_scratch_bytes(rows, cols, &batch);
    uint32_t n_pad = 1;
    while (n_pad < cols) n_pad <<= 1;
    for (size_t first = 0; first < rows; first += batch) {
        const unsigned blocks = (unsigned)(rows - first < batch ? rows - first : batch);
        if (largest) {
            sort_rows_kernel<true><<<blocks, kSortThreads, 0, stream>>>(in, values, indices, static_cast<u64*>(scratch), cols, k,
                                                                       n_pad, first);
        } else {
            sort_rows_kernel<false><<<blocks, kSortThreads, 0, stream>>>(in, values, indices, static_cast<u64*>(scratch), cols, k,
                                                                        n_pad, first);
        }
        if (cudaError_t e = cudaGetLastError(); e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_topk_rows(const float* in, float* values, float* indices, size_t rows, size_t cols, size_t k,
                             bool largest, int sm_count, cudaStream_t stream) {
    if (rows == 0) return cudaSuccess;
    TopKParams p;
    p.in = in;
    p.values = values;
    p.indices = indices;
    p.cols = cols;
    p.k = k;
    p.largest = largest ? 1 : 0;
    p.cluster = cols <= 16384 ? 1 : cols <= 32768 ? 2 : cols <= 65536 ? 4 : 8;
    p.slice = (uint32_t)(((cols + p.cluster - 1) / p.cluster + 3) / 4 * 4);
    p.k_pad = 2;  // (an even number of slots: what follows them starts on 16 bytes)
    while (p.k_pad < k) p.k_pad <<= 1;
    // The short way (k <= 256) needs no keys in shared memory; if one of its lists overflows, the
    // long way sweeps global memory.  Otherwise the keys are kept when they fit.
    p.list_cap = k <= (size_t)kWidest ? 4 * (p.k_pad < 64 ? 64 : p.k_pad) : 0;
    const size_t entries = p.k_pad + 2 * p.list_cap + (p.cluster > 1 && p.list_cap != 0 ? (size_t)p.cluster * p.k_pad : 0);
    p.in_shared = p.list_cap == 0 && p.slice <= (uint32_t)kSliceMax &&
                  entries * 8 + (size_t)p.slice * 4 + 4096 <= 227 * 1024 ? 1 : 0;
    p.wait_limit_ns = kDefaultWaitLimitNs;
    // Beyond k 128 lists overflow more often than not, and a block that holds its slice has fewer beside it to hide the radix
    // selection: 4096 x 16,384, k 256: 840 us with held slices, 483 without (k 100: 115 and 120).  Where all blocks are resident at once,
    // three on each SM, it does not matter: 64 x 16,384, k 200: 23 to 34 us held (as lists overflow), 37 not.
    const bool held = p.list_cap != 0 && p.slice <= kHeldMax && (k <= 128 || rows * p.cluster <= 3 * (size_t)sm_count);
    const int threads = !held || k > 32 ? kWidest : p.slice <= 4096 && k <= 32 ? 64 : 128;
    auto kernel = largest ? topk_rows_kernel<true, false, kWidest, true> : topk_rows_kernel<false, false, kWidest, true>;
    if (held && threads == 64) kernel = largest ? topk_rows_kernel<true, true, 64, false> : topk_rows_kernel<false, true, 64, false>;
    else if (held && threads == 128) kernel = largest ? topk_rows_kernel<true, true, 128, false> : topk_rows_kernel<false, true, 128, false>;
    else if (held && k <= 64) kernel = largest ? topk_rows_kernel<true, true, kWidest, false> : topk_rows_kernel<false, true, kWidest, false>;
    else if (held) kernel = largest ? topk_rows_kernel<true, true, kWidest, true> : topk_rows_kernel<false, true, kWidest, true>;
    const size_t shared = entries * 8 + (p.in_shared ? (size_t)p.slice * 4 + 32 : held ? (p.slice / 4 + threads - 1) / threads * threads * 16 + 32 : 0);
    if (rows * (size_t)p.cluster > 0x7FFFFFFFull) return cudaErrorInvalidConfiguration;
    // (whatever the size: what a block may use without asking counts the kernel's own arrays as well)
    static OncePerDevice lifted[10];
    OncePerDevice& done = lifted[(largest ? 1 : 0) + (!held ? 0 : threads == 64 ? 2 : threads == 128 ? 4 : k <= 64 ? 6 : 8)];
    if (const cudaError_t e = allow_all_dynamic_shared_once(done, kernel); e != cudaSuccess) return e;
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3((unsigned)(rows * p.cluster));
    config.blockDim = dim3((unsigned)threads);
    config.dynamicSmemBytes = shared;
    config.stream = stream;
    cudaLaunchAttribute attribute[1];
    attribute[0].id = cudaLaunchAttributeClusterDimension;
    attribute[0].val.clusterDim.x = (unsigned)p.cluster;
    attribute[0].val.clusterDim.y = 1;
    attribute[0].val.clusterDim.z = 1;
    config.attrs = attribute;
    config.numAttrs = p.cluster > 1 ? 1 : 0;  // a row of one CTA is an ordinary launch
    return cudaLaunchKernelEx(&config, kernel, p);
}

}  // namespace psx
