// The survivor stage: a CTA per row -- a warp per row for many greedy rows -- turns the row pass's candidates into a token.
//
// Input per row: for each part its raw max / tail sum-exp and a few dozen candidates (raw logit,
// column, flags).  The stage
//   1. joins the parts' partial log-sum-exp (raw, and processed when a full-vocabulary top-p or
//      min-p needs it): M = max m_i, Z = sum z_i * exp(m_i - M) + sum over candidates, in double;
//   2. keeps the candidates at or above the largest part threshold (only those can survive any
//      filter) and applies penalty and temperature with the reference's float operations;
//   3. decides src/generation.cpp:80-152 on that short list: as a rule with integer sums over the entries that come
//      before an entry (merge_rows_list_impl.cuh), and where a list does not fit or a decision is too close to its level by
//      replaying the reference's own order and precision -- the k-th value with its ties, softmax sums in column order,
//      the top-p walk in ascending (value, column) order against 1 - (double)top_p, min-p against the first
//      maximum, the inverse-CDF walk in column order against the row's uniform -- all in double (merge_rows_impl.cuh);
//   4. writes the token, float(log(exp(l - M) / Z)) of the raw logits (src/generation.cpp:156),
//      a row status and the distances of the two decisions from their boundaries.
// Reads a few KB per row and never touches the logits -- except for a row that does not fit the
// lists (more survivors or ties than they hold): that row is decided from the logits themselves
// by the same CTA (general_row_impl.cuh).
#ifdef PSX_STAGE_CLOCKS
// Profiling build only: thread 0 of each row's CTA stamps the SM clock at the stage boundaries.
__device__ unsigned long long g_merge_clocks[1024 * 16];
#define PSX_MERGE_STAGE(i) \
    do { if (threadIdx.x == 0) g_merge_clocks[(size_t)(blockIdx.x & 1023) * 16 + (i)] = clock64(); } while (0)
// wall-clock (globaltimer) stamps of each CTA: entry, after the wait for the row pass, exit
__device__ unsigned long long g_merge_times[1024 * 4];
#define PSX_MERGE_TIME(i) \
    do { if (threadIdx.x == 0) { unsigned long long t_; asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_)); \
         g_merge_times[(size_t)(blockIdx.x & 1023) * 4 + (i)] = t_; } } while (0)
#else
#define PSX_MERGE_TIME(i) do {} while (0)
#endif
#include "general_row_impl.cuh"
#include "merge_rows_impl.cuh"
#include "merge_rows_list_impl.cuh"
#include "peer_exchange.cuh"

#include <algorithm>

namespace psx {

namespace {

// What the lists of a row do not decide, by the whole block: of a greedy row the parts' maxima are known all the same.
template <bool kGreedy>
__device__ __forceinline__ void replay_row(const MergeParams& p, const int64_t row, unsigned long long* dyn) {
    if constexpr (kGreedy) {
        if (p.general == 1 && p.parts <= 32 && survivor::row_fits(p)) {
            const survivor::RowView v = survivor::view_of_row(p, row);
            survivor::PartsJoined j;
            survivor::load_parts(p, v, j);
            survivor::join_parts(p, v, j);
            j.bad &= 3u;  // (that a list ran over is known)
            if (!survivor::settle_bad_row(v, j, j.y_max)) survivor::greedy_row(p, row, j.raw_max, j.y_max, dyn);
            return;
        }
    }
    if (p.general != 2) survivor::merge_row(p, row, dyn);  // too many for the list, or a decision too close to its level
    if (p.general != 0 && p.logits != nullptr) {
        // A row the candidate lists could not decide is decided from the row itself.
        __syncthreads();
        if (p.general == 2 || p.row_status[row] == PSX_ROW_TOO_WIDE) survivor::general_row(p, row, dyn);
    }
}

// Greedy, a warp per row and up to eight rows per block.  A greedy row has a few candidates per part: latency bound, a trip to memory and two
// exponentials, for which eight warps are seven too many once there are more rows than blocks fit the GPU at once.  1024 x 49,152, the whole
// call: 45.2 us with a block per row (2.3 rounds of them), 40.8 so; 4000 x 8000: 59 and 41 us.
// A row that its warp cannot decide is left to its block, the block's rows one after another.  Such rows lie side by side (padding) or a power of two
// apart, so a block's rows lie an odd number of blocks apart, and as many blocks share the rows as the GPU holds.  1024 x 49,152 with 64 constant
// rows side by side: 183 us by blocks, 583 with eight neighbours to a block, 102 so; every fourth row constant: 223, 252, 140; a quarter at random: 223, 415, 221;
// all: 593, 756, 318.
__global__ void __launch_bounds__(kMergeThreads, 3) merge_greedy_rows_kernel(const __grid_constant__ MergeParams p) {
    extern __shared__ __align__(16) unsigned long long dyn[];
    __shared__ uint32_t s_left;  // rows that their warps could not decide
    const int warp = threadIdx.x >> 5;
    const int64_t mine = blockIdx.x + (int64_t)gridDim.x * warp;
    if (threadIdx.x == 0) s_left = 0;
    __syncthreads();
    grid_dependency_wait();        // everything this kernel reads was written by the kernel before it
    grid_dependents_may_launch();  // a row pass that follows reads none of this kernel's results
    if (mine < p.rows && !survivor::list_greedy_by_warp(p, survivor::view_of_row(p, p.row_begin + mine))) {
        if ((threadIdx.x & 31) == 0) atomicOr(&s_left, 1u << warp);
    }
    __syncthreads();
    for (uint32_t left = s_left; left; left &= left - 1) {
        replay_row<true>(p, p.row_begin + blockIdx.x + (int64_t)gridDim.x * (__ffs(left) - 1), dyn);
        __syncthreads();
    }
}

template <int kKind>
__global__ void __launch_bounds__(kMergeThreads, kKind == survivor::kListNucleus ? 2 : 3) merge_rows_kernel(const __grid_constant__ MergeParams p) {
    extern __shared__ __align__(16) unsigned long long dyn[];
    const int64_t row = p.row_begin + blockIdx.x;
    PSX_MERGE_TIME(0);
    bool arrived = true;
    if (p.arrivals != nullptr) {
        // Lists that other GPUs write (peer_exchange.cuh): nothing here is read before the row's arrival
        // counter says that every shard's record is complete -- this GPU's own among them, so the kernel
        // before this one is not waited for as a whole, and the kernel after this one may start at once.
        grid_dependents_may_launch();
        __shared__ int s_arrived;
        if (threadIdx.x == 0) s_arrived = wait_until_at_least(p.arrivals + row, p.arrivals_target, p.arrivals_wait_ns) ? 1 : 0;
        __syncthreads();
        arrived = s_arrived != 0;
    }
    auto ready = [&]() {
        if (p.arrivals != nullptr) return;
        grid_dependency_wait();        // everything this kernel reads was written by the kernel before it
        grid_dependents_may_launch();  // a row pass that follows reads none of this kernel's results
        PSX_MERGE_TIME(1);
    };
    if (p.general == 2) ready();
    if (!arrived) {
        if (threadIdx.x == 0) {
            p.tokens[row] = -1;
            p.log_probs[row] = 0.0f;
            p.row_status[row] = PSX_ROW_DEVICE_TIMEOUT;
            if (p.diag) p.diag[row] = psx_row_diag{0, 0, INFINITY, INFINITY};
        }
    } else if (p.general == 2 || !survivor::list_row<kKind>(p, row, survivor::view_of_row(p, row), dyn, ready)) {
        __syncthreads();
        replay_row<kKind == survivor::kListGreedy>(p, row, dyn);
    }
    if (p.arrivals != nullptr) {
        __syncthreads();
        if (p.publish && (int)threadIdx.x < p.peers.world) {  // one thread per rank: the row's 16 bytes, then the count
            const PeerLayout& l = p.peers;
            const int64_t within = row - (int64_t)l.rank * l.rows_per_rank;
            char* block = l.base[threadIdx.x] + l.results_offset + (int64_t)l.rank * peer_results_block_bytes(l.rows_per_rank);
            reinterpret_cast<int64_t*>(block)[within] = p.tokens[row];
            reinterpret_cast<float*>(block + 8 * l.rows_per_rank)[within] = p.log_probs[row];
            reinterpret_cast<int32_t*>(block + 12 * l.rows_per_rank)[within] = p.row_status[row];
            add_release_system(reinterpret_cast<uint32_t*>(l.base[threadIdx.x] + l.flags_offset) + l.rank, 1u);  // (a release)
        }
        grid_dependency_wait();  // (so that this kernel's end still implies the end of the kernel before it)
    }
    PSX_MERGE_TIME(2);
}

}  // namespace

#ifdef PSX_STAGE_CLOCKS
extern "C" __attribute__((visibility("default"))) int psx_debug_merge_clocks(unsigned long long* out, int n) {
    return (int)cudaMemcpyFromSymbol(out, g_merge_clocks, sizeof(unsigned long long) * n);
}
extern "C" __attribute__((visibility("default"))) int psx_debug_merge_times(unsigned long long* out, int n) {
    return (int)cudaMemcpyFromSymbol(out, g_merge_times, sizeof(unsigned long long) * n);
}
#endif

size_t merge_rows_shared_bytes(int sort_capacity, int gather_capacity, bool overlay) {
    const size_t list = (size_t)sort_capacity * 8, rest = (size_t)sort_capacity * (8 + 8 + 1), gathered = (size_t)gather_capacity * 8;
    return list + (overlay ? (rest > gathered ? rest : gathered) : rest + gathered) + 16;
}

int merge_slot_shift(int parts, int part_cap, int expected) {
    int shift = 0;
    // room for about twice what is expected, inside a list, inside what 16 fetches per thread reach
    while ((1 << shift) < 2 * expected && (2 << shift) <= part_cap && ((long long)parts << (shift + 1)) <= 16 * kMergeThreads) {
        ++shift;
    }
    return shift;
}

cudaError_t configure_merge_rows() {
    cudaError_t e = allow_all_dynamic_shared(merge_rows_kernel<survivor::kListGreedy>);
    if (e == cudaSuccess) e = allow_all_dynamic_shared(merge_greedy_rows_kernel);
    if (e == cudaSuccess) e = allow_all_dynamic_shared(merge_rows_kernel<survivor::kListTopK>);
    if (e == cudaSuccess) e = allow_all_dynamic_shared(merge_rows_kernel<survivor::kListNucleus>);
    return e;
}

namespace {
auto kernel_for(const MergeParams& p) {
    if (!p.do_sample) return merge_rows_kernel<survivor::kListGreedy>;
    return p.top_k > 0 && p.top_k < p.vocab ? merge_rows_kernel<survivor::kListTopK> : merge_rows_kernel<survivor::kListNucleus>;
}
}  // namespace

cudaError_t launch_merge_rows(const MergeParams& p, int sm_count, cudaStream_t stream, uint64_t* launched) {
    if (p.rows <= 0) return cudaSuccess;
    // The same condition as the kernel's: the overlaid layout is for plans without a top-k.
    const bool overlay = p.overlay != 0 && p.logits != nullptr && !(p.do_sample && p.top_k > 0 && p.top_k < p.vocab);
    const size_t shared = merge_rows_shared_bytes(p.sort_capacity, p.gather_capacity, overlay);
    MergeParams with_size = p;
    with_size.dyn_bytes = (int32_t)shared;
    if (launched != nullptr) ++*launched;
    // A warp per greedy row where a block each would take a second round (three to an SM), up to eight parts.  The whole call by blocks and by warps, us:
    // three parts, 49,152 columns: 400 rows 18.3 and 18.0, 500 25.2 and 23.0, 1024 45.2 and 40.8; five parts, 81,920: 450 rows 33.6 and 33.2, 1024 66.1 and
    // 62.5 (65,537, up to 512 rows: 32.1 and 32.9); eight parts, 128,256: 450 rows 47.6 and 47.1, 1024 97.2 and 93.6; sixteen, 262,144: 500 rows 92.7 and 93.9.
    // Rows that are handed on whole, 1024 x 600: 19 and 26.
    if (!p.do_sample && p.rows > 3 * sm_count && p.parts <= 8 && p.whole_rows == 0 && p.arrivals == nullptr && p.survivor_cols == nullptr) {
        const unsigned blocks = (unsigned)std::max<int64_t>(3 * sm_count - 1, (p.rows + survivor::kListWarps - 1) / survivor::kListWarps) | 1u;
        return launch_overlapping(merge_greedy_rows_kernel, dim3(blocks), dim3(kMergeThreads), shared, stream, with_size);
    }
    return launch_overlapping(kernel_for(p), dim3((unsigned)p.rows), dim3(kMergeThreads), shared, stream, with_size);
}

}  // namespace psx
