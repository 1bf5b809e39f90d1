// Row primitives beside the sampling path: softmax_rows, logsumexp_rows and gather_rows of the
// reference's DeviceBackend (include/pulsatrix/device_backend.hpp:456,465,596; CPU semantics
// src/cpu_backend.cpp:292-338,459-466; the reference's CUDA kernels run one thread per row,
// src/gpu_kernels.cuh:315-365, or one thread per element, :665).
//
// softmax / logsumexp read every element once and (softmax) write it once:
//   - a row of up to 32,768 columns belongs to as few warps as hold it with eight 128-bit vectors per lane (one warp up
//     to 1024 columns, four up to 4096, 16 from 8192 on): all of a lane's loads are in flight at once, and few warps meet.
//     Rows that do not start on a 16-byte boundary are taken as the aligned vectors they span; a result that lies differently
//     against the boundary is written element by element, and beyond 8190 columns or so takes the way below;
//   - a longer row is a thread-block cluster's: up to eight CTAs of 16,384 columns (beyond 131,072 columns 32,768), so that two
//     CTAs share an SM; the row's maximum and sum meet in distributed shared memory;
//   - beyond 262,144 columns one CTA walks the row three times.
// Float arithmetic like the reference's: exp(x - max) as one ex2 of (x - max) * log2(e) (relative
// error below 1e-5, against the reference's CPU/GPU tolerance of 1e-4), float sums in a fixed tree
// (the same input gives the same bits; the reference's sequential sum differs from it by rounding
// only), y = e / sum, lse = max + logf(sum).  The quotient is e * (1 / sum) with its remainder put back once (Markstein, "Computation of
// elementary functions on the IBM RISC System/6000", 1990): correctly rounded but for a rare last bit, three operations in place of a divide.
#include <cooperative_groups.h>

#include "psx_device.cuh"
#include "row_ops.cuh"

namespace psx {

namespace {

namespace cg = cooperative_groups;

constexpr int kCtaThreads = 512;
constexpr int kCtaVecs = 16;            // float4 per thread
constexpr int kCtaCols = kCtaThreads * kCtaVecs * 4;  // 32,768
constexpr int kMaxCluster = 8;

__device__ __forceinline__ float warp_sum_f(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    return v;
}

__device__ __forceinline__ float quotient(float e, float sum, float reciprocal) {
    const float q = __fmul_rn(e, reciprocal);
    return __fmaf_rn(__fmaf_rn(-q, sum, e), reciprocal, q);
}

// ---- a few warps per row -----------------------------------------------------------------------------
// kWarps warps hold a row, kVecs vectors per lane; with one warp per row a CTA has eight rows.
// HBM bound.  8192 x 4096 softmax: 16 warps with two vectors per lane took 58.6 us, four with eight take 43.5 (6.2 TB/s);
// 65,536 x 128: 69.6 us with 32 scalar loads per lane, 12.3 now.
// kAlike: a row of the result lies against the boundary like the row of the input; else it is written element by element.
template <bool kSoftmax, int kWarps, int kVecs, bool kAlike = true>
__global__ void __launch_bounds__(kWarps == 1 ? 256 : kWarps * 32) few_warps_kernel(const float* __restrict__ in, float* out, size_t rows,
                                                                                    size_t cols) {
    constexpr int T = kWarps * 32;
    const size_t row = kWarps == 1 ? (size_t)blockIdx.x * 8 + (threadIdx.x >> 5) : blockIdx.x;
    if (kWarps == 1 && row >= rows) return;
    const int tid = kWarps == 1 ? threadIdx.x & 31 : threadIdx.x, lane = tid & 31;
    __shared__ float s_max[kWarps], s_sum[kWarps];
    // the row as aligned vectors; what lies outside it in the first and the last of them is left out
    const float* x = in + row * cols;
    const int before = (int)((reinterpret_cast<uintptr_t>(x) >> 2) & 3), last = (before + (int)cols + 3) / 4 - 1;
    const int after = 4 * (last + 1) - before - (int)cols;
    const float4* x4 = reinterpret_cast<const float4*>(x - before);
    float4 v[kVecs];
    float m = -INFINITY;
#pragma unroll
    for (int k = 0; k < kVecs; ++k) {
        const int j = k * T + tid;
        v[k] = make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
        if (j <= last) v[k] = x4[j];
    }
#pragma unroll
    for (int k = 0; k < kVecs; ++k) {
        const int j = k * T + tid;
        if (k == 0 && j == 0) {
            if (before > 0) v[k].x = -INFINITY;
            if (before > 1) v[k].y = -INFINITY;
            if (before > 2) v[k].z = -INFINITY;
        }
        if (j == last) {
            if (after > 0) v[k].w = -INFINITY;
            if (after > 1) v[k].z = -INFINITY;
            if (after > 2) v[k].y = -INFINITY;
        }
        m = fmax3(fmax3(v[k].x, v[k].y, v[k].z), v[k].w, m);
    }
    m = warp_max(m);
    if (kWarps > 1) {
        if (lane == 0) s_max[tid >> 5] = m;
        __syncthreads();
        m = s_max[0];
#pragma unroll
        for (int w = 1; w < kWarps; ++w) m = fmaxf(m, s_max[w]);
    }
    float s = 0.0f;
#pragma unroll
    for (int k = 0; k < kVecs; ++k) {
        v[k].x = __expf(v[k].x - m); v[k].y = __expf(v[k].y - m); v[k].z = __expf(v[k].z - m); v[k].w = __expf(v[k].w - m);
        s += (v[k].x + v[k].y) + (v[k].z + v[k].w);
    }
    s = warp_sum_f(s);
    if (kWarps > 1) {
        if (lane == 0) s_sum[tid >> 5] = s;
        __syncthreads();
        s = 0.0f;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) s += s_sum[w];
    }
    if (kSoftmax) {
        const float r = __frcp_rn(s);
        float* y = out + row * cols - before;
#pragma unroll
        for (int k = 0; k < kVecs; ++k) {
            const int j = k * T + tid;
            if (j > last) continue;
            const float4 q = make_float4(quotient(v[k].x, s, r), quotient(v[k].y, s, r), quotient(v[k].z, s, r), quotient(v[k].w, s, r));
            if (!kAlike || (j == 0 && before > 0) || (j == last && after > 0)) {
                const float c[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (!(j == 0 && i < before) && !(j == last && i >= 4 - after)) y[4 * j + i] = c[i];
                }
            } else {
                reinterpret_cast<float4*>(y)[j] = q;
            }
        }
    } else if (tid == 0) {
        out[row] = m + logf(s);
    }
}

// ---- one cluster per row ---------------------------------------------------------------------------
// Block-wide max / sum in a fixed order; `scratch` holds one float per warp.
__device__ __forceinline__ float block_max_f(float v, float* scratch) {
    v = warp_max(v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = v;
    __syncthreads();
    float r = scratch[0];
#pragma unroll
    for (int w = 1; w < kCtaThreads / 32; ++w) r = fmaxf(r, scratch[w]);
    return r;
}
__device__ __forceinline__ float block_sum_f(float v, float* scratch) {
    v = warp_sum_f(v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = v;
    __syncthreads();
    float r = 0.0f;
#pragma unroll
    for (int w = 0; w < kCtaThreads / 32; ++w) r += scratch[w];
    return r;
}

template <bool kSoftmax, int kVecs>
__global__ void __launch_bounds__(kCtaThreads, kVecs <= 8 ? 2 : 1) cluster_rows_kernel(const float* __restrict__ in, float* out, size_t rows,
                                                                     size_t cols, int vector_ok) {
    cg::cluster_group cluster = cg::this_cluster();
    const unsigned ctas = cluster.num_blocks(), rank = cluster.block_rank();
    const size_t row = blockIdx.x / ctas;
    __shared__ float s_warp[kCtaThreads / 32];
    __shared__ float s_share[2];  // this CTA's maximum and sum, read by the others of the cluster
    const int tid = threadIdx.x;
    // the CTA's slice of the row: whole float4 vectors, the same count for every CTA but the last
    const size_t vecs = (cols + 3) / 4, per = (vecs + ctas - 1) / ctas;
    const size_t begin = min((size_t)rank * per * 4, cols), end = min(begin + per * 4, cols);
    const float* x = in + row * cols;
    float v[kVecs * 4];
    float m = -INFINITY;
    if (vector_ok) {  // rows start on 16-byte boundaries: cols % 4 == 0 and an aligned base
#pragma unroll
        for (int k = 0; k < kVecs; ++k) {
            const size_t j = begin + ((size_t)k * kCtaThreads + tid) * 4;
            float4 d = make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
            if (j < end) d = *reinterpret_cast<const float4*>(x + j);
            v[4 * k] = d.x; v[4 * k + 1] = d.y; v[4 * k + 2] = d.z; v[4 * k + 3] = d.w;
            m = fmaxf(fmaxf(m, fmaxf(d.x, d.y)), fmaxf(d.z, d.w));
        }
    } else {
#pragma unroll
        for (int k = 0; k < kVecs * 4; ++k) {
            const size_t j = begin + (size_t)k * kCtaThreads + tid;
            v[k] = j < end ? x[j] : -INFINITY;
            m = fmaxf(m, v[k]);
        }
    }
    m = block_max_f(m, s_warp);
    if (ctas > 1) {
        if (tid == 0) s_share[0] = m;
        cluster.sync();
        for (unsigned r = 0; r < ctas; ++r) m = fmaxf(m, *cluster.map_shared_rank(&s_share[0], r));
    }
    float s = 0.0f;
#pragma unroll
    for (int k = 0; k < kVecs * 4; ++k) {
        v[k] = __expf(v[k] - m);  // (slots past the slice hold -inf: they give 0)
        s += v[k];
    }
    s = block_sum_f(s, s_warp);
    if (ctas > 1) {
        if (tid == 0) s_share[1] = s;
        cluster.sync();
        s = 0.0f;
        for (unsigned r = 0; r < ctas; ++r) s += *cluster.map_shared_rank(&s_share[1], r);
        cluster.sync();  // nobody leaves while its shared memory may still be read
    }
    if (kSoftmax) {
        float* y = out + row * cols;
        const float q = __frcp_rn(s);
        if (vector_ok) {
#pragma unroll
            for (int k = 0; k < kVecs; ++k) {
                const size_t j = begin + ((size_t)k * kCtaThreads + tid) * 4;
                if (j < end) {
                    *reinterpret_cast<float4*>(y + j) =
                        make_float4(quotient(v[4 * k], s, q), quotient(v[4 * k + 1], s, q), quotient(v[4 * k + 2], s, q), quotient(v[4 * k + 3], s, q));
                }
            }
        } else {
#pragma unroll
            for (int k = 0; k < kVecs * 4; ++k) {
                const size_t j = begin + (size_t)k * kCtaThreads + tid;
                if (j < end) y[j] = quotient(v[k], s, q);
            }
        }
    } else if (rank == 0 && tid == 0) {
        out[row] = m + logf(s);
    }
}

// ---- rows beyond a cluster's reach: one CTA, three walks -----------------------------------------------
template <bool kSoftmax>
__global__ void __launch_bounds__(kCtaThreads) long_rows_kernel(const float* in, float* out, size_t rows, size_t cols) {
    __shared__ float s_warp[kCtaThreads / 32];
    const size_t row = blockIdx.x;
    const float* x = in + row * cols;
    float m = -INFINITY;
    for (size_t j = threadIdx.x; j < cols; j += kCtaThreads) m = fmaxf(m, x[j]);
    m = block_max_f(m, s_warp);
    float s = 0.0f;
    for (size_t j = threadIdx.x; j < cols; j += kCtaThreads) s += __expf(x[j] - m);
    s = block_sum_f(s, s_warp);
    if (kSoftmax) {
        float* y = out + row * cols;
        for (size_t j = threadIdx.x; j < cols; j += kCtaThreads) y[j] = __expf(x[j] - m) / s;  // (out may alias in: element by element)
    } else if (threadIdx.x == 0) {
        out[row] = m + logf(s);
    }
}

template <bool kSoftmax>
cudaError_t launch_rows(const float* in, float* out, size_t rows, size_t cols, cudaStream_t stream) {
    if (rows == 0 || cols == 0) return cudaSuccess;
    if (rows > 0x7FFFFFFFull / kMaxCluster) return cudaErrorInvalidConfiguration;
    const bool on_boundaries = cols % 4 == 0 && reinterpret_cast<uintptr_t>(in) % 16 == 0;
    const bool alike = !kSoftmax || (reinterpret_cast<uintptr_t>(in) - reinterpret_cast<uintptr_t>(out)) % 16 == 0;
    const size_t most = on_boundaries ? cols / 4 : (cols + 6) / 4;  // vectors a row spans
    // A result that lies differently against the boundary than the input is written element by element, up to where the cluster
    // kernel's scalar reads and writes take over (65,536 x 128: 416 -> 18.6 us, 4000 x 6001: 53.3 -> 39.1; 2000 x 12,001
    // would take 49.3 so and takes 45.1 there).
    if (most <= (alike ? (size_t)kCtaThreads * kCtaVecs : (size_t)2048)) {
        auto launch = [&](void (*like)(const float*, float*, size_t, size_t), void (*unlike)(const float*, float*, size_t, size_t), int warps) {
            const unsigned blocks = (unsigned)(warps == 1 ? (rows + 7) / 8 : rows);
            (alike ? like : unlike)<<<blocks, warps == 1 ? 256 : warps * 32, 0, stream>>>(in, out, rows, cols);
            return cudaGetLastError();
        };
        if (most <= 32) return launch(few_warps_kernel<kSoftmax, 1, 1>, few_warps_kernel<kSoftmax, 1, 1, !kSoftmax>, 1);
        if (most <= 64) return launch(few_warps_kernel<kSoftmax, 1, 2>, few_warps_kernel<kSoftmax, 1, 2, !kSoftmax>, 1);
        if (most <= 128) return launch(few_warps_kernel<kSoftmax, 1, 4>, few_warps_kernel<kSoftmax, 1, 4, !kSoftmax>, 1);
        if (most <= 256) return launch(few_warps_kernel<kSoftmax, 1, 8>, few_warps_kernel<kSoftmax, 1, 8, !kSoftmax>, 1);
        if (most <= 512) return launch(few_warps_kernel<kSoftmax, 4, 4>, few_warps_kernel<kSoftmax, 4, 4, !kSoftmax>, 4);
        if (most <= 1024) return launch(few_warps_kernel<kSoftmax, 4, 8>, few_warps_kernel<kSoftmax, 4, 8, !kSoftmax>, 4);
        if (most <= 2048) return launch(few_warps_kernel<kSoftmax, 8, 8>, few_warps_kernel<kSoftmax, 8, 8, !kSoftmax>, 8);
        if (most <= 4096) return launch(few_warps_kernel<kSoftmax, 16, 8>, nullptr, 16);
        return launch(few_warps_kernel<kSoftmax, 16, 16>, nullptr, 16);
    }
    if (cols > (size_t)kCtaCols * kMaxCluster) {
        long_rows_kernel<kSoftmax><<<(unsigned)rows, kCtaThreads, 0, stream>>>(in, out, rows, cols);
        return cudaGetLastError();
    }
    // half of a CTA's reach where eight CTAs will do
    const size_t reach = cols <= (size_t)kCtaCols / 2 * kMaxCluster ? kCtaCols / 2 : kCtaCols;
    const unsigned ctas = (unsigned)((cols + reach - 1) / reach);
    const bool aligned = cols % 4 == 0 && reinterpret_cast<uintptr_t>(in) % 16 == 0 &&
                         (!kSoftmax || reinterpret_cast<uintptr_t>(out) % 16 == 0);
    // a float4 slice per thread needs per-CTA slices of at most kCtaCols columns: true by the choice of `ctas`
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3((unsigned)rows * ctas);
    config.blockDim = dim3(kCtaThreads);
    config.stream = stream;
    cudaLaunchAttribute attribute[1];
    attribute[0].id = cudaLaunchAttributeClusterDimension;
    attribute[0].val.clusterDim.x = ctas;
    attribute[0].val.clusterDim.y = 1;
    attribute[0].val.clusterDim.z = 1;
    config.attrs = attribute;
    config.numAttrs = 1;
    // the fewest vectors per thread that cover a CTA's slice
    const size_t slice = ((cols + 3) / 4 + ctas - 1) / ctas;  // float4 vectors
    const int vec_ok = aligned ? 1 : 0;
    if (slice <= (size_t)kCtaThreads * 2) return cudaLaunchKernelEx(&config, cluster_rows_kernel<kSoftmax, 2>, in, out, rows, cols, vec_ok);
    if (slice <= (size_t)kCtaThreads * 4) return cudaLaunchKernelEx(&config, cluster_rows_kernel<kSoftmax, 4>, in, out, rows, cols, vec_ok);
    if (slice <= (size_t)kCtaThreads * 8) return cudaLaunchKernelEx(&config, cluster_rows_kernel<kSoftmax, 8>, in, out, rows, cols, vec_ok);
    return cudaLaunchKernelEx(&config, cluster_rows_kernel<kSoftmax, kCtaVecs>, in, out, rows, cols, vec_ok);
}

// ---- gather_rows -----------------------------------------------------------------------------------------
// One CTA per output row; 128-bit copies when the rows allow it.
__global__ void __launch_bounds__(256) gather_rows_kernel(const float* __restrict__ table, const float* __restrict__ indices,
                                                          float* __restrict__ out, size_t count, size_t dim, int vector_ok) {
    for (size_t i = blockIdx.x; i < count; i += gridDim.x) {
        const float* row = table + (size_t)indices[i] * dim;  // whole-number floats, as the reference passes them
        float* dst = out + i * dim;
        if (vector_ok) {
            for (size_t d = threadIdx.x; d < dim / 4; d += blockDim.x) {
                reinterpret_cast<float4*>(dst)[d] = reinterpret_cast<const float4*>(row)[d];
            }
        } else {
            for (size_t d = threadIdx.x; d < dim; d += blockDim.x) dst[d] = row[d];
        }
    }
}

}  // namespace

cudaError_t launch_softmax_rows(const float* in, float* out, size_t rows, size_t cols, cudaStream_t stream) {
    return launch_rows<true>(in, out, rows, cols, stream);
}

cudaError_t launch_logsumexp_rows(const float* in, float* out, size_t rows, size_t cols, cudaStream_t stream) {
    return launch_rows<false>(in, out, rows, cols, stream);
}

cudaError_t launch_gather_rows(const float* table, const float* indices, float* out, size_t count, size_t dim,
                               cudaStream_t stream) {
    if (count == 0 || dim == 0) return cudaSuccess;
    const bool aligned = dim % 4 == 0 && reinterpret_cast<uintptr_t>(table) % 16 == 0 && reinterpret_cast<uintptr_t>(out) % 16 == 0;
    const unsigned blocks = (unsigned)(count < 65535u * 16u ? count : 65535u * 16u);
    gather_rows_kernel<<<blocks, 256, 0, stream>>>(table, indices, out, count, dim, aligned ? 1 : 0);
    return cudaGetLastError();
}

}  // namespace psx
