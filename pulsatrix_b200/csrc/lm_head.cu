// The language-model head on the device: logits[m][j] = sum_p hidden[m][p] * w_j[p], the step right
// before the sampling path (src/tied_lm_head_module.cpp:31-53: gemm_ex(hidden, E^T); an untied head
// is a bias-free Linear, src/linear_module.cpp: gemm(hidden, W)).
//
// Exact by construction: the reference's CPU backend forms every logit as one float accumulator
// that takes the products in ascending p, each product rounded, then the sum rounded
// (src/cpu_backend.cpp:188-196 and GemmRowRange; its x86-64 build has no fused multiply-add).  A
// thread here owns a few vocabulary entries and a few rows of hidden states, and does exactly that for each pair: a
// rounded product, a rounded sum, p ascending.  The logits are therefore the reference's bit for bit,
// and so is every token drawn from them.  (Tensor cores would round differently -- TF32 products,
// tree-shaped sums -- so they are not used here.)
//
// Bound: from about 12 rows up the FP32 pipes (two operations per multiply-add, 128 lanes per SM: 17.4 T of them a
// second, 1.14 ms for 64 rows of 151,936 x 2048), below by HBM -- the weights are read once, 4 * vocab * d bytes.  What
// has to stay out of the way of either:
//   - shared-memory reads.  A 128-bit read occupies the pipe for four cycles even where all lanes read the same
//     address, so a thread that owns one entry waits for hidden states (sixteen reads per feature for 64 rows, against
//     128 operations: 2.7 ms for 64 rows).  With four entries by up to sixteen rows per thread the reads take 60 % of the
//     time that the operations do: 1.54 ms, 0.81 of the pipe's rate in the full rounds.
//   - issue slots.  Two rows go through one packed operation (f32x2): the FP32 pipe is as busy, the issue slots are half
//     free for the reads.  The product is fma.rn.f32x2(h, w, -0.0), which is the rounded product (x + -0.0 = x for
//     every x, zeros of either sign among them), with the -0.0 from the kernel's arguments: a mul.rn.f32x2 ahead of an
//     add.rn.f32x2 is contracted into one fused operation by the compiler whatever its rounding suffix says.
//   - an empty last round.  The CTAs are as many as the GPU holds, each works through whole tiles of 128 entries a
//     warp (256 in the layouts of eight entries per lane), and what is left after the last full round is handed out in tiles of 32 entries
//     a warp or a multiple of it, the smallest that goes round once (151,936 entries are 2.005 rounds of 256 x 296: a third round of
//     whole tiles would take half as long again); see Head::kBalanced for one and two rows.
// The weights arrive by cp.async, S chunks of features deep; the hidden states of a chunk come with them,
// 4 bytes at a time, transposed on the way ([feature][row]), so that a pair of rows is one 64-bit operand.
// Two weight layouts:
//   - token-major (vocab x d, the tied embedding): staged [entry][feature], a lane's entries 32 apart, four features
//     of an entry per read (pitch of 4 floats more than the chunk: eight lanes' reads fall into distinct banks);
//   - feature-major (d x vocab, an untied Linear): staged [feature][entry], a lane's entries side by side, one read.
#include "lm_head.cuh"

#include <algorithm>

#include <cuda_pipeline_primitives.h>

#include "psx_device.cuh"

namespace psx {

namespace {

struct HeadParams {
    const float* hidden;
    const float* weight;
    float* logits;
    int rows;
    int64_t d, vocab, row_stride;
    int width;            // balanced: entries of a CTA's tile
    int vector_ok;        // the weights may be copied 16 bytes at a time
    int full_rounds;      // rounds of whole tiles (kEntries per lane)
    int last_entries;     // entries per lane in the round after them (0: none)
    float minus_zero;
};

typedef unsigned long long pair32;  // two floats, the lower one in the lower half

__device__ __forceinline__ pair32 make_pair32(float lo, float hi) {
    pair32 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void split_pair32(pair32 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
// acc + h * w in both halves, the product rounded and the sum rounded (minus_zero: {-0.0, -0.0}, unknown to the compiler).
__device__ __forceinline__ void multiply_add(pair32& acc, pair32 h, pair32 w, pair32 minus_zero) {
    pair32 product;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(product) : "l"(h), "l"(w), "l"(minus_zero));
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(acc) : "l"(product));
}

// R: rows per thread; G: row groups (warps that share their entries); H: warps side by side along the vocabulary;
// KC: features per chunk; S: chunks in flight and at work.
template <int R, int G, int H, int KC, int S, int EM, bool kTokenMajor>
struct Head {
    static constexpr int kThreads = 32 * G * H;
    static constexpr int kRows = R * G;
    static constexpr int kUnroll = 4;                // sixteen features a turn
    static constexpr int kTile = 32 * EM * H;  // entries of a whole tile of the CTA
    static constexpr int kPitch = KC + 4;            // token-major: floats per staged entry
    static constexpr int kWeightFloats = kTokenMajor ? kTile * kPitch : KC * kTile;
    static constexpr int kStageFloats = kWeightFloats + KC * kRows;
    static constexpr size_t kSharedBytes = (size_t)S * kStageFloats * sizeof(float);
    // One or two rows of a token-major head: every CTA gets the same share of the vocabulary, in tiles that may leave
    // lanes idle (151,936 entries are 4.01 rounds of 128 x 296; the weights' traffic is the bound, not the lanes: 243 -> 215 us).
    // A feature-major head loses more by copies that start off the 128-byte lines than it gains.
    static constexpr bool kBalanced = kTokenMajor && R * G <= 2;

    // Asks for chunk c of the E * 32 * H entries from j0 on, and for the rows' hidden states of the chunk.
    template <int E>
    static __device__ __forceinline__ void stage(const HeadParams& p, float* buffer, int64_t j0, int c) {
        constexpr int kRowFloats = 32 * E * H;                   // feature-major: floats per staged feature
        const int width = kBalanced ? p.width : kRowFloats;
        const int tid = threadIdx.x;
        const int64_t k0 = (int64_t)c * KC;
        const int kc = (int)min((int64_t)KC, p.d - k0);
        if (kTokenMajor) {
            if (p.vector_ok && kc == KC) {
                constexpr int kPieces = KC / 4;
#pragma unroll 8
                for (int q = tid; q < width * kPieces; q += kThreads) {
                    const int r = q / kPieces, piece = q % kPieces;
                    const int64_t j = min(j0 + r, p.vocab - 1);  // (past the vocabulary: the last entry again, never stored)
                    __pipeline_memcpy_async(buffer + r * kPitch + piece * 4, p.weight + j * p.d + k0 + piece * 4, 16);
                }
            } else {
                for (int q = tid; q < width * KC; q += kThreads) {
                    const int r = q / KC, f = q % KC;
                    const int64_t j = min(j0 + r, p.vocab - 1);
                    if (f < kc) __pipeline_memcpy_async(buffer + r * kPitch + f, p.weight + j * p.d + k0 + f, 4);
                }
            }
        } else {
            if (p.vector_ok && j0 + width <= p.vocab && width % 4 == 0) {
                const int pieces = width / 4;
#pragma unroll 8
                for (int q = tid; q < KC * pieces; q += kThreads) {
                    const int f = q / pieces, piece = q % pieces;
                    if (f < kc) __pipeline_memcpy_async(buffer + f * kRowFloats + piece * 4, p.weight + (k0 + f) * p.vocab + j0 + piece * 4, 16);
                }
            } else {
                for (int q = tid; q < KC * width; q += kThreads) {
                    const int f = q / width, r = q % width;
                    const int64_t j = min(j0 + r, p.vocab - 1);
                    if (f < kc) __pipeline_memcpy_async(buffer + f * kRowFloats + r, p.weight + (k0 + f) * p.vocab + j, 4);
                }
            }
        }
        float* h = buffer + kWeightFloats;
        for (int q = tid; q < p.rows * KC; q += kThreads) {
            const int m = q / KC, f = q % KC;
            if (f < kc) __pipeline_memcpy_async(h + f * kRows + m, p.hidden + (int64_t)m * p.d + k0 + f, 4);
        }
    }

    // The products of one feature with this thread's rows, for E entries.
    template <int E>
    static __device__ __forceinline__ void take(pair32 (&acc)[E][(R + 1) / 2], float (&single)[E], const float* h, const float (&w)[E], pair32 minus_zero) {
        if (R == 1) {
#pragma unroll
            for (int e = 0; e < E; ++e) single[e] = __fadd_rn(single[e], __fmul_rn(h[0], w[e]));
        } else {
            pair32 h2[(R + 1) / 2];
            if (R >= 4) {
#pragma unroll
                for (int r = 0; r < R / 4; ++r) {
                    const ulonglong2 v = reinterpret_cast<const ulonglong2*>(h)[r];
                    h2[2 * r] = v.x;
                    h2[2 * r + 1] = v.y;
                }
            } else {
                h2[0] = *reinterpret_cast<const pair32*>(h);
            }
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const pair32 w2 = make_pair32(w[e], w[e]);
#pragma unroll
                for (int r = 0; r < R / 2; ++r) multiply_add(acc[e][r], h2[r], w2, minus_zero);
            }
        }
    }

    // Tiles j0, j0 + step, ... (count of them) of E entries per lane.
    template <int E>
    static __device__ __forceinline__ void tiles(const HeadParams& p, float* shared, int64_t j0, int64_t step, int count) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, group = warp % G, side = warp / G;
        const int chunks = (int)((p.d + KC - 1) / KC);
        const pair32 minus_zero = make_pair32(p.minus_zero, p.minus_zero);
        pair32 acc[E][(R + 1) / 2];
        float single[E];
        auto clear = [&]() {
#pragma unroll
            for (int e = 0; e < E; ++e) {
                single[e] = 0.0f;
#pragma unroll
                for (int r = 0; r < (R + 1) / 2; ++r) acc[e][r] = 0ull;
            }
        };
        clear();
        // One stream of chunks over all the tiles: what is asked for next may belong to the next tile.
        int ask_chunk = 0, ask_tile = 0, ask_slot = 0;
        auto ask = [&]() {
            if (ask_tile < count) {
                stage<E>(p, shared + ask_slot * kStageFloats, j0 + ask_tile * step, ask_chunk);
                if (++ask_chunk == chunks) { ask_chunk = 0; ++ask_tile; }
                ask_slot = ask_slot + 1 == S ? 0 : ask_slot + 1;
            }
            __pipeline_commit();
        };
        for (int i = 0; i < S - 1; ++i) ask();
        int slot = 0;
        for (int tile = 0; tile < count; ++tile) {
            for (int c = 0; c < chunks; ++c) {
                __pipeline_wait_prior(S - 2);
                __syncthreads();  // the chunk has landed for everybody, and everybody has finished with the slot asked for below
                ask();
                const float* buffer = shared + slot * kStageFloats;
                const float* h = buffer + kWeightFloats + group * R;
                slot = slot + 1 == S ? 0 : slot + 1;
                const int kc = (int)min((int64_t)KC, p.d - (int64_t)c * KC);
                if (kTokenMajor) {
                    const float* mine = buffer + (side * 32 * E + lane) * kPitch;
                    if (kc == KC) {
#pragma unroll(kUnroll)
                        for (int f = 0; f < KC; f += 4) {
                            float4 w4[E];
#pragma unroll
                            for (int e = 0; e < E; ++e) w4[e] = *reinterpret_cast<const float4*>(mine + e * 32 * kPitch + f);
                            float w[E];
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
#pragma unroll
                                for (int e = 0; e < E; ++e) w[e] = i == 0 ? w4[e].x : i == 1 ? w4[e].y : i == 2 ? w4[e].z : w4[e].w;
                                take<E>(acc, single, h + (f + i) * kRows, w, minus_zero);
                            }
                        }
                    } else {  // the last, shorter chunk: no padded products (they could turn a -0 sum into +0)
                        for (int f = 0; f < kc; ++f) {
                            float w[E];
#pragma unroll
                            for (int e = 0; e < E; ++e) w[e] = mine[e * 32 * kPitch + f];
                            take<E>(acc, single, h + f * kRows, w, minus_zero);
                        }
                    }
                } else {
                    const float* mine = buffer + side * 32 * E + lane * E;
#pragma unroll(4 * kUnroll)
                    for (int f = 0; f < KC; ++f) {
                        if (f < kc) {
                            float w[E];
                            if (E % 4 == 0) {
#pragma unroll
                                for (int e = 0; e + 3 < E; e += 4) {
                                    const float4 v = *reinterpret_cast<const float4*>(mine + f * 32 * E * H + e);
                                    w[e] = v.x; w[e + 1] = v.y; w[e + 2] = v.z; w[e + 3] = v.w;
                                }
                            } else {
#pragma unroll
                                for (int e = 0; e < E; ++e) w[e] = mine[f * 32 * E * H + e];
                            }
                            take<E>(acc, single, h + f * kRows, w, minus_zero);
                        }
                    }
                }
            }
            const int64_t first = j0 + tile * step + side * 32 * E, end = kBalanced ? min(p.vocab, j0 + tile * step + p.width) : p.vocab;
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const int64_t j = first + (kTokenMajor ? e * 32 + lane : lane * E + e);
                if (j < end) {
                    if (R == 1) {
                        p.logits[(int64_t)group * p.row_stride + j] = single[e];
                    } else {
#pragma unroll
                        for (int r = 0; r < R / 2; ++r) {
                            float lo, hi;
                            split_pair32(acc[e][r], lo, hi);
                            const int m = group * R + 2 * r;
                            if (m < p.rows) p.logits[(int64_t)m * p.row_stride + j] = lo;
                            if (m + 1 < p.rows) p.logits[(int64_t)(m + 1) * p.row_stride + j] = hi;
                        }
                    }
                }
            }
            clear();
        }
        __syncthreads();  // (the next call starts with its slots from the beginning)
    }
};

// The tiles of the last round: E to EM entries per lane, as many as it says.
template <class K, int E, int EM, bool kTokenMajor>
__device__ __forceinline__ void last_tiles(const HeadParams& p, float* shared, int64_t j0) {
    if constexpr (E < EM) {
        if (p.last_entries > E) return last_tiles<K, E + 1, EM, kTokenMajor>(p, shared, j0);
    }
    if constexpr (EM == 8 && !kTokenMajor) {
        // A last tile that is not whole would come in 4 bytes at a time, and the wider it is the longer the others would wait for it: it is moved back,
        // onto entries that its neighbour forms as well, bit for bit.  (48 rows of 65,536 x 2048, feature-major: 874 and 480 us.)
        constexpr int kWidth = K::kTile / EM * E;
        if (p.vector_ok && p.vocab >= kWidth) j0 = min(j0, p.vocab - kWidth);
    }
    K::template tiles<E>(p, shared, j0, 0, 1);
}

template <int R, int G, int H, int KC, int S, int kCtas, int EM, bool kTokenMajor>
__global__ void __launch_bounds__(32 * G * H, kCtas) head_kernel(const __grid_constant__ HeadParams p) {
    typedef Head<R, G, H, KC, S, EM, kTokenMajor> K;
    extern __shared__ __align__(16) float head_shared[];
    if (p.rows < K::kRows) {  // rows that are not there multiply by zero
        for (int i = threadIdx.x; i < S * KC * K::kRows; i += K::kThreads) {
            const int slot = i / (KC * K::kRows), at = i % (KC * K::kRows);
            if (at % K::kRows >= p.rows) head_shared[slot * K::kStageFloats + K::kWeightFloats + at] = 0.0f;
        }
    }
    if (K::kBalanced) {
        const int64_t j0 = (int64_t)blockIdx.x * p.width, step = (int64_t)gridDim.x * p.width;
        if (j0 < p.vocab) K::template tiles<EM>(p, head_shared, j0, step, (int)((p.vocab - j0 + step - 1) / step));
        return;
    }
    const int64_t round = (int64_t)gridDim.x * K::kTile;
    if (p.full_rounds > 0) K::template tiles<EM>(p, head_shared, (int64_t)blockIdx.x * K::kTile, round, p.full_rounds);
    const int64_t j0 = p.full_rounds * round + (int64_t)blockIdx.x * 32 * p.last_entries * H;
    if (p.last_entries == 0 || j0 >= p.vocab) return;
    last_tiles<K, 1, EM, kTokenMajor>(p, head_shared, j0);
}

template <int R, int G, int H, int KC, int S, int kCtas, int EM, bool kTokenMajor>
cudaError_t launch_one(HeadParams p, int sm_count, cudaStream_t stream) {
    typedef Head<R, G, H, KC, S, EM, kTokenMajor> K;
    const auto kernel = head_kernel<R, G, H, KC, S, kCtas, EM, kTokenMajor>;
    static OncePerDevice configured;  // (per instantiation)
    if (const cudaError_t e = allow_all_dynamic_shared_once(configured, kernel); e != cudaSuccess) return e;
    // Every CTA that the GPU holds at once takes whole tiles round after round; the rest goes round once, in the
    // smallest tiles with which it does.
    const int64_t lanes = 32 * H;  // entries of a CTA's tile per entry of a lane
    const int64_t slots = (int64_t)sm_count * kCtas;
    if (K::kBalanced) {
        const int64_t rounds = (p.vocab + slots * K::kTile - 1) / (slots * K::kTile), share = (p.vocab + slots * rounds - 1) / (slots * rounds);
        p.width = (int)((share + 3) / 4 * 4);
        kernel<<<(unsigned)std::min(slots, (p.vocab + p.width - 1) / p.width), K::kThreads, K::kSharedBytes, stream>>>(p);
        return cudaGetLastError();
    }
    p.full_rounds = (int)(p.vocab / (slots * K::kTile));
    const int64_t rest = p.vocab - p.full_rounds * slots * K::kTile;
    p.last_entries = (int)((rest + slots * lanes - 1) / (slots * lanes));
    const int64_t grid = p.full_rounds > 0 ? slots : (rest + lanes * p.last_entries - 1) / (lanes * p.last_entries);
    kernel<<<(unsigned)grid, K::kThreads, K::kSharedBytes, stream>>>(p);
    return cudaGetLastError();
}

template <bool kTokenMajor>
cudaError_t launch_group(const HeadParams& p, int sm_count, cudaStream_t stream) {
    // Rows per thread, row groups, warps along the vocabulary; features per chunk, chunks; CTAs per SM; entries per lane.
    // The fastest of the layouts that were timed (the logits alone, us; token-major / feature-major of 151,936 x 2048, then of 32,000 x 4096;
    // behind the bar the next wider layout, which these rows had before there was one for them):
    //    1 row    204 / 201                                        8 rows   295 / 306    206 / 250
    //    6 rows   288 / 304    150 / 248  |  293 / 304   203 / 248     12 rows   392 / 428    207 / 300  |  459 / 438   293 / 334
    //   16 rows   447 / 443    246 / 354                          24 rows   641 / 658    383 / 373  |  806 / 877   448 / 475
    //   32 rows   786 / 898    441 / 504                          48 rows  1207 / 1203   586 / 576  | 1479 / 1457  819 / 846
    //   64 rows  1512 / 1504   824 / 861
    // Up to two rows a lane takes one entry, which leaves room for longer runs of an entry's features per chunk (256 bytes:
    // HBM serves 5.9 TB/s in runs of 256 bytes, 5.0 in runs of 128); from four rows on the reads of the hidden states weigh, so four, or eight
    // where the rows leave the registers for it.  Token-major, up to 16 rows, chunks of 32 features gain for the same reason (16 rows: 463 us and
    // 308 with 16 features); feature-major a chunk of 32 is more rows of the matrix and no longer a run (9 to 12 rows: 537 us for 428).
    // groups: what an SM has of the vocabulary, in the 64 entries that a CTA takes per entry of a lane.  Where the next wider layout fills its rounds better it
    // is the faster one all the same (2048 features, us, the layout of the row count and the wider one): token-major, 16 rows, 100,000 entries (11 groups) 338 and 325;
    // 32 rows, 16,000 (2) 175 and 165, 80,000 (9) 469 and 452, 151,552 (16) 788 and 778, 227,328 of 1024 features (24) 683 and 587, but 100,000 (11) 574 and 626;
    // feature-major, 12 rows, 90,000 (10) 441 and 430; 24 rows, 80,000 (9) 502 and 481, and where the copies are of 4 bytes 75,777 (9) 760 and 617, 90,001 (10) 887
    // and 736, 130,001 (14) 1180 and 1087, but 100,001 (11) 825 and 879.
    const int64_t lanes = 64 * (int64_t)sm_count, groups = (p.vocab + lanes - 1) / lanes;
    if (p.rows <= 1) return kTokenMajor ? launch_one<1, 1, 4, 64, 2, 3, 1, true>(p, sm_count, stream) : launch_one<1, 1, 4, 32, 4, 3, 1, false>(p, sm_count, stream);
    if (p.rows <= 2) return kTokenMajor ? launch_one<2, 1, 4, 64, 2, 3, 1, true>(p, sm_count, stream) : launch_one<2, 1, 4, 32, 3, 3, 1, false>(p, sm_count, stream);
    if (p.rows <= 4) return launch_one<2, 2, 2, 32, 2, 3, 4, kTokenMajor>(p, sm_count, stream);
    if (kTokenMajor && p.rows <= 6) return launch_one<2, 3, 2, 32, 2, 3, 4, true>(p, sm_count, stream);
    if (p.rows <= 8) return launch_one<4, 2, 2, 16, 2, 4, 4, kTokenMajor>(p, sm_count, stream);
    if (p.rows <= 12 && kTokenMajor) return launch_one<4, 3, 2, 32, 2, 2, 4, true>(p, sm_count, stream);
    if (p.rows <= 12 && !(groups >= 9 && groups <= 12)) return launch_one<4, 3, 2, 16, 2, 4, 4, false>(p, sm_count, stream);
    if (p.rows <= 16) return kTokenMajor && groups != 11 && groups != 12 ? launch_one<8, 2, 2, 32, 2, 2, 4, true>(p, sm_count, stream)
                                                                                        : launch_one<8, 2, 2, 16, 2, 4, 4, kTokenMajor>(p, sm_count, stream);
    const bool wider_24 = !kTokenMajor && (groups == 9 || (!p.vector_ok && (groups == 10 || groups == 14)));
    if (p.rows <= 24 && !wider_24) return launch_one<4, 6, 2, 16, 2, 2, 8, kTokenMajor>(p, sm_count, stream);
    if (p.rows <= 32) {
        const bool eight = kTokenMajor && p.rows > 24 && ((groups >= 3 && groups <= 6) || (groups >= 10 && groups <= 14) || (groups >= 17 && groups <= 22));
        return eight ? launch_one<16, 2, 2, 16, 2, 2, 8, true>(p, sm_count, stream) : launch_one<8, 4, 2, 16, 3, 2, 4, kTokenMajor>(p, sm_count, stream);
    }
    if (p.rows <= 48) return launch_one<8, 6, 2, 16, 2, 1, 8, kTokenMajor>(p, sm_count, stream);
    return launch_one<16, 4, 2, 16, 3, 2, 4, kTokenMajor>(p, sm_count, stream);
}

}  // namespace

cudaError_t launch_lm_head(const float* hidden, int64_t rows, int64_t d, const float* weight, int64_t vocab, bool token_major,
                           float* logits, int64_t row_stride, int sm_count, cudaStream_t stream) {
    if (rows <= 0 || vocab <= 0) return cudaSuccess;
    if (d <= 0 || (d + 15) / 16 > 0x7FFFFFFF || vocab > (int64_t(1) << 38)) return cudaErrorInvalidValue;
    HeadParams p{};
    p.weight = weight;
    p.d = d;
    p.vocab = vocab;
    p.row_stride = row_stride;
    p.vector_ok = (token_major ? d : vocab) % 4 == 0 && reinterpret_cast<uintptr_t>(weight) % 16 == 0 ? 1 : 0;
    p.minus_zero = -0.0f;
    // Rows go through in groups of up to 64; every group reads the weights once.
    for (int64_t m0 = 0; m0 < rows; m0 += 64) {
        p.rows = (int)std::min<int64_t>(64, rows - m0);
        p.hidden = hidden + m0 * d;
        p.logits = logits + m0 * row_stride;
        const cudaError_t e = token_major ? launch_group<true>(p, sm_count, stream) : launch_group<false>(p, sm_count, stream);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace psx
