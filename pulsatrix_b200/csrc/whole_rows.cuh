// Launch interface of sampling from the whole distribution (whole_rows.cu).
#pragma once

#include "psx_device.cuh"

struct psx_row_diag;  // include/psx_b200.h

namespace psx {

constexpr int kSegmentVecs = 128;  // float4 vectors of a segment: four per lane of the warp that weighs it

// What a warp reports about its segment of a row.
struct SegmentStats {
    double raw_sum;   // sum of exp(l - raw_max) over the segment's logits
    double mass;      // sum of exp(y - y_max) over its processed logits
    float raw_max;
    float y_max;      // after penalty, ban and temperature; -inf when everything is banned
    uint32_t alive;   // logits whose processed value is above -inf
    uint32_t nonfinite;
};

struct WholeRowParams {
    const float* logits;
    int64_t row_stride;
    int64_t rows;
    int64_t vocab;
    const int64_t* history_ids;      // null: no repetition penalty
    const int64_t* history_offsets;
    const int64_t* banned_ids;
    int32_t num_banned;
    float penalty;
    int32_t apply_temperature;
    float temperature;
    int32_t segments;                // per row
    int32_t segments_per_warp;       // filled in by launch_whole_rows
    int32_t inputs_ready;            // as in ScanParams
    SegmentStats* stats;             // rows * segments; another set than the call before, as ScanParams::wait_before_writes = 0 wants
    const double* uniforms;
    int64_t* tokens;
    float* log_probs;
    int32_t* row_status;
    psx_row_diag* diag;              // may be null
};

// The segments a row of `vocab` logits is cut into, whatever its alignment.
inline int64_t whole_row_segments(int64_t vocab) { return ((vocab + 3 + 3) / 4 + kSegmentVecs - 1) / kSegmentVecs; }
cudaError_t launch_whole_rows(const WholeRowParams& p, cudaStream_t stream);  // two kernels

}  // namespace psx
