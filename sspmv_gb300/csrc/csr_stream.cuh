// csr_stream.cuh -- the nonzero-split stream kernel (csr_stream.cu): device
// view of a row-ordered run of nonzeros, its plan and its launchers.  Used by
// CSR (default kernel), the long rows of the sliced formats and the request
// server's batches.
#pragma once

#include "common.cuh"
#include "plan.cuh"

namespace sspmv {

// What the kernel reads besides x and y: the nonzeros in row order and the
// plan's arrays (StreamPlan).
struct StreamView {
    const int32_t *col = nullptr;
    const void *val = nullptr;
    const int4 *rec = nullptr;
    const int4 *split = nullptr;
    const uint8_t *ends = nullptr;
    const int32_t *nzrow = nullptr;
    const int32_t *empty = nullptr;
    int64_t windows = 0;
    uint32_t nnz = 0;
    int32_t window = 0;
    int32_t nempty = 0;
    int32_t nsplit = 0;
    int32_t vec = 0;  // 16-byte aligned col and val: vector loads
};

// Steps per window (1 to 5) for nnz elements in steps of `step`, the first of
// `first` elements, and warps_per_sm warps at once.
int window_steps(int64_t nnz, int step, int first, int warps_per_sm);

// Builds (once) the stream plan of m rows given by row_offset (m + 1
// entries, nnz > 0); row_offset is not read after the call's work on `s`.
// row_map: y row of each row (rows then all nonempty; null: the row itself),
// owned by the caller and kept as long as the plan.
// window, over: elements per window and past it that its warp may read to
// finish a row (0, -1: the stream kernel's own).  nempty: the rows without
// elements where the caller has counted them and `over` leaves no row to split
// (-1: counted here, which waits for the device).
sspmv_status ensure_stream_plan(StreamPlan &sp, int64_t m, int64_t nnz, const int32_t *row_offset,
                                const int32_t *row_map, int32_t value_type, sspmv_stream_t s, int window = 0,
                                int over = -1, int64_t nempty = -1);
void free_stream_plan(StreamPlan &sp, sspmv_stream_t s);
StreamView stream_view(const StreamPlan &sp, int64_t nnz, const int32_t *col, const void *val);

// The kernel steps through X and Y in 32-bit byte strides.
inline bool stream_takes_strides(int64_t ldx, int64_t ldy, size_t value_bytes) {
    return (uint64_t)ldx * value_bytes <= 0xffffffffu && (uint64_t)ldy * value_bytes <= 0xffffffffu;
}

// Y = alpha * A * X + beta * Y on the rows of the plan, K right-hand sides
// (1, 2, 4 or 8), but for the split rows, whose pieces it leaves: one launch.
// cols: rows of X.
template <typename V, int K>
sspmv_status launch_stream_windows(const StreamView &v, StreamPlan &sp, V alpha, const V *x, int64_t ldx, V beta,
                                   V *y, int64_t ldy, int64_t cols, sspmv_stream_t s);

// Finishes the rows whose pieces a kernel over the plan's windows has left in
// tail_val and head_val: one launch, none without such rows.  It follows that
// kernel (or one launched behind it) directly and starts under its last wave.
template <typename V, int K>
sspmv_status launch_split_rows(const StreamView &v, StreamPlan &sp, V alpha, V beta, V *y, int64_t ldy,
                               sspmv_stream_t s);

template <typename V, int K>
inline sspmv_status launch_stream_view(const StreamView &v, StreamPlan &sp, V alpha, const V *x, int64_t ldx, V beta,
                                       V *y, int64_t ldy, int64_t cols, sspmv_stream_t s) {
    SSPMV_TRY((launch_stream_windows<V, K>(v, sp, alpha, x, ldx, beta, y, ldy, cols, s)));
    return launch_split_rows<V, K>(v, sp, alpha, beta, y, ldy, s);
}

}  // namespace sspmv
