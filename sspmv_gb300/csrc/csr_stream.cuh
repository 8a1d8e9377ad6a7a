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
    int32_t nshared = 0;  // nempty where the stream kernel's windows write those rows, else 0
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
// elements where the caller has counted them and no row is split (-1: counted
// here, which waits for the device); counted: if there are any, per tile of
// stream_tile_rows(m) rows, .x of those with elements.
int64_t stream_tile_rows(int64_t m);  // a multiple of 1024
sspmv_status ensure_stream_plan(StreamPlan &sp, int64_t m, int64_t nnz, const int32_t *row_offset,
                                const int32_t *row_map, int32_t value_type, sspmv_stream_t s, int window = 0,
                                int over = -1, int64_t nempty = -1, const int2 *counted = nullptr);
void free_stream_plan(StreamPlan &sp, sspmv_stream_t s);
StreamView stream_view(const StreamPlan &sp, int64_t nnz, const int32_t *col, const void *val);

// KL values to p, one vector store when `vec` (p aligned to it).
template <typename V, int KL, bool BIG = false>
__device__ __forceinline__ void st_cols(V *__restrict__ p, bool vec, const V (&o)[KL]) {
    if constexpr (KL * sizeof(V) == 16) {
        if (vec) {
            if constexpr (sizeof(V) == 8) {
                const double2 v = make_double2(o[0], o[1]);
                if constexpr (BIG) __stcs(reinterpret_cast<double2 *>(p), v);  // leaves L2 to X
                else *reinterpret_cast<double2 *>(p) = v;
            } else {
                const float4 v = make_float4(o[0], o[1], o[2], o[3]);
                if constexpr (BIG) __stcs(reinterpret_cast<float4 *>(p), v);
                else *reinterpret_cast<float4 *>(p) = v;
            }
            return;
        }
    }
#pragma unroll
    for (int q = 0; q < KL; q++) p[q] = o[q];
}

// The rows without nonzeros are a list of the plan, taken by warps of their own
// behind the windows' in the same launch, kEmptyUnit entries each: eight rows a
// group of lanes in flight together, 16 bytes of a row of Y a lane.  4M rows with
// 10k nonzeros, FP64, 9.4 us (with alpha and beta 14.5): shared out to the
// windows, which are as few as the nonzeros, 473 us (1616); 1M rows with 5% empty
// 85.4 shared and 84.0 so, 7267 rows with 363 empty (714 windows) 3.9 and 3.5.
// Only a list of at most an eighth of the windows is left to those, a row each.
constexpr int kEmptyUnit = 256;
inline __host__ __device__ int64_t empty_units(int64_t nempty) { return (nempty + kEmptyUnit - 1) / kEmptyUnit; }

template <typename V, int K>
__device__ __forceinline__ void scale_empty_rows(const StreamView &A, int64_t unit, V beta, V *__restrict__ y,
                                                 uint64_t yrow, bool yvec) {
    constexpr int G = K * (int)sizeof(V) > 16 ? K * (int)sizeof(V) / 16 : 1;  // lanes per row of Y
    constexpr int KL = K / G, NG = 32 / G;
    const int lane = threadIdx.x & 31, gi = lane / G;
    const int64_t i0 = unit * kEmptyUnit;
    char *yq = reinterpret_cast<char *>(y + (lane % G) * KL);
    for (int j = 0; j < kEmptyUnit; j += 8 * NG) {
        int row[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int64_t i = i0 + j + u * NG + gi;
            row[u] = i < A.nempty ? __ldcs(A.empty + i) : -1;
        }
        V old[8][KL];
#pragma unroll
        for (int u = 0; u < 8; u++)
#pragma unroll
            for (int q = 0; q < KL; q++)
                old[u][q] = beta != V(0) && row[u] >= 0
                                ? reinterpret_cast<const V *>(yq + (uint64_t)(uint32_t)row[u] * yrow)[q] : V(0);
#pragma unroll
        for (int u = 0; u < 8; u++) {
            if (row[u] < 0) continue;
#pragma unroll
            for (int q = 0; q < KL; q++) old[u][q] = beta == V(0) ? V(0) : beta * old[u][q];
            st_cols<V, KL>(reinterpret_cast<V *>(yq + (uint64_t)(uint32_t)row[u] * yrow), yvec, old[u]);
        }
    }
}

// Rows of at most this many elements are never split (0, -1 for window, over).
constexpr int kStreamWholeRow = 33;

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
