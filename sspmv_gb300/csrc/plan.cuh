// plan.cuh -- library-private per-matrix state hung off sspmv_features.priv.
//
// A plan caches what depends only on the sparsity structure (windows of the
// stream kernel, carry buffers, chosen launch shapes).  It is built on
// the first SpMV of a matrix (or by the converter that made the matrix) and
// freed by sspmv_delete_<fmt>.  Carry buffers are shared by all calls on one
// matrix: calls on the same matrix must be ordered (one stream, or events).
#pragma once

#include "common.cuh"
#include <mutex>

namespace sspmv {

// Scratch of the merge-path kernel: the pieces of rows that cross windows.
struct MergePlan {
    int64_t windows = 0;
    int32_t *carry_row = nullptr;  // row that starts in the window and goes on past it, or -1
    int32_t *has_end = nullptr;    // whether a row ends in the window
    void *carry_val = nullptr;     // kMaxK values a window: sum of the row open at its end
    void *head_val = nullptr;      // kMaxK values: sum of the first ended row, begun earlier
};

constexpr int kMaxK = 8;  // right-hand sides handled per pass

// Schedule of the stream kernel (csr_stream.cu): the nonzeros cut into windows
// of `window` elements.
struct StreamPlan {
    int window = 0;            // 0: not built
    int64_t windows = 0;
    int4 *rec = nullptr;       // [windows] first element, end element, first row, flags: 1 the first row began in an
                               // earlier window, 2 the last one goes on past the window
    int4 *split = nullptr;     // [nsplit] split rows: first window, last window, ordinal
    int64_t nsplit = 0;
    uint8_t *ends = nullptr;   // bit e: nonzero e is the last of its row
    void *tail_val = nullptr;  // [windows * kMaxK] piece of the split row that goes on past the window
    void *head_val = nullptr;  // [windows * kMaxK] last piece of the split row that ends in the window
    int32_t *nzrow = nullptr;  // y row of the i-th nonempty row (null: i itself)
    int32_t *empty = nullptr;  // rows without nonzeros
    int64_t nempty = 0;
    unsigned char *slab = nullptr;  // the allocation that holds all of these (but a caller's nzrow)
};

struct Plan {
    int kind = 0;
    StreamPlan stream;
    MergePlan merge;
    int param = 0;          // kernel parameter set by sspmv_set_kernel (0 = library choice)
    void *extra[12] = {nullptr};  // format-specific device buffers
    int64_t extra_i[12] = {0};
};

// Guards plan creation.  Recursive: building one plan may build another
// (a sliced matrix's overflow rows get their stream plan while the matrix's
// own plan is being built).
using PlanMutex = std::recursive_mutex;
PlanMutex &plan_mutex();
Plan *get_plan(const sspmv_features *f);  // creates an empty plan if needed
void free_plan(sspmv_features *f, sspmv_stream_t s);
int64_t plan_bytes(const sspmv_features *f);  // device memory of the plan as it is

// Allocates (once) the merge-path scratch of a matrix.
sspmv_status ensure_merge_plan(MergePlan &mp, int64_t m, int64_t nnz, int32_t value_type, sspmv_stream_t s);

}  // namespace sspmv
