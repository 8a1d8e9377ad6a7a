// serve.cuh -- device-side batch description shared by the request server
// (server.cu) and the batched stream CSR kernels (csr_stream.cu).
//
// A batch holds many independent requests y = alpha*A*X + beta*Y on CSR
// matrices of any size.  Requests are grouped by (value type, k); group g =
// 4 * (value_type == F64) + log2(k) for k in {1, 2, 4, 8}.  Within a group the
// windows of all requests are numbered consecutively (item i owns global
// windows [window_begin, window_begin + windows of its matrix)), and one
// persistent kernel per group walks the global windows.  Each request is cut
// into exactly the windows the single-matrix stream kernel uses (the matrix's
// own plan), so a request's result does not depend on what else is in the
// batch.
#pragma once

#include "common.cuh"
#include "csr_stream.cuh"

namespace sspmv {

constexpr int kBatchGroups = 8;

inline int batch_group(int32_t value_type, int32_t k) {
    const int lk = k == 8 ? 3 : k == 4 ? 2 : k == 2 ? 1 : 0;
    return (value_type == SSPMV_F64 ? 4 : 0) + lk;
}

struct BatchItem {
    StreamView view;
    const void *x;
    void *y;
    int64_t ldx, ldy;
    double alpha, beta;
    int64_t window_begin;  // first global window of this item in its group
    int64_t split_begin;   // first global split row likewise
    int64_t empty_begin;   // first global unit of rows without nonzeros likewise
    int32_t xvec;          // X rows aligned for vector loads (xrow_vec)
    int32_t yvec;          // Y rows likewise
};

struct BatchHeader {
    int32_t item_begin[kBatchGroups];    // first item of each group (items are stored group by group)
    int32_t n_items[kBatchGroups];
    int64_t total_windows[kBatchGroups];
    int64_t total_splits[kBatchGroups];
    int64_t total_empties[kBatchGroups];
    int64_t slot_base[kBatchGroups];     // first split-row slot of each group
};

// Split-row slots of one batch workspace (one per window): kMaxK values of up
// to 8 bytes for each of a window's two pieces.
constexpr size_t kBatchSlotBytes = 2 * kMaxK * 8;

// Slots for a batch of `requests` matrices of `chunks` 256-nonzero chunks in
// all: a window holds at least 224 nonzeros (window_size), so a matrix of c
// chunks has at most 8 c / 7 + 1 windows.
inline int64_t batch_slots(int64_t chunks, int64_t requests) { return chunks + (chunks + 6) / 7 + requests; }

// The stream kernel's view of a matrix with nonzeros (its plan built on the
// first call).
sspmv_status csr_stream_view(const sspmv_csr *A, StreamView *view, sspmv_stream_t s);

// Persistent grid size of group g (SMs x resident CTAs of its batch kernel).
unsigned csr_batch_grid(int g);

// Launches group g's batched stream kernel and its split-row kernel on stream s.
// Header and items are read from device memory when the kernels run, so the
// launches can be captured once and replayed for every batch.
sspmv_status launch_csr_batch_group(int g, const BatchHeader *d_hdr, const BatchItem *d_items, void *carry,
                                    int64_t carry_slots, sspmv_stream_t s);

}  // namespace sspmv
