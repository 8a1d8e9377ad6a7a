// spmv_csr.cu -- CSR SpMV / SpMM on sm_103a.
//
// Replaces LeSpMV_csr (src/spmv_csr.cpp:165-185) and its three CPU kernels
// (serial, OpenMP per row, nnz-balanced row partition).
//
// Default kernel (kernel_flag 0): the nonzero-split stream kernel
// (csr_stream.cu); a matrix without nonzeros runs merge-path.  kernel_flag 4:
// the pipelined thread-per-row kernel for
// matrices whose rows all have at most 12 nonzeros (csr_pipe_kernel).
// kernel_flag 3: the row-block kernel for matrices whose rows are all short
// (csr_rowblock_kernel; one launch, no fix-up).  kernel_flag 2: merge-path
// (csr_merge_kernel), which needs no plan: also the allocation-free entry
// point's kernel.
//
// kernel_flag 1: vector-per-row kernel, `lanes` threads per row (2..32,
// chosen from the mean row length, or set by the autotuner).
#include <atomic>
#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "plan.cuh"
#include "bulk.cuh"
#include "primitives.cuh"
#include "spmv_common.cuh"
#include "csr_pipe.cuh"
#include "csr_stream.cuh"
#include "serve.cuh"

namespace sspmv {
namespace {

constexpr int kBlock = 256;

// --------------------------------------------------------- merge path --
// The (row end, nonzero) merge sequence cut into windows of kMergeItems items,
// one per warp, whatever the row lengths; no plan: a warp finds its own start
// (a 33-way search of row_offset, four dependent loads for 500k rows, hidden
// by the other warps' gathers), turns the row ends of its window into end bits
// and a row list in shared memory, and then runs steps of 256 nonzeros as the
// stream kernel does -- 8 consecutive nonzeros a lane with all loads in flight,
// one segmented scan of the open sums a step.  A row that crosses windows
// leaves its pieces and is finished by a second kernel in a fixed order.  The
// order of a row's additions depends on row_offset alone, not on K.
// 8M nonzeros of power-law rows, 5% of them empty, K = 1: FP32 43.6 us + 7.4
// for the second kernel (tiles of 2048 items staged in shared memory by 256
// threads, split points from a kernel of their own: 12.6 + 48.7 + 8.8), the
// whole call in FP64 100 -> 70 us; K = 8 on 200k rows, FP64, 331 -> 134 with
// the scratch allocated for the call.  The gathers alone take 28 us: the rest
// is shared-memory and shuffle work queued behind them and the row ends' round
// trip.  Four steps a window measured the same.
constexpr int kMergeBlock = 64;
constexpr int kMergeWarps = kMergeBlock / 32;
constexpr int kMergeSteps = 2;
constexpr int kMergeItems = 256 * kMergeSteps - 8;  // its nonzeros, from an 8-aligned one on, fit the steps

inline int64_t merge_windows(int64_t m, int64_t nnz) {
    return std::max<int64_t>((m + nnz + kMergeItems - 1) / kMergeItems, 1);
}

// Resident CTAs per SM the register budget is set for: K = 1, 2M rows, FP32, 20
// (which spills) / 18 / 16 CTAs 178 / 157 / 160 us.
template <typename V, int K>
constexpr int merge_ctas() {
    return K == 1 ? (sizeof(V) == 8 ? 14 : 18) : K <= 4 ? 10 : 7;
}

// Rows whose end is among the first d items of the merge sequence (the warp's
// lanes together): the smallest p with row_offset[p + 1] + p >= d.
__device__ __forceinline__ int merge_split(const int32_t *__restrict__ row_offset, int64_t m, int64_t nnz, int64_t d,
                                           int lane) {
    int64_t lo = d > nnz ? d - nnz : 0, hi = d < m ? d : m;
    while (lo < hi) {  // warp-uniform
        const int64_t step = (hi - lo + 31) >> 5, p = lo + (lane + 1) * step - 1;
        const unsigned ended =
            __ballot_sync(0xffffffffu, p < hi && (int64_t)ld_x(row_offset + (p < hi ? p + 1 : 0)) + p < d);
        const int64_t next = lo + __popc(ended) * step;
        hi = min(hi, next + step - 1);
        lo = min(next, hi);
    }
    return (int)lo;
}

template <typename V, int K, bool PLAIN>
__global__ void __launch_bounds__(kMergeBlock, (merge_ctas<V, K>())) csr_merge_kernel(
    int64_t windows, int m, int nnz, const int32_t *__restrict__ row_offset, const int32_t *__restrict__ col_index,
    const V *__restrict__ values, int vec, const V *__restrict__ x, int64_t ldx, int xvec, V alpha, V beta,
    V *__restrict__ y, int64_t ldy, int32_t *__restrict__ carry_row, int32_t *__restrict__ has_end,
    V *__restrict__ carry_val, V *__restrict__ head_val) {
    constexpr unsigned kFull = 0xffffffffu;
    constexpr bool kSeed = sizeof(V) == 8;  // as the stream kernel: FP32 adds the carry apart
    constexpr int kHot = K == 1 ? 8 : K == 2 ? 4 : 2;  // gathers of a lane in flight together
    __shared__ uint32_t s_ends[kMergeWarps][8 * kMergeSteps];
    __shared__ unsigned short s_row[kMergeWarps][kMergeItems];
    const int wi = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t w = (int64_t)blockIdx.x * kMergeWarps + wi;
    let_next_start();
    if (w >= windows) return;  // warp-uniform
    uint32_t *ends = s_ends[wi];
    unsigned short *rows = s_row[wi];
    if (lane < 8 * kMergeSteps) ends[lane] = 0;
    const int64_t d0 = w * kMergeItems, d1 = min(d0 + kMergeItems, (int64_t)m + nnz);
    const int i0 = merge_split(row_offset, m, nnz, d0, lane);
    const int j0 = (int)(d0 - i0), b = j0 & ~7;
    __syncwarp();

    // rows that end in the window: end bits and row of the nonempty ones
    int nr = 0, nne = 0, open_start;
    bool head_split = false;  // the first nonempty one began in an earlier window
    for (int base = 0, prev = row_offset[i0];; base += 32) {
        const int64_t p = (int64_t)i0 + base + lane;
        const int re = p < m ? ld_x(row_offset + p + 1) : 0;
        const bool ended = p < m && re + p < d1;
        int rs = __shfl_up_sync(kFull, re, 1);
        if (lane == 0) rs = prev;
        const bool some = ended && re > max(rs, j0);
        const unsigned eb = __ballot_sync(kFull, ended), sb = __ballot_sync(kFull, some);
        if (some) {
            const int pos = re - 1 - b;
            atomicOr(&ends[pos >> 5], 1u << (pos & 31));
            rows[nne + __popc(sb & ((1u << lane) - 1u))] = (unsigned short)(base + lane);
        } else if (ended) {
            if (rs < j0) {  // all of the first row lies in earlier windows
#pragma unroll
                for (int q = 0; q < K; q++) head_val[w * K + q] = V(0);
            } else {  // an empty row
                V *yp = y + p * ldy;
#pragma unroll
                for (int q = 0; q < K; q++) yp[q] = beta == V(0) ? V(0) : beta * yp[q];
            }
        }
        if (base == 0) head_split = __ballot_sync(kFull, some && rs < j0) & 1u;
        nr += __popc(eb);
        nne += __popc(sb);
        if (eb != kFull) {
            open_start = __shfl_sync(kFull, rs, __popc(eb));
            break;
        }
        prev = __shfl_sync(kFull, re, 31);
    }
    const int j1 = (int)(d1 - i0 - nr);
    if (lane == 0) {
        carry_row[w] = i0 + nr < m && open_start >= j0 && open_start < j1 ? i0 + nr : -1;
        has_end[w] = nr > 0;
    }
    __syncwarp();

    V carry[K];  // the open row's sum over the earlier steps
#pragma unroll
    for (int q = 0; q < K; q++) carry[q] = V(0);
    int row = 0;  // ordinal among the window's nonempty rows of the first not yet finished
    auto finished = [&](int idx, const V(&sum)[K]) {
        V *yp = y + ((int64_t)i0 + rows[idx]) * ldy;
#pragma unroll
        for (int q = 0; q < K; q++) yp[q] = row_out(PLAIN, alpha, sum[q], beta, yp + q);
    };
    // unsigned: the last step's e + 256 may pass INT_MAX (nnz up to 2^31 - 1)
    for (uint32_t e = j0 < j1 ? b : j1; e < (uint32_t)j1; e += 256) {  // warp-uniform
        const uint32_t e0 = e + 8u * lane;
        const unsigned in = in_window<8>(e0, j0, j1);
        int c[8];
        V a[8];
        if (in) {
            load_cols8(col_index, e0, nnz, vec != 0, c);
            load_vals8<V>(values, e0, nnz, vec != 0, a);
        }
        const unsigned ebits = (ends[(e0 - b) >> 5] >> ((e0 - b) & 31)) & 0xffu;
        const int mine = __popc(ebits);
        const unsigned before = (1u << lane) - 1u;
        int pos = 0, nend = 0;  // rows ended in the lanes before this one, and in the step
#pragma unroll
        for (int bit = 0; bit < 4; bit++) {
            const unsigned f = __ballot_sync(kFull, (mine >> bit) & 1);
            pos += __popc(f & before) << bit;
            nend += __popc(f) << bit;
        }
        const unsigned flags = __ballot_sync(kFull, mine != 0) & (before | (1u << lane));
        const int dist = flags ? lane - (31 - __clz(flags)) : lane;
        V sum[K], head[K];
#pragma unroll
        for (int q = 0; q < K; q++) {
            sum[q] = kSeed && lane == 0 ? carry[q] : V(0);
            head[q] = V(0);
        }
        bool first = true;
        int idx = row + pos;
#pragma unroll
        for (int h = 0; h < 8; h += kHot) {
            V xv[kHot][K];
            if (in) {
#pragma unroll
                for (int u = 0; u < kHot; u++) ld_xrow<V, K>(x, c[h + u], ldx, xvec != 0, xv[u]);
            }
            if (in != 0xffu) {  // other windows' elements: theirs may be Inf or NaN
#pragma unroll
                for (int u = 0; u < kHot; u++)
                    if (!((in >> (h + u)) & 1u)) {
                        a[h + u] = V(0);
#pragma unroll
                        for (int q = 0; q < K; q++) xv[u][q] = V(0);
                    }
            }
#pragma unroll
            for (int u = 0; u < kHot; u++) {
#pragma unroll
                for (int q = 0; q < K; q++) sum[q] = fma(a[h + u], xv[u][q], sum[q]);
                if ((ebits >> (h + u)) & 1u) {
                    if (first) {
                        first = false;
#pragma unroll
                        for (int q = 0; q < K; q++) head[q] = sum[q];
                    } else {
                        finished(idx, sum);
                    }
                    idx++;
#pragma unroll
                    for (int q = 0; q < K; q++) sum[q] = V(0);
                }
            }
        }
        // segmented inclusive scan of the lanes' open sums
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            if (!__any_sync(kFull, dist >= o)) break;
#pragma unroll
            for (int q = 0; q < K; q++) {
                const V up = __shfl_up_sync(kFull, sum[q], o);
                if (dist >= o) sum[q] += up;
            }
        }
#pragma unroll
        for (int q = 0; q < K; q++) {
            const V cin = __shfl_up_sync(kFull, sum[q], 1), last = __shfl_sync(kFull, sum[q], 31);
            if (lane > 0) head[q] += cin;
            if (!kSeed && pos == 0) head[q] += carry[q];
            carry[q] = kSeed || nend > 0 ? last : carry[q] + last;
        }
        if (mine) {
            if (head_split && pos == 0) {
#pragma unroll
                for (int q = 0; q < K; q++) head_val[w * K + q] = head[q];
            } else {
                finished(row + pos, head);
            }
        }
        if (nend > 0) head_split = false;
        row += nend;
    }
    if (lane == 0) {
#pragma unroll
        for (int q = 0; q < K; q++) carry_val[w * K + q] = carry[q];
    }
}

// Finishes the rows that cross windows: the window where such a row starts
// (carry_row >= 0) adds the following windows' pieces in order.
template <typename V, int K>
__global__ void csr_merge_fixup(int64_t windows, const int32_t *__restrict__ carry_row,
                                const int32_t *__restrict__ has_end, const V *__restrict__ carry_val,
                                const V *__restrict__ head_val, V alpha, V beta, V *__restrict__ y, int64_t ldy) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    wait_for_previous();
    if (t - (threadIdx.x & 31) >= windows) return;  // whole warp past the end
    const int r = t < windows ? carry_row[t] : -1;
    V tot[K];
    chain_sum<V, K, K>(r >= 0, t, windows, 0, has_end, carry_val, head_val, tot);
    if (r >= 0) {
        V *yp = y + (int64_t)r * ldy;
#pragma unroll
        for (int q = 0; q < K; q++) yp[q] = axpby(alpha, tot[q], beta, yp + q);
    }
}

// y = alpha A x + beta y with the pieces of rows that cross windows in q
// (arrays of q.windows entries, the values K apart).
template <typename V, int K>
sspmv_status run_merge(const sspmv_csr *A, const MergePlan &q, V alpha, const V *x, int64_t ldx, V beta, V *y,
                       int64_t ldy, sspmv_stream_t s) {
    const int vec = ((reinterpret_cast<uintptr_t>(A->col_index) | reinterpret_cast<uintptr_t>(A->values)) & 15) == 0;
    auto go = [&](auto kernel) {
        kernel<<<grid_for(q.windows, kMergeWarps), kMergeBlock, 0, cu(s)>>>(
            q.windows, (int)A->f.num_rows, (int)A->f.num_nnzs, A->row_offset, A->col_index, (const V *)A->values, vec,
            x, ldx, xrow_vec(x, ldx, sizeof(V), K), alpha, beta, y, ldy, q.carry_row, q.has_end, (V *)q.carry_val,
            (V *)q.head_val);
    };
    if (alpha == V(1) && beta == V(0)) go(csr_merge_kernel<V, K, true>);  // y = sum
    else go(csr_merge_kernel<V, K, false>);
    SSPMV_LAUNCH_CHECK();
    if (q.windows > 1) {
        SSPMV_CUDA_TRY(launch_behind(csr_merge_fixup<V, K>, grid_for(q.windows, 256), 256, cu(s), q.windows, q.carry_row,
                                     q.has_end, (const V *)q.carry_val, (const V *)q.head_val, alpha, beta, y, ldy));
        SSPMV_LAUNCH_CHECK();
    }
    return SSPMV_OK;
}

constexpr int kVecHoist = 6;

// The vector kernel's element index runs up to 127 past a row's last element in an
// int: matrices with more nonzeros run the default kernel.  (An unsigned or 64-bit
// index costs 10 to 25% with two or more lanes per row.)
constexpr int64_t kVecMaxNnz = INT32_MAX - 128;

template <typename V, int K, int VS, bool PLAIN = false>
__global__ void __launch_bounds__(kBlock, (VS == 1 && K == 1) ? (sizeof(V) == 4 ? 6 : 5) : 1) csr_vector_kernel(
    int m, const int32_t *__restrict__ row_offset, const int32_t *__restrict__ col_index,
    const V *__restrict__ values, const V *__restrict__ x, int64_t ldx, int xvec, V alpha, V beta,
    V *__restrict__ y, int64_t ldy) {
    constexpr int kRowsPerWarp = 32 / VS;
    const int lane = threadIdx.x & 31;
    const int sub = lane % VS;
    const int64_t warp_id = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t base = warp_id * kRowsPerWarp; base < m; base += nwarps * kRowsPerWarp) {
        const int64_t row = base + lane / VS;
        V s[K];
#pragma unroll
        for (int r = 0; r < K; r++) s[r] = V(0);
        int rs = 0, re = 0;
        if (row < m) {
            rs = ld_stream(row_offset + row);
            re = ld_stream(row_offset + row + 1);
        }
        // One lane per row, short rows (every lane of the warp with at most
        // kVecHoist elements): all of a lane's column and value loads, then
        // all its x gathers, are issued before its first FMA -- one memory
        // round trip each instead of one per element (same summation order
        // as the loop).  Measured: FP32 5-point Laplacian 22 -> 17 us; with
        // 2+ lanes per row the loop below was faster.
        const int cnt = re - rs > sub ? (re - rs - sub + VS - 1) / VS : 0;
        const int wmax = (VS == 1 && K <= 2) ? __reduce_max_sync(0xffffffffu, cnt) : kVecHoist + 1;
        if (wmax <= kVecHoist) {
            int c[kVecHoist];
            V a[kVecHoist];
#pragma unroll
            for (int q = 0; q < kVecHoist; q++) {
                c[q] = 0;  // a lane past its elements gathers x row 0 (exists: some lane has elements) with value 0
                a[q] = V(0);
                if (q < cnt) {
                    c[q] = ld_stream(col_index + rs + sub + q * VS);
                    a[q] = ld_stream(values + rs + sub + q * VS);
                }
            }
            V xr[kVecHoist][K];
#pragma unroll
            for (int q = 0; q < kVecHoist; q++)
                if (q < wmax) ld_xrow<V, K>(x, c[q], ldx, xvec != 0, xr[q]);
#pragma unroll
            for (int q = 0; q < kVecHoist; q++)
                if (q < cnt) {  // never 0 * x[0]: x may hold Inf or NaN
#pragma unroll
                    for (int r = 0; r < K; r++) s[r] += a[q] * xr[q][r];
                }
        } else if (row < m) {
            int j = rs + sub;
            for (; j + 3 * VS < re; j += 4 * VS) {  // four independent gathers in flight
                int c[4];
                V a[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    c[u] = ld_stream(col_index + j + u * VS);
                    a[u] = ld_stream(values + j + u * VS);
                }
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    V xr[K];
                    ld_xrow<V, K>(x, c[u], ldx, xvec != 0, xr);
#pragma unroll
                    for (int r = 0; r < K; r++) s[r] += a[u] * xr[r];
                }
            }
            for (; j < re; j += VS) {
                const int c = ld_stream(col_index + j);
                const V a = ld_stream(values + j);
                V xr[K];
                ld_xrow<V, K>(x, c, ldx, xvec != 0, xr);
#pragma unroll
                for (int r = 0; r < K; r++) s[r] += a * xr[r];
            }
        }
#pragma unroll
        for (int r = 0; r < K; r++) s[r] = warp_sum(s[r], VS);
        if (row < m && sub == 0) {
            V *yp = y + row * ldy;
#pragma unroll
            for (int r = 0; r < K; r++) yp[r] = row_out(PLAIN, alpha, s[r], beta, yp + r);
        }
    }
}

template <typename V, int K>
sspmv_status launch_merge(const sspmv_csr *A, Plan *p, V alpha, const V *x, int64_t ldx, V beta, V *y,
                          int64_t ldy, sspmv_stream_t s) {
    SSPMV_TRY(ensure_merge_plan(p->merge, A->f.num_rows, A->f.num_nnzs, A->f.value_type, s));
    return run_merge<V, K>(A, p->merge, alpha, x, ldx, beta, y, ldy, s);
}

template <typename V, int K, int VS>
sspmv_status launch_vector_vs(const sspmv_csr *A, V alpha, const V *x, int64_t ldx, V beta, V *y, int64_t ldy,
                              sspmv_stream_t s) {
    const int64_t m = A->f.num_rows;
    const int64_t warps = (m + (32 / VS) - 1) / (32 / VS);
    const unsigned grid = grid_for(warps * 32, kBlock, (int64_t)num_sms() * 16);
    auto go = [&](auto kernel) {
        kernel<<<grid, kBlock, 0, cu(s)>>>((int)m, A->row_offset, A->col_index, (const V *)A->values, x, ldx,
                                           xrow_vec(x, ldx, sizeof(V), K), alpha, beta, y, ldy);
    };
    if (K == 1 && alpha == V(1) && beta == V(0)) go(csr_vector_kernel<V, K, VS, K == 1>);
    else go(csr_vector_kernel<V, K, VS>);
    SSPMV_LAUNCH_CHECK();
    return SSPMV_OK;
}

template <typename V, int K>
sspmv_status launch_vector(const sspmv_csr *A, Plan *p, V alpha, const V *x, int64_t ldx, V beta, V *y,
                           int64_t ldy, sspmv_stream_t s) {
    int vs = p->param;
    if (vs == 0) {
        double mean = A->f.num_rows > 0 ? (double)A->f.num_nnzs / (double)A->f.num_rows : 1.0;
        vs = 2;
        while (vs < 32 && vs < mean) vs <<= 1;
    }
    switch (vs) {
    case 1: return launch_vector_vs<V, K, 1>(A, alpha, x, ldx, beta, y, ldy, s);
    case 2: return launch_vector_vs<V, K, 2>(A, alpha, x, ldx, beta, y, ldy, s);
    case 4: return launch_vector_vs<V, K, 4>(A, alpha, x, ldx, beta, y, ldy, s);
    case 8: return launch_vector_vs<V, K, 8>(A, alpha, x, ldx, beta, y, ldy, s);
    case 16: return launch_vector_vs<V, K, 16>(A, alpha, x, ldx, beta, y, ldy, s);
    default: return launch_vector_vs<V, K, 32>(A, alpha, x, ldx, beta, y, ldy, s);
    }
}

// ----------------------------------------------------- row-block kernel --
// kernel_flag 3: short rows, one launch, streamed by the copy engine.
//
// The rows are cut into blocks of whole rows: row r opens a block when its
// first nonzero lies in another window of `window` nonzeros than row r - 1's,
// or r is a multiple of kRbRows.  A block therefore holds at most kRbRows
// rows and, with no row longer than kRbMaxRow, at most window + kRbMaxRow - 1
// nonzeros, and no row crosses two blocks: the CTA that takes a block
// finishes its rows itself, with no carries and no fix-up launch (a second
// launch costs about as much as the whole SpMV of an 84 MB matrix).
//
// The grid is persistent (every SM full), CTA g taking blocks g, g + G, ...
// Thread 0 streams each block's row offsets, columns and values into one of
// kRbStages shared-memory stages with three bulk copies (cp.async.bulk, the
// copy engine) completed on the stage's mbarrier, kRbStages blocks ahead of
// the CTA's threads: the matrix moves like a copy, with no per-element load
// instructions and no load latency on the threads' path.  The threads then
// gather x for the block's nonzeros (all gathers of a thread in flight
// together), overwrite each value with its product, and each thread sums its
// rows' products in row order.  The bulk copies cover the 16-byte aligned
// interior of each run; the few elements at its ragged ends are read with
// plain loads.  Deterministic.  Matrices with a row longer than kRbMaxRow use
// the stream kernel instead, and so do arrays not 16-byte aligned.
constexpr int kRbRows = 1024;
constexpr int kRbMaxRow = 64;
constexpr int kRbDefaultWindow = 1024;
constexpr int kRbStages = 2;

// Count of bounded waits that gave up (a copy that never completed) in this
// file's kernels since the library was loaded; read by sspmv_wait_timeouts.
__device__ unsigned long long g_csr_wait_timeouts = 0;

__global__ void rowblock_flags(int m, int lg_window, const int32_t *__restrict__ rp, int32_t *__restrict__ flag) {
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= m) return;
    flag[r] = (r % kRbRows == 0 || (rp[r] >> lg_window) != (rp[r - 1] >> lg_window)) ? 1 : 0;
}

__global__ void rowblock_starts(int m, int nnz, int lg_window, int nb, const int32_t *__restrict__ rp,
                                const int32_t *__restrict__ pos, int2 *__restrict__ blocks) {
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r == 0) blocks[nb] = make_int2(m, nnz);
    if (r >= m) return;
    const bool opens = r % kRbRows == 0 || (rp[r] >> lg_window) != (rp[r - 1] >> lg_window);
    if (opens) blocks[pos[r]] = make_int2((int)r, rp[r]);
}

// Shared-memory layout of one stage (element capacities; every region starts
// on a 16-byte boundary).  A block's run [e0, e1) of an array is copied as
// the 16-byte aligned superset [e0 rounded down, e1 rounded up) -- its
// neighbours' elements ride along -- and element e sits at index
// e - (e0 rounded down), so a region holds the longest run plus 2 x 16 bytes.
template <typename V, int W>
struct RbStage {
    static constexpr int kNz = W + kRbMaxRow + 8;        // columns and values
    static constexpr int kRp = kRbRows + 1 + 7;          // row offsets
    static constexpr size_t kValBytes = (size_t)kNz * sizeof(V);
    static constexpr size_t kColBytes = (size_t)kNz * 4;
    static constexpr size_t kRpBytes = (size_t)kRp * 4;
    static constexpr size_t kBytes = kValBytes + kColBytes + kRpBytes + 32;  // + header
};

template <typename V, int W>
constexpr size_t rowblock_smem() {
    return kRbStages * RbStage<V, W>::kBytes + kRbStages * sizeof(uint64_t);
}

// [a, end) = [lo rounded down, hi rounded up) to 16 bytes, cut at the array's
// last 16-byte boundary (elements beyond it, at most 15 bytes, are read with
// plain loads: a copy never reads past the array).
template <int E>
__device__ __forceinline__ void copy_span(int64_t lo, int64_t hi, int64_t n, int64_t &a, int64_t &end) {
    constexpr int64_t per = 16 / E;
    a = lo / per * per;
    end = min((hi + per - 1) / per * per, n / per * per);
}

template <typename V, int W, bool PLAIN>
__global__ void __launch_bounds__(kBlock) csr_rowblock_kernel(int64_t nb, int m, int64_t nnz,
                                                              const int2 *__restrict__ blocks,
                                                              const int32_t *__restrict__ rp,
                                                              const int32_t *__restrict__ col,
                                                              const V *__restrict__ val, const V *__restrict__ x,
                                                              int64_t ldx, V alpha, V beta, V *__restrict__ y,
                                                              int64_t ldy) {
    using St = RbStage<V, W>;
    constexpr int kPer = (W + kRbMaxRow + kBlock - 1) / kBlock;
    extern __shared__ __align__(16) unsigned char rb_smem[];
    uint64_t *bars = reinterpret_cast<uint64_t *>(rb_smem + kRbStages * St::kBytes);
    auto sval = [&](int s) { return reinterpret_cast<V *>(rb_smem + s * St::kBytes); };
    auto scol = [&](int s) { return reinterpret_cast<int32_t *>(rb_smem + s * St::kBytes + St::kValBytes); };
    auto srp = [&](int s) {
        return reinterpret_cast<int32_t *>(rb_smem + s * St::kBytes + St::kValBytes + St::kColBytes);
    };
    auto shdr = [&](int s) {
        return reinterpret_cast<int32_t *>(rb_smem + s * St::kBytes + St::kValBytes + St::kColBytes + St::kRpBytes);
    };
    const int t = threadIdx.x;
    const int64_t G = gridDim.x;
    const int64_t g = blockIdx.x;

    // Thread 0: start the copies of the CTA's k-th block (bounds lo, hi) into
    // stage k % kRbStages.
    auto issue = [&](int64_t k, int2 lo, int2 hi) {
        const int64_t b = g + k * G;
        if (b >= nb) return;
        const int s = (int)(k % kRbStages);
        int64_t av, ve, ac, ce, ap, pe;
        copy_span<sizeof(V)>(lo.y, hi.y, nnz, av, ve);
        copy_span<4>(lo.y, hi.y, nnz, ac, ce);
        copy_span<4>(lo.x, (int64_t)hi.x + 1, (int64_t)m + 1, ap, pe);
        int32_t *h = shdr(s);
        h[0] = lo.x;
        h[1] = hi.x - lo.x;
        h[2] = lo.y;
        h[3] = hi.y - lo.y;
        h[4] = (hi.y > ve || hi.y > ce || (int64_t)hi.x + 1 > pe) ? 1 : 0;  // part of a run past the copies
        uint32_t tx = 0;
        tx += ve > av ? (uint32_t)((ve - av) * sizeof(V)) : 0u;
        tx += ce > ac ? (uint32_t)((ce - ac) * 4) : 0u;
        tx += pe > ap ? (uint32_t)((pe - ap) * 4) : 0u;
        fence_proxy_async_smem();
        mbar_arrive_expect_tx(&bars[s], tx);
        if (ve > av) bulk_g2s(sval(s), val + av, (uint32_t)((ve - av) * sizeof(V)), &bars[s]);
        if (ce > ac) bulk_g2s(scol(s), col + ac, (uint32_t)((ce - ac) * 4), &bars[s]);
        if (pe > ap) bulk_g2s(srp(s), rp + ap, (uint32_t)((pe - ap) * 4), &bars[s]);
    };

    if (t == 0) {
        for (int s = 0; s < kRbStages; s++) mbar_init(&bars[s], 1);
        fence_mbar_init();
    }
    __syncthreads();
    if (t == 0)
        for (int k = 0; k < kRbStages; k++)
            if (g + k * G < nb) issue(k, blocks[g + k * G], blocks[g + k * G + 1]);

    for (int64_t k = 0;; k++) {
        const int64_t b = g + k * G;
        if (b >= nb) break;
        const int s = (int)(k % kRbStages);
        const uint32_t parity = (uint32_t)((k / kRbStages) & 1);
        // bounds of the block this iteration's stage takes next, loaded now so
        // their latency is spent under this block's work
        const int64_t bn = b + kRbStages * G;
        int2 nlo = make_int2(0, 0), nhi = make_int2(0, 0);
        if (t == 0 && bn < nb) {
            nlo = blocks[bn];
            nhi = blocks[bn + 1];
        }
        // One thread polls; the others sleep at the barrier, then take the
        // completed phase themselves (one poll, for its acquire).
        const bool ok = __syncthreads_and(t == 0 ? mbar_wait(&bars[s], parity) : true);
        if (!ok) {
            // A copy did not complete: record it, wait (bounded) for the
            // CTA's other copies in flight, and leave.
            if (t == 0) {
                atomicAdd(&g_csr_wait_timeouts, 1ull);
                for (int64_t k2 = k + 1; k2 < k + kRbStages && g + k2 * G < nb; k2++)
                    mbar_wait(&bars[k2 % kRbStages], (uint32_t)((k2 / kRbStages) & 1));
            }
            return;
        }
        if (t != 0) mbar_try_wait(&bars[s], parity);
        const int32_t *h = shdr(s);
        const int r0 = h[0], nr = h[1], e0 = h[2], ne = h[3];
        const bool ragged = h[4] != 0;  // the array's last block: read its tail from global memory
        constexpr int kPerV = 16 / (int)sizeof(V);
        const int av = e0 / kPerV * kPerV, ac = e0 / 4 * 4, ap = r0 / 4 * 4;
        V *vs = sval(s);
        const int32_t *cs = scol(s), *ps = srp(s);
        const int64_t vend = nnz / kPerV * kPerV, cend = nnz / 4 * 4, pend = ((int64_t)m + 1) / 4 * 4;
        if (ne > 0) {
            const int last = ne - 1;
            int c[kPer];
            V a[kPer];
#pragma unroll
            for (int j = 0; j < kPer; j++) {
                // past the block's end: the last column again (a valid gather
                // kept in flight with the others) and a zero value; each
                // thread reads only values it overwrites itself
                const int i = t + j * kBlock;
                const int e = e0 + min(i, last);
                if (!ragged) {
                    c[j] = cs[e - ac];
                    a[j] = i > last ? V(0) : vs[e - av];
                } else {
                    c[j] = e < cend ? cs[e - ac] : ld_stream(col + e);
                    a[j] = i > last ? V(0) : e < vend ? vs[e - av] : ld_stream(val + e);
                }
            }
            V xv[kPer];
#pragma unroll
            for (int j = 0; j < kPer; j++) xv[j] = ld_x(x + (int64_t)c[j] * ldx);
#pragma unroll
            for (int j = 0; j < kPer; j++) {
                const int i = t + j * kBlock;
                if (i < ne) vs[e0 + i - av] = a[j] * xv[j];
            }
        }
        __syncthreads();
        // Row sums: L lanes per row, L from the block's mean row length, so
        // that a warp's lanes read neighbouring products (one lane per row of
        // 32 nonzeros would put all 32 lanes of a warp on one bank).
        auto rows = [&](auto lanes) {
            constexpr int L = decltype(lanes)::value;
            const int lane = t & 31, sub = lane % L;
            for (int base = (t >> 5) * (32 / L); base < nr; base += kBlock / L) {
                const int i = base + lane / L;
                V sum = V(0);
                int r = r0 + i;
                if (i < nr) {
                    int rs, re;
                    if (!ragged) {
                        rs = ps[r - ap];
                        re = ps[r + 1 - ap];
                    } else {
                        rs = r < pend ? ps[r - ap] : ld_stream(rp + r);
                        re = r + 1 < pend ? ps[r + 1 - ap] : ld_stream(rp + r + 1);
                    }
                    for (uint32_t e = rs + sub; e < (uint32_t)re; e += L) sum += vs[e - av];
                }
                if constexpr (L > 1) sum = warp_sum(sum, L);
                if (i < nr && sub == 0) {
                    V *yp = y + (int64_t)r * ldy;
                    *yp = row_out(PLAIN, alpha, sum, beta, yp);
                }
            }
        };
        const int mean = nr > 0 ? ne / nr : 0;
        if (mean < 6) rows(std::integral_constant<int, 1>());
        else if (mean < 12) rows(std::integral_constant<int, 2>());
        else if (mean < 24) rows(std::integral_constant<int, 4>());
        else rows(std::integral_constant<int, 8>());
        __syncthreads();  // stage s free
        if (t == 0) issue(k + kRbStages, nlo, nhi);
    }
}

// Plan slots of the row-block kernel: extra[4] blocks (int2, nb + 1),
// extra_i[4] = nb (-1: a row longer than kRbMaxRow, kernel not usable),
// extra_i[5] = longest row, extra_i[6] = window of the blocks built.
sspmv_status ensure_rowblock_plan(const sspmv_csr *A, Plan *p, int window, sspmv_stream_t s) {
    if (p->extra_i[4] != 0 && (p->extra_i[4] < 0 || p->extra_i[6] == window)) return SSPMV_OK;
    std::lock_guard<PlanMutex> g(plan_mutex());
    if (p->extra_i[4] != 0 && (p->extra_i[4] < 0 || p->extra_i[6] == window)) return SSPMV_OK;
    const int64_t m = A->f.num_rows, nnz = A->f.num_nnzs;
    int32_t longest = 0;
    SSPMV_TRY(max_row_length(A->row_offset, m, &longest, s));
    p->extra_i[5] = longest;
    if (longest > kRbMaxRow) {
        p->extra_i[4] = -1;
        return SSPMV_OK;
    }
    int lg = 0;
    while ((1 << lg) < window) lg++;
    int32_t *pos = nullptr;
    SSPMV_TRY(dalloc(&pos, (size_t)m, s));
    rowblock_flags<<<grid_for(m, 256), 256, 0, cu(s)>>>((int)m, lg, A->row_offset, pos);
    SSPMV_LAUNCH_CHECK();
    int32_t nb = 0;
    sspmv_status st = exclusive_scan_i32(pos, pos, m, &nb, s);
    if (st != SSPMV_OK) {
        dfree(pos, s);
        return st;
    }
    int2 *blocks = nullptr;
    st = dalloc(&blocks, (size_t)nb + 1, s);
    if (st != SSPMV_OK) {
        dfree(pos, s);
        return st;
    }
    rowblock_starts<<<grid_for(m, 256), 256, 0, cu(s)>>>((int)m, (int)nnz, lg, nb, A->row_offset, pos, blocks);
    SSPMV_LAUNCH_CHECK();
    dfree(pos, s);
    if (p->extra[4]) dfree(p->extra[4], s);
    p->extra[4] = blocks;
    p->extra_i[6] = window;
    p->extra_i[4] = nb;
    return SSPMV_OK;
}

template <typename V, int W, bool PLAIN>
sspmv_status go_rowblock_k(const sspmv_csr *A, const int2 *blocks, int64_t nb, V alpha, const V *x, int64_t ldx,
                           V beta, V *y, int64_t ldy, sspmv_stream_t s) {
    constexpr size_t smem = rowblock_smem<V, W>();
    // resident CTAs per SM, set once per instantiation after its shared
    // memory attribute (a thread that reads it non-zero may launch)
    static std::atomic<int> per_sm{0};
    if (per_sm.load(std::memory_order_acquire) == 0) {
        SSPMV_CUDA_TRY(cudaFuncSetAttribute(csr_rowblock_kernel<V, W, PLAIN>,
                                            cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        int n = 0;
        SSPMV_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, csr_rowblock_kernel<V, W, PLAIN>, kBlock,
                                                                     smem));
        per_sm.store(n > 0 ? n : 1, std::memory_order_release);
    }
    const int64_t grid = std::min<int64_t>(nb, (int64_t)num_sms() * per_sm.load(std::memory_order_acquire));
    csr_rowblock_kernel<V, W, PLAIN><<<(unsigned)grid, kBlock, smem, cu(s)>>>(
        nb, (int)A->f.num_rows, A->f.num_nnzs, blocks, A->row_offset, A->col_index, (const V *)A->values, x, ldx,
        alpha, beta, y, ldy);
    SSPMV_LAUNCH_CHECK();
    return SSPMV_OK;
}

template <typename V, int W>
sspmv_status go_rowblock(const sspmv_csr *A, const int2 *blocks, int64_t nb, V alpha, const V *x, int64_t ldx,
                         V beta, V *y, int64_t ldy, sspmv_stream_t s) {
    if (alpha == V(1) && beta == V(0))
        return go_rowblock_k<V, W, true>(A, blocks, nb, alpha, x, ldx, beta, y, ldy, s);
    return go_rowblock_k<V, W, false>(A, blocks, nb, alpha, x, ldx, beta, y, ldy, s);
}

// Sets *launched = false (nothing launched) when the matrix has a row longer
// than kRbMaxRow or arrays that are not 16-byte aligned; the caller then runs
// another kernel.
template <typename V>
sspmv_status launch_rowblock(const sspmv_csr *A, Plan *p, V alpha, const V *x, int64_t ldx, V beta, V *y,
                             int64_t ldy, sspmv_stream_t s, bool *launched) {
    *launched = false;
    const uintptr_t bases = reinterpret_cast<uintptr_t>(A->row_offset) | reinterpret_cast<uintptr_t>(A->col_index) |
                            reinterpret_cast<uintptr_t>(A->values);
    if ((bases & 15) != 0) return SSPMV_OK;
    int window = p->param > 0 ? p->param : kRbDefaultWindow;
    if (window != 512 && window != 1024 && window != 2048 && window != 4096) window = kRbDefaultWindow;
    SSPMV_TRY(ensure_rowblock_plan(A, p, window, s));
    if (p->extra_i[4] < 0) return SSPMV_OK;
    const int2 *blocks = (const int2 *)p->extra[4];
    const int64_t nb = p->extra_i[4];
    switch (window) {
    case 512: SSPMV_TRY((go_rowblock<V, 512>(A, blocks, nb, alpha, x, ldx, beta, y, ldy, s))); break;
    case 2048: SSPMV_TRY((go_rowblock<V, 2048>(A, blocks, nb, alpha, x, ldx, beta, y, ldy, s))); break;
    case 4096: SSPMV_TRY((go_rowblock<V, 4096>(A, blocks, nb, alpha, x, ldx, beta, y, ldy, s))); break;
    default: SSPMV_TRY((go_rowblock<V, 1024>(A, blocks, nb, alpha, x, ldx, beta, y, ldy, s))); break;
    }
    *launched = true;
    return SSPMV_OK;
}

template <typename V, int K>
sspmv_status launch_stream(const sspmv_csr *A, Plan *p, V alpha, const V *x, int64_t ldx, V beta, V *y,
                           int64_t ldy, sspmv_stream_t s) {
    if (A->f.num_nnzs == 0 || !stream_takes_strides(ldx, ldy, sizeof(V)))
        return launch_merge<V, K>(A, p, alpha, x, ldx, beta, y, ldy, s);
    StreamView v;
    SSPMV_TRY(csr_stream_view(A, &v, s));
    return launch_stream_view<V, K>(v, p->stream, alpha, x, ldx, beta, y, ldy, A->f.num_cols, s);
}

// kernel_flag 0 (default): stream kernel (merge-path for a matrix without
// nonzeros; the request server's batched CSR work sums in the same order, so
// a request's result does not depend on whether it was batched); 1: vector;
// 2: merge-path; 3: row-block; 4: pipelined thread per row (3 and 4 fall
// back to the default on matrices they do not take).
template <typename V, int K>
sspmv_status csr_pass(const sspmv_csr *A, Plan *p, V alpha, const V *x, int64_t ldx, V beta, V *y,
                      int64_t ldy, sspmv_stream_t s) {
    if (A->f.kernel_flag == 1 && A->f.num_nnzs <= kVecMaxNnz)
        return launch_vector<V, K>(A, p, alpha, x, ldx, beta, y, ldy, s);
    if (A->f.kernel_flag == 2) return launch_merge<V, K>(A, p, alpha, x, ldx, beta, y, ldy, s);
    if constexpr (K == 1) {
        if (A->f.kernel_flag == 3) {
            bool launched = false;
            SSPMV_TRY(launch_rowblock<V>(A, p, alpha, x, ldx, beta, y, ldy, s, &launched));
            if (launched) return SSPMV_OK;
        }
        if (A->f.kernel_flag == 4) {
            bool launched = false;
            SSPMV_TRY(launch_csr_pipe<V>(A, p, alpha, x, ldx, beta, y, ldy, s, &launched));
            if (launched) return SSPMV_OK;
        }
    }
    return launch_stream<V, K>(A, p, alpha, x, ldx, beta, y, ldy, s);
}

}  // namespace

sspmv_status check_spmm_args(const sspmv_features *f, int32_t k, const void *X, int64_t ldx, const void *Y,
                             int64_t ldy) {
    if (k < 1) return fail(SSPMV_INVALID_ARG, "k must be >= 1 (got %d)", k);
    if (ldx < k || ldy < k) return fail(SSPMV_INVALID_ARG, "ldx/ldy must be >= k");
    if ((f->num_cols > 0 && !X) || (f->num_rows > 0 && !Y)) return fail(SSPMV_INVALID_ARG, "null x or y");
    if (!valid_vt(f->value_type)) return fail(SSPMV_INVALID_ARG, "bad value_type");
    return SSPMV_OK;
}

sspmv_status spmm_csr_impl(double alpha, const sspmv_csr *A, int32_t k, const void *X, int64_t ldx, double beta,
                           void *Y, int64_t ldy, sspmv_stream_t s) {
    if (!A) return fail(SSPMV_INVALID_ARG, "null matrix");
    SSPMV_TRY(check_spmm_args(&A->f, k, X, ldx, Y, ldy));
    if (A->f.num_rows == 0) return SSPMV_OK;
    Plan *p = get_plan(&A->f);
    if (!p) return fail(SSPMV_OUT_OF_MEMORY, "plan allocation failed");
    return dispatch_value(A->f.value_type, [&](auto tag) -> sspmv_status {
        using V = decltype(tag);
        return for_rhs_chunks<V>(k, (const V *)X, (V *)Y, [&](int32_t step, const V *xs, V *ys) {
            const V a = (V)alpha, b = (V)beta;
            switch (step) {
            case 8: return csr_pass<V, 8>(A, p, a, xs, ldx, b, ys, ldy, s);
            case 4: return csr_pass<V, 4>(A, p, a, xs, ldx, b, ys, ldy, s);
            case 2: return csr_pass<V, 2>(A, p, a, xs, ldx, b, ys, ldy, s);
            default: return csr_pass<V, 1>(A, p, a, xs, ldx, b, ys, ldy, s);
            }
        });
    });
}

sspmv_status ensure_merge_plan(MergePlan &mp, int64_t m, int64_t nnz, int32_t value_type, sspmv_stream_t s) {
    if (mp.windows) return SSPMV_OK;
    std::lock_guard<PlanMutex> g(plan_mutex());
    if (mp.windows) return SSPMV_OK;
    MergePlan q;
    const int64_t nw = merge_windows(m, nnz);
    const size_t bytes = (size_t)nw * kMaxK * vsize(value_type);
    sspmv_status st = dalloc(&q.carry_row, (size_t)nw, s);
    if (st == SSPMV_OK) st = dalloc(&q.has_end, (size_t)nw, s);
    if (st == SSPMV_OK) st = dalloc((unsigned char **)&q.carry_val, bytes, s);
    if (st == SSPMV_OK) st = dalloc((unsigned char **)&q.head_val, bytes, s);
    if (st != SSPMV_OK) {
        dfree(q.carry_row, s);
        dfree(q.has_end, s);
        dfree(q.carry_val, s);
        return st;
    }
    mp = q;
    std::atomic_thread_fence(std::memory_order_release);
    mp.windows = nw;  // published last
    return SSPMV_OK;
}

sspmv_status csr_stream_view(const sspmv_csr *A, StreamView *view, sspmv_stream_t s) {
    Plan *p = get_plan(&A->f);
    if (!p) return fail(SSPMV_OUT_OF_MEMORY, "plan allocation failed");
    SSPMV_TRY(ensure_stream_plan(p->stream, A->f.num_rows, A->f.num_nnzs, A->row_offset, nullptr, A->f.value_type, s));
    *view = stream_view(p->stream, A->f.num_nnzs, A->col_index, A->values);
    return SSPMV_OK;
}

}  // namespace sspmv

using namespace sspmv;

extern "C" sspmv_status sspmv_LeSpMV_csr(double alpha, const sspmv_csr *A, const void *x, double beta, void *y,
                                         sspmv_stream_t stream) {
    return spmm_csr_impl(alpha, A, 1, x, 1, beta, y, 1, stream);
}

extern "C" sspmv_status sspmv_spmm_csr(double alpha, const sspmv_csr *A, int32_t k, const void *X, int64_t ldx,
                                       double beta, void *Y, int64_t ldy, sspmv_stream_t stream) {
    return spmm_csr_impl(alpha, A, k, X, ldx, beta, Y, ldy, stream);
}

extern "C" double sspmv_algorithmic_bytes_csr(const sspmv_csr *A, int32_t k, int32_t beta_nonzero) {
    const double sv = (double)vsize(A->f.value_type);
    return (double)A->f.num_nnzs * (sv + 4.0) + (double)(A->f.num_rows + 1) * 4.0 +
           (double)k * (double)A->f.num_cols * sv + (double)k * (double)A->f.num_rows * sv * (beta_nonzero ? 2.0 : 1.0);
}

// ===================================================== allocation-free CSR ===
//
// sspmv_LeSpMV_csr_noalloc: the merge-path CSR SpMV (one right-hand side)
// with its scratch -- the pieces of rows that cross windows -- in a fixed
// device array that every GPU loading this library holds until the process
// exits, so the call itself allocates nothing.
//
// Who needs it: code that cannot call cudaMalloc at SpMV time.  An iterative
// solver or serving loop whose device heap is carved up by its own pool
// allocator up front (a cudaMalloc there either fails or steals memory the
// pool has promised elsewhere); a latency-bound loop where the implicit device
// synchronisation of cudaMalloc/cudaFree is not acceptable; a component
// running under a strict device-memory budget enforced outside this library.
// The regular entry point builds a per-matrix plan on first use and keeps it
// in device memory it allocates; this one does not.
//
// Limits and rules:
//  - scratch is kNoAllocScratchBytes (16 MiB), of which a window of
//    kMergeItems merge items takes kNoAllocWindowBytes; num_rows + num_nnzs
//    may be at most kNoAllocMaxItems (about 238 million), which is within it;
//    larger matrices get SSPMV_INVALID_ARG.
//  - the first call on a device looks up the array's device address
//    (cudaGetSymbolAddress) with that device current; make that first call
//    before any stream capture.  The address is kept per device and per
//    context: after a cudaDeviceReset the next call looks it up again.
//  - every call writes all the scratch it later reads,
//    so nothing has to be cleared between calls; but all calls share the one
//    array: calls that overlap on the GPU (different streams, or a graph
//    replayed concurrently) race on it and must be serialised by the caller.
namespace {

constexpr size_t kNoAllocScratchBytes = 16u << 20;
constexpr size_t kNoAllocWindowBytes = 4 + 4 + 2 * 8;  // carry_row, has_end, carry and head values
constexpr int64_t kNoAllocMaxItems = 238594048;
static_assert((kNoAllocMaxItems / kMergeItems + 1) * kNoAllocWindowBytes + 4 * 256 <= kNoAllocScratchBytes);

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mutex;
void *g_noalloc_ptr[kNoAllocMaxDevices] = {nullptr};
unsigned long long g_noalloc_ctx[kNoAllocMaxDevices] = {0};

// The scratch array's device address on the current device, looked up with
// cudaGetSymbolAddress the first time this device (context) is seen.
sspmv_status noalloc_scratch(void **out) {
    int dev = 0;
    SSPMV_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kNoAllocMaxDevices) return fail(SSPMV_NOT_SUPPORTED, "device ordinal %d too large", dev);
    SSPMV_CUDA_TRY(cudaSetDevice(dev));  // makes the device's primary context current (allocates nothing)
    const unsigned long long ctx = current_context_id();
    std::lock_guard<std::mutex> g(g_noalloc_mutex);
    if (!g_noalloc_ptr[dev] || g_noalloc_ctx[dev] != ctx || ctx == 0) {
        void *p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p)
            return fail(SSPMV_CUDA_ERROR, "cudaGetSymbolAddress(scratch) on device %d: %s", dev, cudaGetErrorString(e));
        g_noalloc_ptr[dev] = p;
        g_noalloc_ctx[dev] = ctx;
    }
    *out = g_noalloc_ptr[dev];
    return SSPMV_OK;
}

inline size_t align256(size_t v) { return (v + 255) & ~(size_t)255; }

}  // namespace

extern "C" sspmv_status sspmv_LeSpMV_csr_noalloc(double alpha, const sspmv_csr *A, const void *x, double beta,
                                                 void *y, sspmv_stream_t s) {
    if (!A) return fail(SSPMV_INVALID_ARG, "null matrix");
    SSPMV_TRY(check_spmm_args(&A->f, 1, x, 1, y, 1));
    const int64_t m = A->f.num_rows, nnz = A->f.num_nnzs;
    if (m == 0) return SSPMV_OK;
    if (m + nnz > kNoAllocMaxItems)
        return fail(SSPMV_INVALID_ARG,
                    "sspmv_LeSpMV_csr_noalloc: num_rows + num_nnzs = %lld exceeds the fixed scratch limit of %lld; "
                    "use sspmv_LeSpMV_csr",
                    (long long)(m + nnz), (long long)kNoAllocMaxItems);
    void *base = nullptr;
    SSPMV_TRY(noalloc_scratch(&base));
    MergePlan q;
    q.windows = merge_windows(m, nnz);
    unsigned char *b = (unsigned char *)base;
    q.carry_row = (int32_t *)b;
    b += align256((size_t)q.windows * 4);
    q.has_end = (int32_t *)b;
    b += align256((size_t)q.windows * 4);
    q.carry_val = b;
    b += align256((size_t)q.windows * 8);
    q.head_val = b;
    return dispatch_value(A->f.value_type, [&](auto tag) -> sspmv_status {
        using V = decltype(tag);
        return run_merge<V, 1>(A, q, (V)alpha, (const V *)x, 1, (V)beta, (V *)y, 1, s);
    });
}

namespace sspmv {
sspmv_status dia_wait_timeouts(unsigned long long *out);
}

extern "C" sspmv_status sspmv_wait_timeouts(int64_t *count) {
    if (!count) return fail(SSPMV_INVALID_ARG, "null output");
    unsigned long long v = 0, w = 0;
    SSPMV_CUDA_TRY(cudaMemcpyFromSymbol(&v, g_csr_wait_timeouts, sizeof(v)));
    SSPMV_TRY(sspmv::dia_wait_timeouts(&w));
    *count = (int64_t)(v + w);
    return SSPMV_OK;
}
