// csr_stream.cu -- the nonzero-split stream kernel on sm_103a: CSR's default
// SpMV / SpMM, row-sorted COO's, the long rows of the sliced formats and the request server's
// batches.
//
// The nonzeros are cut into windows of T elements (window_size); a warp owns
// the rows that start in its window and walks their nonzeros in steps of 256,
// a group of G lanes the 8 G consecutive ones at 8 G g.  What the plan
// precomputes keeps row_offset and every search out of the kernel: a record
// per window (first and end element, first row) and one bit per nonzero, set
// where a row ends.  A lane's bits give its row ends; a prefix count of the
// set bits gives its first row.
//
// What bounds it: the x gathers, one L1-to-L2 request per gathered line and
// clock of an SM (2.9e11/s over the GPU), and in FP64 the narrow FP64 pipe,
// which is paid per warp instruction.  Every shuffle and shared-memory access
// queues behind the gathers of the other warps in the same pipe (profiled at
// over 100 cycles each), so the work after the gathers is a chain of as few of
// them as possible: row ends come from the plan's bits by ballots, the open
// sums of the lanes are joined by one segmented shuffle scan no deeper than
// the longest run of lanes without a row end, and a row's sum is stored by the
// lane that ends it.  An earlier form that marked row starts in shared memory
// (row_offset read per chunk, a five-step prefix scan, a second launch for rows
// crossing 256-element chunks) took, per SpMV: 1024^2 Laplacian FP64 33.4 us
// (now 20.7), uniform 2M x 32 FP64 315 us (271), banded 2M FP64 85 us (60),
// power-law 4M FP32 with alpha and beta 339 us (268).  Columns
// loaded a step ahead, a cp.async.bulk L2 prefetch of later windows and all
// finished rows through shared memory were slower, too (fewer warps, or more
// queued accesses).
//
// K right-hand sides: the G lanes of a group hold K / G columns each, 16 bytes
// of a row of X per lane, so that a warp instruction reads whole rows -- one
// request per row of up to 128 bytes instead of one per 16 bytes.  alpha == 1
// and beta == 0 (PLAIN) has its own instantiation; otherwise finished rows are
// collected in shared memory, up to kStage per step, and scaled (y read) 32 /
// G rows at a time: scattered multiplies would cost a full warp instruction of
// the FP64 pipe each.  SpMM on power-law rows, before and now: 1M FP64 k = 4
// 297 -> 192 us, k = 8 448 -> 331 us, 2M FP32 k = 8 318 -> 229 us; with alpha
// and beta FP64 k = 8 banded 372 -> 245 us.
//
// A warp reads up to kOver elements past its window to finish its last row.
// A row that goes on further is split: every window it meets leaves its piece
// and a second kernel (launched only when the matrix has split rows) adds each
// one's pieces in a fixed order, eight lanes a row.  (The last warp to finish,
// found by a counter per row, adding the pieces instead cost a memory fence per
// window: power-law 4M FP32 365 us against 303.)  Rows without nonzeros are a
// list, which warps behind the windows' write (scale_empty_rows).  No atomics
// on y: sums depend on the matrix alone, and a request's batch runs the same
// windows with the same code, so its result does not depend on the batch.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <vector>

#include "common.cuh"
#include "csr_stream.cuh"
#include "plan.cuh"
#include "primitives.cuh"
#include "serve.cuh"
#include "spmv_common.cuh"

namespace sspmv {
namespace {

constexpr int kBlock = 64;
constexpr int kWarps = kBlock / 32;
constexpr int kOver = 32;  // elements a warp reads past its window to finish its last row
static_assert(kStreamWholeRow == kOver + 1);
constexpr unsigned kFull = 0xffffffffu;
constexpr int kPlanBlock = 256;
constexpr int64_t kPlanTile = 1024;   // rows a block of the plan's kernels takes at least
constexpr int64_t kPlanTiles = 2048;  // blocks at most: their counts are read by the host and by every block

// Resident CTAs per SM the register budget is set for: the best of 16 to 24
// (FP32) and 12 to 18 (FP64) for K = 1; spills and fewer warps cost about the
// same beyond.
template <typename V, int K, bool BIG = false, bool PLAIN = true>
constexpr int stream_min_ctas() {
    if (K == 1) return sizeof(V) == 8 ? 15 : 20;
    return BIG ? (PLAIN ? 10 : 8) : sizeof(V) == 8 ? 12 : 14;
}

// Elements per window: whole steps of 256 less what the last row may run past
// the window, the number of steps by what the last wave of warps leaves idle
// (window_steps).
int window_size(int64_t nnz, int32_t value_type) {
    const int ctas = value_type == SSPMV_F64 ? stream_min_ctas<double, 1>() : stream_min_ctas<float, 1>();
    return 256 * window_steps(nnz, 256, 256 - kOver, ctas * kWarps) - kOver;
}

// BIG: X does not fit in L2, a gather is a random HBM access: a step's columns
// and values are all loaded before its gathers.
template <typename V, int K, bool BIG = false>
struct StreamShape {
    static constexpr int G = K * (int)sizeof(V) > 16 ? K * (int)sizeof(V) / 16 : 1;  // lanes per row of X
    static constexpr int KL = K / G;                                                 // columns per lane
    static constexpr int NG = 32 / G;
    static constexpr int kStep = 256;     // elements per step: 8 G per group
    // Rows of a step collected in shared memory for scaling (all of them for
    // K = 1); further ones are scaled where they end.
    static constexpr int kStage = K == 1 ? 256 : 64;
    // FP64: the open sum starts the next step's first lane (an add costs a warp
    // instruction of the narrow pipe).  FP32: it is added to that step's sum,
    // and each 8 elements are summed on their own first: long chains of adds to
    // a large sum would lose more bits than the rows' sums lose in chunks.
    static constexpr bool kSeed = sizeof(V) == 8;
    static constexpr int kHot = KL * sizeof(V) == 16 && !BIG ? 4 : 8;  // gathers of a lane in flight together
};

// End bits of the 8 G elements at e0 (a multiple of 8 G; the mask is padded
// to whole words).
template <int G>
__device__ __forceinline__ unsigned load_ends(const uint8_t *__restrict__ ends, uint32_t e0, uint32_t nnz) {
    if (e0 >= nnz) return 0u;
    if constexpr (G == 1) return __ldcs(ends + (e0 >> 3));
    else if constexpr (G == 2) return __ldcs(reinterpret_cast<const unsigned short *>(ends + (e0 >> 3)));
    else return __ldcs(reinterpret_cast<const unsigned *>(ends + (e0 >> 3)));
}

// KL values at p, one vector load / store when `vec` (p aligned to it).
template <typename V, int KL>
__device__ __forceinline__ void ld_cols(const V *__restrict__ p, bool vec, V (&out)[KL]) {
    if constexpr (KL * sizeof(V) == 16) {
        if (vec) {
            if constexpr (sizeof(V) == 8) {
                const double2 v = __ldg(reinterpret_cast<const double2 *>(p));
                out[0] = v.x;
                out[1] = v.y;
            } else {
                const float4 v = __ldg(reinterpret_cast<const float4 *>(p));
                out[0] = v.x; out[1] = v.y; out[2] = v.z; out[3] = v.w;
            }
            return;
        }
    } else if constexpr (KL * sizeof(V) == 8 && KL == 2) {
        if (vec) {
            const float2 v = __ldg(reinterpret_cast<const float2 *>(p));
            out[0] = v.x;
            out[1] = v.y;
            return;
        }
    }
#pragma unroll
    for (int q = 0; q < KL; q++) out[q] = ld_x(p + q);
}

// y of a finished row, the same instructions wherever it is inlined (a batch
// gives the bits of a lone call).
template <typename V>
__device__ __forceinline__ V scaled(V alpha, V sum, V beta, V y) {
    return beta == V(0) ? alpha * sum : fma(alpha, sum, beta * y);
}

// Where the pieces of split rows are left (slot = window plus the matrix's
// first slot: a batch gives every request its own).
template <typename V>
struct StreamSlots {
    V *tail_val, *head_val;
    int64_t shift;
};

// Window w of a matrix, run by one warp.  s_y: the warp's kStage * K values of
// shared memory (not PLAIN).
template <typename V, int K, bool PLAIN, bool BIG = false>
__device__ __forceinline__ void stream_window(const StreamView &A, const V *__restrict__ x, uint32_t xrow, V alpha,
                                              V beta, V *__restrict__ y, uint32_t yrow, const int64_t w,
                                              const StreamSlots<V> &sl, bool xvec, bool yvec,
                                              V *__restrict__ s_y) {
    using S = StreamShape<V, K, BIG>;
    constexpr int G = S::G, KL = S::KL, NG = S::NG, kStep = S::kStep, kStage = S::kStage, kHot = S::kHot;
    constexpr bool kSeed = S::kSeed;
    const int lane = threadIdx.x & 31, gi = lane / G, q0 = (lane % G) * KL;
    const V *val = static_cast<const V *>(A.val);
    const bool vec = A.vec != 0;
    // the first step's loads wait for nothing but the window's index; a
    // group's elements are 8 G consecutive ones, taken 8 at a time
    uint32_t e0 = (uint32_t)w * (uint32_t)A.window + 8u * G * gi;
    constexpr int NB = BIG ? G : 1;  // blocks of 8 elements loaded together
    int cb[NB][8];
    V ab[NB][8];
#pragma unroll
    for (int j = 0; j < NB; j++) load_cols8(A.col, e0 + 8 * j, A.nnz, vec, cb[j]);
    unsigned ebits = load_ends<G>(A.ends, e0, A.nnz);
    const int4 rec = __ldg(A.rec + w);
    const uint32_t eA = (uint32_t)rec.x, eB = (uint32_t)rec.y;
    const char *xq = reinterpret_cast<const char *>(x + q0);
    char *yq = reinterpret_cast<char *>(y + q0);
    int row = rec.z;                 // ordinal (among the nonempty rows) of the first row not yet finished
    bool head_split = rec.w & 1;     // the first row began in an earlier window
    auto row_of = [&](int ordinal) { return (uint32_t)(A.nzrow ? __ldg(A.nzrow + ordinal) : ordinal); };
    auto y_of = [&](int ordinal) { return reinterpret_cast<V *>(yq + (uint64_t)row_of(ordinal) * yrow); };
    V carry[KL];  // the open row's sum over the earlier steps: added to a step's sum, not the start of one
#pragma unroll
    for (int q = 0; q < KL; q++) carry[q] = V(0);
    bool later = false;

    for (;;) {
#pragma unroll
        for (int j = 0; j < NB; j++) load_vals8<V>(val, e0 + 8 * j, A.nnz, vec, ab[j]);
        // from the end bits, under the loads: rows ended before this group
        // (pos) and in the whole step (nend), and the groups back to the one
        // whose last end opened this group's running sum (dist)
        ebits &= in_window<8 * G>(e0, eA, eB);
        const int mine = __popc(ebits);
        const unsigned before = (1u << (gi * G)) - 1u;  // lanes of the groups before this one
        int pos = 0, nend = 0;
#pragma unroll
        for (int bit = 0; (1 << bit) <= 8 * G; bit++) {
            const unsigned m = __ballot_sync(kFull, (lane % G) == 0 && ((mine >> bit) & 1));
            pos += __popc(m & before) << bit;
            nend += __popc(m) << bit;
        }
        const unsigned flags = __ballot_sync(kFull, mine != 0) & (before | (1u << (gi * G)));
        const int dist = flags ? gi - (31 - __clz(flags)) / G : gi;

        // row `idx` of the step is complete
        auto finished = [&](int idx, const V(&sum)[KL]) {
            if constexpr (PLAIN) {
                st_cols<V, KL, BIG>(y_of(row + idx), yvec, sum);
            } else if (K == 1 || idx < kStage) {
                st_cols<V, KL>(s_y + idx * K + q0, true, sum);
            } else {
                V *yp = y_of(row + idx);
                V o[KL];
#pragma unroll
                for (int q = 0; q < KL; q++) o[q] = scaled(alpha, sum[q], beta, beta == V(0) ? V(0) : yp[q]);
                st_cols<V, KL, BIG>(yp, yvec, o);
            }
        };
        V y_old[PLAIN ? 1 : KL];  // y of the step's first finished rows, loaded under the gathers
        if constexpr (!PLAIN) {
#pragma unroll
            for (int q = 0; q < KL; q++) y_old[q] = V(0);
            if (beta != V(0) && gi < nend && !(head_split && gi == 0)) {
                const V *yp = y_of(row + gi);
#pragma unroll
                for (int q = 0; q < KL; q++) y_old[q] = yp[q];
            }
        }

        V sum[KL], head[KL];
#pragma unroll
        for (int q = 0; q < KL; q++) {
            sum[q] = kSeed && gi == 0 ? carry[q] : V(0);
            head[q] = V(0);
        }
        bool first = true;
        int idx = pos;  // ordinal in the step of the row that ends next
#pragma unroll
        for (int j = 0; j < G; j++) {
            const unsigned in = in_window<8>(e0 + 8 * j, eA, eB), eb = (ebits >> (8 * j)) & 0xffu;
            V run[KL];  // the open row's sum over the group's earlier elements
#pragma unroll
            for (int q = 0; q < KL; q++) run[q] = V(0);
            if (!kSeed && j > 0) {
#pragma unroll
                for (int q = 0; q < KL; q++) {
                    run[q] = sum[q];
                    sum[q] = V(0);
                }
            }
            int(&c)[8] = cb[NB > 1 ? j : 0];
            V(&a)[8] = ab[NB > 1 ? j : 0];
            if (NB == 1 && j > 0) {
                load_cols8(A.col, e0 + 8 * j, A.nnz, vec, c);
                load_vals8<V>(val, e0 + 8 * j, A.nnz, vec, a);
            }
#pragma unroll
            for (int h = 0; h < 8; h += kHot) {
                V xv[kHot][KL];
                if (in) {
#pragma unroll
                    for (int u = 0; u < kHot; u++)
                        ld_cols<V, KL>(reinterpret_cast<const V *>(xq + (uint64_t)(uint32_t)c[h + u] * xrow), xvec,
                                       xv[u]);
                }
                if (in != 0xffu) {  // other windows' elements: theirs may be Inf or NaN
#pragma unroll
                    for (int u = 0; u < kHot; u++)
                        if (!((in >> (h + u)) & 1u)) {
                            a[h + u] = V(0);
#pragma unroll
                            for (int q = 0; q < KL; q++) xv[u][q] = V(0);
                        }
                }
#pragma unroll
                for (int u = 0; u < kHot; u++) {
#pragma unroll
                    for (int q = 0; q < KL; q++) sum[q] = fma(a[h + u], xv[u][q], sum[q]);
                    if ((eb >> (h + u)) & 1u) {
                        if (!kSeed && j > 0) {
#pragma unroll
                            for (int q = 0; q < KL; q++) {
                                sum[q] += run[q];
                                run[q] = V(0);
                            }
                        }
                        if (first) {
                            first = false;
#pragma unroll
                            for (int q = 0; q < KL; q++) head[q] = sum[q];
                        } else {
                            finished(idx, sum);
                        }
                        idx++;
#pragma unroll
                        for (int q = 0; q < KL; q++) sum[q] = V(0);
                    }
                }
            }
            if (!kSeed && j > 0) {
#pragma unroll
                for (int q = 0; q < KL; q++) sum[q] += run[q];
            }
        }
        // segmented inclusive scan of the open sums over the groups
#pragma unroll
        for (int o = 1; o < NG; o <<= 1) {
            if (!__any_sync(kFull, dist >= o)) break;
#pragma unroll
            for (int q = 0; q < KL; q++) {
                const V up = __shfl_up_sync(kFull, sum[q], o * G);
                if (dist >= o) sum[q] += up;
            }
        }
        V cin[KL];
#pragma unroll
        for (int q = 0; q < KL; q++) cin[q] = __shfl_up_sync(kFull, sum[q], G);
        if (mine) {
            if (gi > 0) {
#pragma unroll
                for (int q = 0; q < KL; q++) head[q] += cin[q];
            }
            if (!kSeed && pos == 0 && later) {
#pragma unroll
                for (int q = 0; q < KL; q++) head[q] += carry[q];
            }
            if (head_split && pos == 0) {
                V *hp = sl.head_val + (w + sl.shift) * kMaxK + q0;
#pragma unroll
                for (int q = 0; q < KL; q++) hp[q] = head[q];
            } else {
                finished(pos, head);
            }
        }
        if constexpr (!PLAIN) {
            __syncwarp();
            for (int i = gi; i < nend && i < kStage; i += NG) {
                if (head_split && i == 0) continue;
                V *yp = y_of(row + i);
                V o[KL];
#pragma unroll
                for (int q = 0; q < KL; q++)
                    o[q] = scaled(alpha, s_y[i * K + q0 + q], beta,
                                  i < NG ? y_old[q] : beta == V(0) ? V(0) : yp[q]);
                st_cols<V, KL, BIG>(yp, yvec, o);
            }
            __syncwarp();
        }
        e0 += kStep;
        const bool more = e0 - 8u * G * gi < eB;  // warp-uniform
        if (more || (rec.w & 2)) {
#pragma unroll
            for (int q = 0; q < KL; q++) {
                const V last = __shfl_sync(kFull, sum[q], (NG - 1) * G + lane % G);
                carry[q] = kSeed || nend > 0 ? last : carry[q] + last;
            }
        }
        if (nend > 0) head_split = false;
        row += nend;
        if (!more) break;
        later = true;
#pragma unroll
        for (int j = 0; j < NB; j++) load_cols8(A.col, e0 + 8 * j, A.nnz, vec, cb[j]);
        ebits = load_ends<G>(A.ends, e0, A.nnz);
    }

    if (A.nshared > 0) {  // the rows without nonzeros: this window's share
        const int64_t i0 = A.nshared * w / A.windows, i1 = A.nshared * (w + 1) / A.windows;
        for (int64_t i = i0 + lane; i < i1; i += 32) {
            V *ye = reinterpret_cast<V *>(reinterpret_cast<char *>(y) + (uint64_t)(uint32_t)__ldg(A.empty + i) * yrow);
#pragma unroll
            for (int q = 0; q < K; q++) ye[q] = beta == V(0) ? V(0) : beta * ye[q];
        }
    }
    if ((rec.w & 2) && gi == 0) {  // the last row goes on past the window
        V *cp = sl.tail_val + (w + sl.shift) * kMaxK + q0;
#pragma unroll
        for (int q = 0; q < KL; q++) cp[q] = carry[q];
    }
}

// Split row sp (first window, last window, ordinal), kSplitLanes lanes: its
// pieces in a fixed order -- lane l adds windows w0 + l, w0 + l + 8, ..., then
// a shuffle tree.  All lanes of the warp call it (any: whether the lane's row
// exists).
constexpr int kSplitLanes = 8;

template <typename V, int K>
__device__ __forceinline__ void stream_split_row(bool any, const int4 sp, const int32_t *__restrict__ nzrow,
                                                 const StreamSlots<V> &sl, V alpha, V beta, V *__restrict__ y,
                                                 int64_t ldy) {
    const int lane = threadIdx.x & (kSplitLanes - 1);
    V tot[K], y_old[K];
#pragma unroll
    for (int q = 0; q < K; q++) tot[q] = y_old[q] = V(0);
    V *yp = y;
    if (any && lane == 0) {  // nothing the windows write: loaded while they still run
        yp += (int64_t)(nzrow ? __ldg(nzrow + sp.z) : sp.z) * ldy;
        if (beta != V(0)) {
#pragma unroll
            for (int q = 0; q < K; q++) y_old[q] = yp[q];
        }
    }
    wait_for_previous();
    if (any) {
        for (int u = sp.x + lane; u <= sp.y; u += kSplitLanes) {
            const V *p = (u == sp.y ? sl.head_val : sl.tail_val) + (u + sl.shift) * kMaxK;
#pragma unroll
            for (int q = 0; q < K; q++) tot[q] += p[q];
        }
    }
#pragma unroll
    for (int q = 0; q < K; q++) tot[q] = warp_sum(tot[q], kSplitLanes);
    if (any && lane == 0) {
#pragma unroll
        for (int q = 0; q < K; q++) yp[q] = scaled(alpha, tot[q], beta, y_old[q]);
    }
}

template <typename V, int K>
__global__ void __launch_bounds__(256) csr_split_kernel(int64_t n, const int4 *__restrict__ split,
                                                        const int32_t *__restrict__ nzrow, const StreamSlots<V> sl,
                                                        V alpha, V beta, V *__restrict__ y, int64_t ldy) {
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kSplitLanes;
    const bool any = i < n;
    stream_split_row<V, K>(any, any ? __ldg(split + i) : make_int4(0, -1, 0, 0), nzrow, sl, alpha, beta, y, ldy);
}

// PLAIN: alpha == 1 and beta == 0 (y = sum): row writes carry no FP64
// multiply.
template <typename V, int K, bool PLAIN, bool BIG = false>
__global__ void __launch_bounds__(kBlock, (stream_min_ctas<V, K, BIG, PLAIN>())) csr_stream_kernel(
    const StreamView A, const V *__restrict__ x, uint32_t xrow, V alpha, V beta, V *__restrict__ y, uint32_t yrow,
    const StreamSlots<V> sl, int xvec, int yvec) {
    const int64_t w = (int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5);
    __shared__ __align__(16) V s_y[kWarps][PLAIN ? 1 : StreamShape<V, K>::kStage * K];
    let_next_start();
    if (w >= A.windows) {
        if (A.nshared == 0) scale_empty_rows<V, K>(A, w - A.windows, PLAIN ? V(0) : beta, y, yrow, yvec != 0);
        return;
    }
    stream_window<V, K, PLAIN, BIG>(A, x, xrow, alpha, beta, y, yrow, w, sl, xvec != 0, yvec != 0,
                               s_y[threadIdx.x >> 5]);
}

// Whether rows of Y may be written with vector stores (as xrow_vec for X).
template <typename V>
int yrow_vec(const V *y, int64_t ldy, int k) {
    return xrow_vec(y, ldy, sizeof(V), k);
}

// ------------------------------------------------------------------ plan --
// A row that goes on more than `over` elements past its first window is split.
__device__ __forceinline__ bool row_is_split(const int32_t *__restrict__ rp, int64_t row, int T, int over) {
    return (int64_t)rp[row + 1] > ((int64_t)(rp[row] / T) + 1) * T + over;
}

// The rows in tiles (stream_tile_rows), a block each: tiles[b] counts its rows with
// nonzeros (.x) and its split rows (.y).
__global__ void __launch_bounds__(kPlanBlock) stream_count_tiles(int64_t m, int64_t rows, int T, int over,
                                                                 const int32_t *__restrict__ rp,
                                                                 int2 *__restrict__ tiles,
                                                                 unsigned long long *__restrict__ nsplit) {
    __shared__ int s_sum[2][kPlanBlock / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t i0 = (int64_t)blockIdx.x * rows, i1 = min(i0 + rows, m);
    int n = 0, k = 0;
    for (int64_t i = i0 + threadIdx.x; i < i1; i += kPlanBlock) {
        n += rp[i + 1] != rp[i];
        k += row_is_split(rp, i, T, over);
    }
    n = warp_sum(n);
    k = warp_sum(k);
    if (lane == 0) {
        s_sum[0][warp] = n;
        s_sum[1][warp] = k;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    for (int w = 1; w < kPlanBlock / 32; w++) {
        n += s_sum[0][w];
        k += s_sum[1][w];
    }
    tiles[blockIdx.x] = make_int2(n, k);
    if (blockIdx.x == 0) *nsplit = 0;
}

// End bits (ends starts at zero) and, LISTS, the two row lists: pos[i] = rows with
// nonzeros before row i, from the tiles' counts and the block's own flags.  Flags,
// a scan of three kernels, the lists and the bits in launches of their own took a
// first product on 7,267 rows with 5% empty 86 us, 67 so.
template <bool LISTS>
__global__ void __launch_bounds__(kPlanBlock) stream_fill_rows(int64_t m, int64_t rows, const int32_t *__restrict__ rp,
                                                               const int2 *__restrict__ tiles,
                                                               uint32_t *__restrict__ ends, int32_t *__restrict__ pos,
                                                               int32_t *__restrict__ nzrow,
                                                               int32_t *__restrict__ empty) {
    __shared__ int s_sum[kPlanBlock / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t i0 = (int64_t)blockIdx.x * rows, i1 = min(i0 + rows, m);
    int before = 0;  // rows with nonzeros before the chunk
    if constexpr (LISTS) {
        for (int t = threadIdx.x; t < (int)blockIdx.x; t += kPlanBlock) before += tiles[t].x;
        before = warp_sum(before);
        if (lane == 0) s_sum[warp] = before;
        __syncthreads();
        before = 0;
        for (int w = 0; w < kPlanBlock / 32; w++) before += s_sum[w];
    }
    for (int64_t b = i0; b < i1; b += kPlanBlock) {  // block-uniform
        const int64_t i = b + threadIdx.x;
        int end = 0;
        bool some = false;
        if (i < i1) {
            end = rp[i + 1];
            some = end != rp[i];
        }
        if (some) atomicOr(ends + ((uint32_t)(end - 1) >> 5), 1u << ((end - 1) & 31));
        if constexpr (LISTS) {
            const unsigned f = __ballot_sync(kFull, some);
            __syncthreads();  // s_sum of the chunk before is read
            if (lane == 0) s_sum[warp] = __popc(f);
            __syncthreads();
            int at = before + __popc(f & ((1u << lane) - 1u));
            for (int w = 0; w < kPlanBlock / 32; w++) {
                if (w < warp) at += s_sum[w];
                before += s_sum[w];
            }
            if (i < i1) {
                pos[i] = at;
                if (some) nzrow[at] = (int32_t)i;
                else empty[i - at] = (int32_t)i;
            }
        }
    }
}

// First row r with rp[r] >= e (m if none): the warp's lanes together.
__device__ __forceinline__ int first_row_from(const int32_t *__restrict__ rp, int m, int64_t e, int lane) {
    return e > 0 ? (int)warp_last_le(rp, m, (int32_t)(e - 1), lane) + 1 : 0;
}

// Window records, and the list of split rows (in any order: each is summed
// on its own); nsplit starts at zero.  A warp per window, for the searches.
__global__ void stream_windows(int64_t nw, int T, int over, int m, int64_t nnz, const int32_t *__restrict__ rp,
                               const int32_t *__restrict__ pos, int4 *__restrict__ rec, int4 *__restrict__ split,
                               unsigned long long *__restrict__ nsplit) {
    const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (w >= nw) return;  // warp-uniform
    const int64_t a = w * T, b = min(a + T, nnz);
    const int r = first_row_from(rp, m, a, lane), r2 = first_row_from(rp, m, b, lane);
    if (lane != 0) return;
    auto ordinal = [&](int row) { return pos && row < m ? pos[row] : row; };
    int64_t eA = rp[r], eB;
    int first = ordinal(r), flags = 0;
    if (eA > a && row_is_split(rp, r - 1, T, over)) {  // row r - 1 began in an earlier window
        flags |= 1;
        eA = a;
        first = ordinal(r - 1);
    }
    if (r2 > r) {  // the last row that starts here
        if (row_is_split(rp, r2 - 1, T, over)) {
            flags |= 2;
            eB = b;
            split[atomicAdd(nsplit, 1ull)] = make_int4((int)w, (int)(((int64_t)rp[r2] - 1) / T), ordinal(r2 - 1), 0);
        } else {
            eB = rp[r2];
        }
    } else if (flags & 1) {
        eB = min((int64_t)rp[r], b);
        if (rp[r] > b) flags |= 2;
    } else {
        eB = eA;  // inside a row that an earlier window finishes
    }
    rec[w] = make_int4((int)eA, (int)eB, first, flags);
}

}  // namespace

// Warps of equal work run in waves of what the SMs hold, so few windows cost as
// many steps as their last wave: 1024^2 Laplacian FP64 (4560 warps at once)
// 23.2 us in 2.4 waves of two steps, 25.6 in 1.2 of four, 21.2 in one of five;
// FP32 (6080) 14.9, 14.2 and 14.9.  kStart: a warp's start, in steps.  Many
// waves overlap, and longer windows leave fewer rows to finish (power-law 4M
// FP32: 289 us with one step, 275 with two, 272 with three to five).
int window_steps(int64_t nnz, int step, int first, int warps_per_sm) {
    constexpr double kStart = 0.35;
    const double slots = (double)num_sms() * warps_per_sm;
    int best = 1;
    double best_cost = 0;
    for (int n = 1; n <= 5; n++) {
        const double waves = (double)nnz / ((double)(n - 1) * step + first) / slots;
        const double cost = (waves <= 6 ? std::ceil(waves) : waves + 0.5) * (n + kStart);
        if (n == 1 || cost < best_cost) {
            best = n;
            best_cost = cost;
        }
    }
    return best;
}

int64_t stream_tile_rows(int64_t m) {
    return kPlanTile * std::max<int64_t>(1, (m + kPlanTile * kPlanTiles - 1) / (kPlanTile * kPlanTiles));
}

void free_stream_plan(StreamPlan &sp, sspmv_stream_t s) {
    dfree(sp.slab, s);
    sp = StreamPlan();
}

sspmv_status ensure_stream_plan(StreamPlan &sp, int64_t m, int64_t nnz, const int32_t *row_offset,
                                const int32_t *row_map, int32_t value_type, sspmv_stream_t s, int window, int over,
                                int64_t nempty, const int2 *counted) {
    if (sp.window) return SSPMV_OK;
    std::lock_guard<PlanMutex> g(plan_mutex());
    if (sp.window) return SSPMV_OK;
    const int T = window > 0 ? window : window_size(nnz, value_type);
    if (over < 0) over = kOver;
    const int64_t nw = (nnz + T - 1) / T, rows = stream_tile_rows(m), tiles = (m + rows - 1) / rows;
    const size_t sv = vsize(value_type), words = (size_t)(nnz + 31) / 32;
    StreamPlan q;
    unsigned char *count = nullptr;  // the number of split rows, then the tiles' counts
    int32_t *pos = nullptr;
    auto build = [&]() -> sspmv_status {
        SSPMV_TRY(dalloc(&count, 16 + (size_t)tiles * sizeof(int2), s));
        unsigned long long *nsplit = (unsigned long long *)count;
        int2 *tile = (int2 *)(count + 16);
        if (nempty < 0) {
            stream_count_tiles<<<(unsigned)tiles, kPlanBlock, 0, cu(s)>>>(m, rows, T, over, row_offset, tile, nsplit);
            SSPMV_LAUNCH_CHECK();
        }
        if (nempty >= 0) {
            q.nempty = nempty;
        } else {
            std::vector<int2> h((size_t)tiles);
            SSPMV_CUDA_TRY(cudaMemcpyAsync(h.data(), tile, h.size() * sizeof(int2), cudaMemcpyDeviceToHost, cu(s)));
            SSPMV_CUDA_TRY(cudaStreamSynchronize(cu(s)));
            q.nempty = m;
            for (const int2 &t : h) {
                q.nempty -= t.x;
                q.nsplit += t.y;
            }
        }
        const bool lists = q.nempty > 0;
        size_t bytes = 0;
        auto part = [&](size_t n) {
            const size_t at = bytes;
            bytes += (n + 255) / 256 * 256;
            return at;
        };
        const size_t rec = part((size_t)nw * sizeof(int4)), split = part((size_t)q.nsplit * sizeof(int4)),
                     ends = part(words * 4), piece = q.nsplit > 0 ? (size_t)nw * kMaxK * sv : 0, tail = part(piece),
                     head = part(piece), nz = part(lists ? (size_t)(m - q.nempty) * 4 : 0),
                     em = part((size_t)q.nempty * 4);
        SSPMV_TRY(dalloc(&q.slab, bytes, s));
        q.rec = (int4 *)(q.slab + rec);
        q.split = (int4 *)(q.slab + split);
        q.ends = q.slab + ends;
        q.tail_val = q.slab + tail;
        q.head_val = q.slab + head;
        q.nzrow = lists ? (int32_t *)(q.slab + nz) : const_cast<int32_t *>(row_map);
        q.empty = (int32_t *)(q.slab + em);
        if (lists) SSPMV_TRY(dalloc(&pos, (size_t)m, s));
        SSPMV_CUDA_TRY(cudaMemsetAsync(q.ends, 0, words * 4, cu(s)));
        auto fill = [&](auto kernel) {
            kernel<<<(unsigned)tiles, kPlanBlock, 0, cu(s)>>>(m, rows, row_offset, counted ? counted : tile,
                                                              (uint32_t *)q.ends, pos, q.nzrow, q.empty);
        };
        if (lists) fill(stream_fill_rows<true>);
        else fill(stream_fill_rows<false>);
        SSPMV_LAUNCH_CHECK();
        stream_windows<<<grid_for(nw, 8), 256, 0, cu(s)>>>(nw, T, over, (int)m, nnz, row_offset, pos, q.rec, q.split,
                                                             nsplit);
        SSPMV_LAUNCH_CHECK();
        return SSPMV_OK;
    };
    const sspmv_status st = build();
    dfree(pos, s);
    dfree(count, s);
    if (st != SSPMV_OK) {
        free_stream_plan(q, s);
        return st;
    }
    q.windows = nw;
    sp = q;
    std::atomic_thread_fence(std::memory_order_release);
    sp.window = T;  // published last
    return SSPMV_OK;
}

StreamView stream_view(const StreamPlan &sp, int64_t nnz, const int32_t *col, const void *val) {
    StreamView v;
    v.col = col;
    v.val = val;
    v.rec = sp.rec;
    v.split = sp.split;
    v.ends = sp.ends;
    v.nzrow = sp.nzrow;
    v.empty = sp.empty;
    v.windows = sp.windows;
    v.nnz = (uint32_t)nnz;
    v.window = sp.window;
    v.nempty = (int32_t)sp.nempty;
    v.nshared = sp.nempty <= sp.windows / 8 ? (int32_t)sp.nempty : 0;
    v.nsplit = (int32_t)sp.nsplit;
    v.vec = ((reinterpret_cast<uintptr_t>(col) | reinterpret_cast<uintptr_t>(val)) & 15) == 0;
    return v;
}

// An X of more bytes than this does not stay in L2 (129 MB, less what the matrix
// and Y take): its gathers wait for HBM, and the form that loads all of a step's
// columns and values before its first gathers, with twice the gathers in flight,
// fewer warps and Y written past L2 is the faster one.  For rows of X of 32 bytes
// (of 64 the registers do not hold it).  FP32, k = 8: 83 MB power-law 314 us, 297
// so, uniform 278 and 241, banded 144 and 152; 64 MB power-law 214 and 222; 512 MB
// 5.02 ms and 4.72.  With alpha and beta 83 MB 396 and 415, 96 MB 488 and 490,
// 134 MB 804 and 783.  FP64, k = 4: 96 MB 541 and 531, 64 MB 337 and 351.
constexpr int64_t kBigX = int64_t(80) << 20;
constexpr int64_t kBigXScaled = int64_t(100) << 20;

template <typename V, int K>
sspmv_status launch_stream_windows(const StreamView &v, StreamPlan &sp, V alpha, const V *x, int64_t ldx, V beta,
                                   V *y, int64_t ldy, int64_t cols, sspmv_stream_t s) {
    const StreamSlots<V> sl{(V *)sp.tail_val, (V *)sp.head_val, 0};
    const uint32_t xrow = (uint32_t)(ldx * (int64_t)sizeof(V)), yrow = (uint32_t)(ldy * (int64_t)sizeof(V));
    auto go = [&](auto kernel) {
        kernel<<<grid_for(v.windows + (v.nshared > 0 ? 0 : empty_units(v.nempty)), kWarps), kBlock, 0, cu(s)>>>(
            v, x, xrow, alpha, beta, y, yrow, sl, xrow_vec(x, ldx, sizeof(V), K), yrow_vec(y, ldy, K));
    };
    const bool plain = alpha == V(1) && beta == V(0);
    bool big = false;
    if constexpr (K * sizeof(V) == 32) {
        big = cols * ldx * (int64_t)sizeof(V) > (plain ? kBigX : kBigXScaled);
        if (big && plain) go(csr_stream_kernel<V, K, true, true>);
        else if (big) go(csr_stream_kernel<V, K, false, true>);
    }
    if (!big && plain) go(csr_stream_kernel<V, K, true>);
    else if (!big) go(csr_stream_kernel<V, K, false>);
    SSPMV_LAUNCH_CHECK();
    return SSPMV_OK;
}

template <typename V, int K>
sspmv_status launch_split_rows(const StreamView &v, StreamPlan &sp, V alpha, V beta, V *y, int64_t ldy,
                               sspmv_stream_t s) {
    if (v.nsplit == 0) return SSPMV_OK;
    const StreamSlots<V> sl{(V *)sp.tail_val, (V *)sp.head_val, 0};
    SSPMV_CUDA_TRY(launch_behind(csr_split_kernel<V, K>, grid_for(v.nsplit * kSplitLanes, 256), 256, cu(s), v.nsplit,
                                 v.split, v.nzrow, sl, alpha, beta, y, ldy));
    SSPMV_LAUNCH_CHECK();
    return SSPMV_OK;
}

#define SSPMV_STREAM_INST(V, K)                                                                                \
    template sspmv_status launch_stream_windows<V, K>(const StreamView &, StreamPlan &, V, const V *, int64_t, \
                                                      V, V *, int64_t, int64_t, sspmv_stream_t);               \
    template sspmv_status launch_split_rows<V, K>(const StreamView &, StreamPlan &, V, V, V *, int64_t,        \
                                                  sspmv_stream_t);
SSPMV_STREAM_INST(float, 1)
SSPMV_STREAM_INST(float, 2)
SSPMV_STREAM_INST(float, 4)
SSPMV_STREAM_INST(float, 8)
SSPMV_STREAM_INST(double, 1)
SSPMV_STREAM_INST(double, 2)
SSPMV_STREAM_INST(double, 4)
SSPMV_STREAM_INST(double, 8)
#undef SSPMV_STREAM_INST

// ---------------------------------------------------- batched (serving) --
namespace {

// Index of the item owning global window (or split row) i: the last item
// whose first one, items[mid].*begin, is <= i (increasing within a group).
__device__ __forceinline__ int batch_item_of(const BatchItem *__restrict__ items, int n, int64_t i,
                                             int64_t BatchItem::*begin) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(&(items[mid].*begin)) <= i) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Persistent stream kernel over the windows of every request of group g and
// then the units of their lists of rows without nonzeros:
// warp i of the grid takes global windows i, i + warps, ...  A request is cut
// into the windows a lone sspmv_spmm_csr call uses (the matrix's own plan),
// and the pieces of its split rows go to per-batch slots, so its result does
// not depend on the rest of the batch and equals the single-request call's.
template <typename V, int K>
__global__ void __launch_bounds__(kBlock, (stream_min_ctas<V, K>() * 3 / 4)) csr_batch_kernel(int g, const BatchHeader *__restrict__ hdr,
                                                           const BatchItem *__restrict__ all_items,
                                                           V *__restrict__ tail_val, V *__restrict__ head_val) {
    const int n = hdr->n_items[g];
    const int64_t total = hdr->total_windows[g];
    const int64_t base = hdr->slot_base[g];
    const BatchItem *items = all_items + hdr->item_begin[g];
    const int64_t warps = (int64_t)gridDim.x * kWarps;
    __shared__ __align__(16) V s_y[kWarps][StreamShape<V, K>::kStage * K];
    for (int64_t gw = (int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5); gw < total; gw += warps) {
        const BatchItem *q = items + batch_item_of(items, n, gw, &BatchItem::window_begin);
        const StreamSlots<V> sl{tail_val, head_val, base + q->window_begin};
        stream_window<V, K, false>(q->view, (const V *)q->x, (uint32_t)(q->ldx * (int64_t)sizeof(V)), (V)q->alpha,
                                   (V)q->beta, (V *)q->y, (uint32_t)(q->ldy * (int64_t)sizeof(V)),
                                   gw - q->window_begin, sl, q->xvec != 0, q->yvec != 0, s_y[threadIdx.x >> 5]);
    }
    const int64_t units = hdr->total_empties[g];
    for (int64_t gu = (int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5); gu < units; gu += warps) {
        const BatchItem *q = items + batch_item_of(items, n, gu, &BatchItem::empty_begin);
        scale_empty_rows<V, K>(q->view, gu - q->empty_begin, (V)q->beta, (V *)q->y,
                               (uint64_t)q->ldy * sizeof(V), q->yvec != 0);
    }
}

// The split rows of every request of group g, kSplitLanes lanes each.
template <typename V, int K>
__global__ void __launch_bounds__(256) csr_batch_split_kernel(int g, const BatchHeader *__restrict__ hdr,
                                                              const BatchItem *__restrict__ all_items,
                                                              V *__restrict__ tail_val, V *__restrict__ head_val) {
    const int n = hdr->n_items[g];
    const int64_t total = hdr->total_splits[g];
    const int64_t base = hdr->slot_base[g];
    const BatchItem *items = all_items + hdr->item_begin[g];
    const int64_t stride = ((int64_t)gridDim.x * blockDim.x) / kSplitLanes;
    const int64_t i0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kSplitLanes;
    const int64_t w0 = i0 - (threadIdx.x & 31) / kSplitLanes;  // the warp's first row: trip count the same for its lanes
    for (int64_t d = 0; w0 + d < total; d += stride) {
        const int64_t i = i0 + d;
        const bool any = i < total;
        const BatchItem *q = items + (any ? batch_item_of(items, n, i, &BatchItem::split_begin) : 0);
        const StreamSlots<V> sl{tail_val, head_val, base + q->window_begin};
        stream_split_row<V, K>(any, any ? __ldg(q->view.split + (i - q->split_begin)) : make_int4(0, -1, 0, 0),
                               q->view.nzrow, sl, (V)q->alpha, (V)q->beta, (V *)q->y, q->ldy);
    }
}

// Resident CTAs per SM of csr_batch_kernel<V, K>.
template <typename V, int K>
int batch_blocks_per_sm() {
    static int blocks = 0;
    if (blocks == 0) {
        int b = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, csr_batch_kernel<V, K>, kBlock, 0) != cudaSuccess ||
            b < 1)
            b = 1;
        blocks = b;
    }
    return blocks;
}

template <typename V, int K>
sspmv_status launch_batch_vk(int g, const BatchHeader *hdr, const BatchItem *items, void *carry, int64_t slots,
                             sspmv_stream_t s) {
    unsigned char *c = (unsigned char *)carry;
    V *tail_val = (V *)c;
    V *head_val = (V *)(c + (size_t)slots * kMaxK * 8);
    const unsigned grid = (unsigned)(num_sms() * batch_blocks_per_sm<V, K>());
    csr_batch_kernel<V, K><<<grid, kBlock, 0, cu(s)>>>(g, hdr, items, tail_val, head_val);
    SSPMV_LAUNCH_CHECK();
    csr_batch_split_kernel<V, K><<<(unsigned)num_sms(), 256, 0, cu(s)>>>(g, hdr, items, tail_val, head_val);
    SSPMV_LAUNCH_CHECK();
    return SSPMV_OK;
}

}  // namespace

unsigned csr_batch_grid(int g) {
    int b = 1;
    switch (g) {
    case 0: b = batch_blocks_per_sm<float, 1>(); break;
    case 1: b = batch_blocks_per_sm<float, 2>(); break;
    case 2: b = batch_blocks_per_sm<float, 4>(); break;
    case 3: b = batch_blocks_per_sm<float, 8>(); break;
    case 4: b = batch_blocks_per_sm<double, 1>(); break;
    case 5: b = batch_blocks_per_sm<double, 2>(); break;
    case 6: b = batch_blocks_per_sm<double, 4>(); break;
    default: b = batch_blocks_per_sm<double, 8>(); break;
    }
    return (unsigned)(num_sms() * b);
}

sspmv_status launch_csr_batch_group(int g, const BatchHeader *d_hdr, const BatchItem *d_items, void *carry,
                                    int64_t carry_slots, sspmv_stream_t s) {
    switch (g) {
    case 0: return launch_batch_vk<float, 1>(g, d_hdr, d_items, carry, carry_slots, s);
    case 1: return launch_batch_vk<float, 2>(g, d_hdr, d_items, carry, carry_slots, s);
    case 2: return launch_batch_vk<float, 4>(g, d_hdr, d_items, carry, carry_slots, s);
    case 3: return launch_batch_vk<float, 8>(g, d_hdr, d_items, carry, carry_slots, s);
    case 4: return launch_batch_vk<double, 1>(g, d_hdr, d_items, carry, carry_slots, s);
    case 5: return launch_batch_vk<double, 2>(g, d_hdr, d_items, carry, carry_slots, s);
    case 6: return launch_batch_vk<double, 4>(g, d_hdr, d_items, carry, carry_slots, s);
    case 7: return launch_batch_vk<double, 8>(g, d_hdr, d_items, carry, carry_slots, s);
    }
    return fail(SSPMV_INVALID_ARG, "batch group %d out of range", g);
}

}  // namespace sspmv
