// sliced.cu -- ELL, S-ELL, SELL-c-sigma and SELL-c-R on sm_103a: GPU
// converters from CSR, SpMV / SpMM kernels, export to the reference layout.
//
// All four share one device layout: a slab of chunks, chunk c holding C rows
// in slot-major order (slot k of the chunk's row r at chunk_ptr[c] + k*C + r,
// padding col -1 / value 0 after each row's last nonzero).  ELL is the case
// of one chunk of C = num_rows rows (the reference's column-major ELL).
// A thread owns one (stored) row: the C threads of a chunk read C consecutive
// slots per step, and a warp covers 32/C chunks.  A row stops at its first
// padding slot, so padding costs at most one partially used sector per row
// instead of being streamed.  SELL variants write y through `reorder`.
//
// Converters (bit-exact logical content vs the reference):
//   ELL          include/sparse_conversion.h:187-248
//   S-ELL        include/sparse_conversion.h:258-334
//   SELL-c-sigma include/sparse_conversion.h:337-479 (sort: nnz desc, row desc)
//   SELL-c-R     include/sparse_conversion.h:483-598
// The per-slice sort is a stable LSD radix sort of keys
// slice*(maxlen+1) + (maxlen - len) over rows fed in descending row order.
#include <algorithm>
#include <cstring>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "csr_stream.cuh"
#include "plan.cuh"
#include "primitives.cuh"
#include "spmv_common.cuh"

namespace sspmv {
sspmv_status check_dims(int32_t vt, int64_t m, int64_t n, int64_t nnz);
void init_features(sspmv_features *f, int32_t vt, int64_t m, int64_t n, int64_t nnz, int32_t owns);
}  // namespace sspmv

using namespace sspmv;

namespace {

constexpr int kBlock = 256;

// ------------------------------------------------------------------ SpMV --
// A thread per stored row reads its slots (C consecutive rows read together)
// up to its first padding slot, so a warp runs as long as its longest row.
// Where a few long rows would keep most lanes of their warps idle, rows longer
// than a cap (chosen once per matrix by choose_cap) are left out: they are
// copied once into compact arrays, whole, and multiplied by the stream kernel
// (csr_stream.cu), every lane busy whatever the row lengths, which writes
// their y through the plan's row list.  The compact copy also skips the
// padding of the short rows that share a long row's chunk (slot-major storage
// puts them in the same sectors).  Moving only the part of a row past the cap
// (the thread's partial sum, a CSR pass over short tails, a warp per 2048
// elements of long ones and a pass that adds the three) took five launches one
// after another: SELL-c-sigma (4096, 32) on power-law 1M FP64 136 us of GPU time,
// now 84 in three launches that overlap.

// S: slots of a row whose loads are in flight together (column and value
// loads of S slots, then their x gathers, then the FMAs in slot order).
// FLAT (ELL of up to 12 slots in FP32, but 7 and 8): a row's slots loaded unconditionally
// (a slot past the width reads the last one again, padding gathers x[0]) with
// registers for all of them: two memory latencies per row instead of two per
// four slots -- banded 1M FP32 24.9 -> 17.9 us, 5-point Laplacian 1M 15.6 -> 11.9.
// With a test around each load the compiler holds a thread to 32 registers
// and orders a load after another's use; in FP64, whose pipe is the bound,
// that form at full occupancy is the faster one (banded 2M 56 us against 63
// FLAT).
// Four slots in FP64 with registers for 6 CTAs (S-ELL, 2.9M banded rows, 115 us
// at 8, 94 so), except (WAVE) for a grid that 8 take in one wave and 6 do not
// (254,620 banded rows, 14.3 us at 6, 10.9 so), for one wave of long rows (200k
// rows of 64, 58 and 48) and for chunks of one or two slots (1M rows of 2, 12.4
// and 11.0).
template <typename V, int K, int S, bool FLAT, bool WAVE>
constexpr int sliced_min_ctas() {
    if (K > 1) return K * sizeof(V) <= 16 ? 6 : 4;
    if (!FLAT) return sizeof(V) == 8 && S == 4 && !WAVE ? 6 : 8;
    return S > 10 ? 4 : S > 8 ? 5 : S > 6 ? 6 : 7;
}

// TWO: S slots at a time while there are S, without a test around each load,
// then one by one: S-ELL in FP32, 5-point Laplacian 4M 79 us with tested loads,
// 66 so, and 61 without a grid that strides over the rows; FP64, 1M rows of 30,
// 147 and 114.  Otherwise the loads of a step are tested and those past the width
// left out: for the widths that would be read mostly one by one.
template <typename V, int K, int S, bool PLAIN, bool FLAT, bool TWO>
__device__ __forceinline__ void sliced_row(
    int64_t i, int C, const int64_t *__restrict__ chunk_ptr, const int32_t *__restrict__ reorder,
    const int32_t *__restrict__ col, const V *__restrict__ val, const V *__restrict__ x, int64_t ldx, int xvec,
    V alpha, V beta, V *__restrict__ y, int64_t ldy, int64_t cap) {
    const int64_t c = div_nonneg(i, C);
    const int r = (int)(i - c * C);
    const int64_t base = ld_stream(chunk_ptr + c);
    const int64_t w = div_nonneg(ld_stream(chunk_ptr + c + 1) - base, C);
    const int32_t *cp = col + base + r;
    const V *vp = val + base + r;
    if (w > cap && ld_stream(cp + cap * C) >= 0) return;  // longer than the cap: the stream kernel's row
    V s[K];
#pragma unroll
    for (int q = 0; q < K; q++) s[q] = V(0);
    if constexpr (TWO) {
        int64_t k = 0;
        bool open = true;
        for (; k + S <= w; k += S) {
            int cc[S];
            V aa[S];
#pragma unroll
            for (int u = 0; u < S; u++) {
                cc[u] = ld_stream(cp + (k + u) * C);
                aa[u] = ld_stream(vp + (k + u) * C);
            }
#pragma unroll
            for (int u = 0; u < S; u++)
                if (cc[u] >= 0) {
                    V xr[K];
                    ld_xrow<V, K>(x, cc[u], ldx, xvec, xr);
#pragma unroll
                    for (int q = 0; q < K; q++) s[q] += aa[u] * xr[q];
                }
            if (cc[S - 1] < 0) {  // padding is a suffix of the row
                open = false;
                break;
            }
        }
        for (; open && k < w; k++) {
            const int cc = ld_stream(cp + k * C);
            if (cc < 0) break;
            const V aa = ld_stream(vp + k * C);
            V xr[K];
            ld_xrow<V, K>(x, cc, ldx, xvec, xr);
#pragma unroll
            for (int q = 0; q < K; q++) s[q] += aa * xr[q];
        }
    } else {
        for (int64_t k = 0; k < w; k += S) {
            int cc[S];
            V aa[S];
#pragma unroll
            for (int u = 0; u < S; u++) {
                cc[u] = -1;
                aa[u] = V(0);
                if (FLAT || k + u < w) {
                    const int64_t at = (FLAT ? min(k + u, w - 1) : k + u) * C;
                    cc[u] = ld_stream(cp + at);
                    aa[u] = ld_stream(vp + at);
                }
                if (FLAT && k + u >= w) cc[u] = -1;
            }
            if constexpr (K == 1) {
                V xv[S];
#pragma unroll
                for (int u = 0; u < S; u++)
                    xv[u] = FLAT ? ld_x(x + (int64_t)max(cc[u], 0) * ldx) : cc[u] >= 0 ? ld_x(x + (int64_t)cc[u] * ldx) : V(0);
#pragma unroll
                for (int u = 0; u < S; u++)
                    if (cc[u] >= 0) s[0] += aa[u] * xv[u];  // never 0 * x[0]: x may hold Inf or NaN
            } else {
#pragma unroll
                for (int u = 0; u < S; u++)
                    if (cc[u] >= 0) {
                        V xr[K];
                        ld_xrow<V, K>(x, cc[u], ldx, xvec, xr);
#pragma unroll
                        for (int q = 0; q < K; q++) s[q] += aa[u] * xr[q];
                    }
            }
            if (cc[S - 1] < 0) break;  // padding is a suffix of the row
        }
    }
    const int64_t row = reorder ? (int64_t)ld_stream(reorder + i) : i;
    V *yp = y + row * ldy;
#pragma unroll
    for (int q = 0; q < K; q++) yp[q] = row_out(PLAIN, alpha, s[q], beta, yp + q);
}

// BEHIND: launched behind the long rows' kernel (launch_behind), with which it
// shares nothing; one block outlasts that kernel, so that what follows is behind
// both.  Not for the forms of more slots (narrow ELL), whose loads the compiler
// no longer keeps in flight with the wait after them (20 -> 28 us).
template <typename V, int K, int S, bool PLAIN = false, bool FLAT = false, bool BEHIND = false, bool STRIDE = false,
          bool WAVE = false, bool TWO = STRIDE>
__global__ void __launch_bounds__(kBlock, (sliced_min_ctas<V, K, S, FLAT, WAVE>())) sliced_spmv_kernel(
    int m, int C, const int64_t *__restrict__ chunk_ptr, const int32_t *__restrict__ reorder,
    const int32_t *__restrict__ col, const V *__restrict__ val, const V *__restrict__ x, int64_t ldx, int xvec,
    V alpha, V beta, V *__restrict__ y, int64_t ldy, int64_t cap) {
    if constexpr (BEHIND) let_next_start();
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if constexpr (STRIDE) {
        for (; i < m; i += (int64_t)gridDim.x * blockDim.x)
            sliced_row<V, K, S, PLAIN, FLAT, TWO>(i, C, chunk_ptr, reorder, col, val, x, ldx, xvec, alpha, beta, y, ldy, cap);
    } else if (i < m) {
        sliced_row<V, K, S, PLAIN, FLAT, TWO>(i, C, chunk_ptr, reorder, col, val, x, ldx, xvec, alpha, beta, y, ldy,
                                               cap);
    }
    if constexpr (BEHIND)
        if (blockIdx.x == 0) wait_for_previous();
}

// Plan building: stored length of every stored row (padding is a suffix:
// binary search for the first slot with col < 0).
__global__ void stored_row_lengths(int64_t m, int C, const int64_t *__restrict__ chunk_ptr,
                                   const int32_t *__restrict__ col, int32_t *__restrict__ len) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t c = div_nonneg(i, C);
        const int r = (int)(i - c * C);
        const int64_t base = chunk_ptr[c];
        const int64_t w = div_nonneg(chunk_ptr[c + 1] - base, C);
        int64_t lo = 0, hi = w;  // first padding slot in [0, w]
        while (lo < hi) {
            const int64_t mid = (lo + hi) >> 1;
            if (col[base + mid * C + r] >= 0) lo = mid + 1;
            else hi = mid;
        }
        len[i] = (int32_t)lo;
    }
}

constexpr int kNumCaps = 12;  // the last: no cap
struct CapList {
    int64_t cap[kNumCaps];
};
constexpr int64_t kNoCap = INT64_MAX;

// What the cost model needs of one cap: warp steps and longest row of the
// thread pass without the rows past the cap, those rows and their nonzeros.
struct CapStats {
    unsigned long long slots, longest, rows, nnz;
};

// A warp per 32 stored rows (the rows a warp of the thread pass runs).
__global__ void __launch_bounds__(kBlock) cap_stats(int64_t m, const int32_t *__restrict__ len, const CapList caps,
                                                    CapStats *__restrict__ out) {
    __shared__ CapStats s_out[kNumCaps];
    const int lane = threadIdx.x & 31;
    for (int t = threadIdx.x; t < kNumCaps; t += kBlock) s_out[t] = CapStats{0, 0, 0, 0};
    __syncthreads();
    unsigned long long slots = 0, longest = 0, rows = 0, nnz = 0;  // lane q: of cap q
    const int64_t warps = ((int64_t)gridDim.x * kBlock) >> 5;
    for (int64_t b = (((int64_t)blockIdx.x * kBlock + threadIdx.x) >> 5) * 32; b < m; b += warps * 32) {
        const int l = b + lane < m ? len[b + lane] : 0;
        const int most = __reduce_max_sync(0xffffffffu, l);
#pragma unroll
        for (int q = 0; q < kNumCaps; q++) {
            unsigned mx = (unsigned)most, over = 0, n = 0;
            if ((int64_t)most > caps.cap[q]) {  // warp-uniform
                const bool past = (int64_t)l > caps.cap[q];
                mx = __reduce_max_sync(0xffffffffu, past ? 0u : (unsigned)l);
                over = __popc(__ballot_sync(0xffffffffu, past));
                n = __reduce_add_sync(0xffffffffu, past ? (unsigned)l : 0u);
            }
            if (lane == q) {
                slots += mx;
                longest = max(longest, (unsigned long long)mx);
                rows += over;
                nnz += n;
            }
        }
    }
    if (lane < kNumCaps) {
        atomicAdd(&s_out[lane].slots, slots);
        atomicMax(&s_out[lane].longest, longest);
        atomicAdd(&s_out[lane].rows, rows);
        atomicAdd(&s_out[lane].nnz, nnz);
    }
    __syncthreads();
    if (threadIdx.x < kNumCaps) {
        CapStats *o = out + threadIdx.x;
        const CapStats v = s_out[threadIdx.x];
        atomicAdd(&o->slots, v.slots);
        atomicMax(&o->longest, v.longest);
        atomicAdd(&o->rows, v.rows);
        atomicAdd(&o->nnz, v.nnz);
    }
}

// Rows past the cap: a one in the upper word and their length in the lower, so
// that one scan counts both.
__global__ void overflow_flags(int64_t m, int64_t cap, const int32_t *__restrict__ len, int64_t *__restrict__ flag) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x)
        flag[i] = (int64_t)len[i] > cap ? (int64_t(1) << 32) + len[i] : 0;
}

// pos: the scan of the flags.  Stored position, y row and first compact element
// of every overflow row (optr[nov] = novf).
__global__ void overflow_rows(int64_t m, int64_t cap, const int32_t *__restrict__ len, const int64_t *__restrict__ pos,
                              const int32_t *__restrict__ reorder, int64_t nov, int32_t novf,
                              int32_t *__restrict__ rows, int32_t *__restrict__ yrow, int32_t *__restrict__ optr) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
        if (i == 0) optr[nov] = novf;
        if ((int64_t)len[i] <= cap) continue;
        const int32_t o = (int32_t)(pos[i] >> 32);
        rows[o] = (int32_t)i;
        yrow[o] = reorder ? reorder[i] : (int32_t)i;
        optr[o] = (int32_t)pos[i];
    }
}

// Copies the overflow rows out of the slab: a warp per 256 consecutive elements
// of the compact arrays (so that a row of 50k elements does not keep one warp),
// eight a lane with their loads in flight together; each element's row is the
// one before's or one soon after.  3.5M elements FP64, C = 4: 43 us (51 with a
// binary search and one element in flight at a time).
constexpr int kCopyTile = 2048;

template <typename V>
__global__ void __launch_bounds__(kBlock) copy_overflow(int64_t nov, int32_t novf, int C,
                                                        const int32_t *__restrict__ rows,
                                                        const int32_t *__restrict__ optr,
                                                        const int64_t *__restrict__ chunk_ptr,
                                                        const int32_t *__restrict__ col, const V *__restrict__ val,
                                                        int32_t *__restrict__ ocol, V *__restrict__ oval) {
    constexpr int U = kCopyTile / kBlock;
    const int lane = threadIdx.x & 31;
    const int64_t e0 = (int64_t)blockIdx.x * kCopyTile + (threadIdx.x >> 5) * (32 * U);  // the warp's elements
    if (e0 >= novf) return;  // warp-uniform
    const int64_t r1 = warp_last_le(optr, nov, (int32_t)(min(e0 + 32 * U, (int64_t)novf) - 1), lane);
    int64_t r = warp_last_le(optr, r1 + 1, (int32_t)e0, lane);
    int64_t i[U], k[U];
#pragma unroll
    for (int u = 0; u < U; u++) {  // the row of each element: this one's or soon after
        const int64_t e = min(e0 + u * 32 + lane, (int64_t)novf - 1);
        if (r < r1 && __ldg(optr + r + 1) <= e) {
            int64_t hi = r1;
            r++;
            while (r < hi) {
                const int64_t mid = (r + hi + 1) >> 1;
                if (__ldg(optr + mid) <= e) r = mid;
                else hi = mid - 1;
            }
        }
        k[u] = e - __ldg(optr + r);
        i[u] = __ldg(rows + r);
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
        const int64_t c = div_nonneg(i[u], C);
        k[u] = __ldg(chunk_ptr + c) + k[u] * C + (i[u] - c * C);
    }
    int32_t oc[U];
    V ov[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
        oc[u] = col[k[u]];
        ov[u] = val[k[u]];
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
        const int64_t e = e0 + u * 32 + lane;
        if (e < novf) {
            ocol[e] = oc[u];
            oval[e] = ov[u];
        }
    }
}

struct SlicedView {
    int64_t m;
    int32_t C;
    const int64_t *chunk_ptr;
    const int32_t *reorder;
    const int32_t *col;
    const void *val;
    int64_t nchunks;  // 0: ELL
    int32_t width;    // ELL
    int64_t cols;     // rows of X
    int32_t align;    // of the chunks' widths
    bool sorted;      // by length over the whole matrix (SELL-c-R)
};

// Cost model of the cap, in picoseconds of GB300 time (fitted to measured
// times of power-law matrices of 0.1-4M rows at caps of 1 to 512).  A nonzero
// costs kNnzPs in either kernel, its x gather; the thread pass no less than
// kWarpSlotPs per warp and slot it runs (a warp runs as many slots as its
// longest row within the cap), nor than a warp of average length's chain,
// kSlotChainPs per slot, plus what its longest thread's chain goes on beyond
// that (1M rows FP64, sigma = 4096: caps of 32, 128, 512 take 115, 171, 396 us;
// 1M even rows of 50 have no such rest: 185 us in the thread pass, 212 through the
// stream kernel); the overflow kOvfRowPs per row and kOvfLaunchPs for its
// launches.
constexpr double kWarpSlotPs = 73.0;
constexpr double kSlotChainPs = 0.5e6;
constexpr double kNnzPs = 3.9;
constexpr double kOvfRowPs = 20.0;
constexpr double kOvfLaunchPs = 5.0e6;
// Rows sorted by length over the whole matrix leave no lane of a warp idle, and the
// longest ones start first: without very long ones they stay in the thread pass
// (SELL-c-R, 1.5M 4x4 block rows of up to 28: FP32 27.3 us with a cap of 8, 19.5
// without; k = 2 28.3 and 20.9; FP64 32.0 and 26.9).
constexpr int64_t kShortRow = 64;
constexpr int64_t kWholeRows = 500000;
constexpr CapList kCaps = {{8, 12, 16, 24, 32, 48, 64, 96, 128, 256, 512, kNoCap}};

// The candidate of least modelled time (ties: no cap, then the largest).
int choose_cap(const CapStats (&st)[kNumCaps], int64_t m, int64_t total_nnz) {
    const double warps = (double)((m + 31) / 32);
    int best = kNumCaps - 1;
    double best_cost = 0;
    for (int t = kNumCaps - 1; t >= 0; t--) {
        const double average = (double)st[t].slots / warps;
        const double thread = std::max({kWarpSlotPs * (double)st[t].slots,
                                        kNnzPs * (double)(total_nnz - (int64_t)st[t].nnz), kSlotChainPs * average}) +
                              kSlotChainPs * ((double)st[t].longest - average);
        const double cost = thread + kNnzPs * (double)st[t].nnz + kOvfRowPs * (double)st[t].rows +
                            (st[t].rows > 0 ? kOvfLaunchPs : 0.0);
        if (t == kNumCaps - 1 || cost < best_cost) {
            best_cost = cost;
            best = t;
        }
    }
    return best;
}

void free_overflow(Plan *p, sspmv_stream_t s) {
    free_stream_plan(p->stream, s);
    dfree(p->extra[0], s);
    p->extra[0] = nullptr;
    p->extra_i[1] = p->extra_i[4] = 0;
}

// Overflow plan of a sliced matrix, built on its first SpMV (and again after
// sspmv_set_kernel changes the cap).  extra[0] y row of every overflow row (the
// stream plan's row list), then, extra_i[8] and [9] bytes on, their columns and
// values; p->stream the stream plan; extra_i[1] overflow rows, [2] the cap, [3] the
// kernel parameter the plan was built for, [4] overflow nonzeros, [5] the
// longest row, [7] built.
sspmv_status ensure_overflow_plan(const sspmv_features *f, const SlicedView &v, Plan *p, sspmv_stream_t s) {
    if (p->extra_i[7] && p->extra_i[3] == p->param) return SSPMV_OK;
    std::lock_guard<PlanMutex> g(plan_mutex());
    if (p->extra_i[7] && p->extra_i[3] == p->param) return SSPMV_OK;
    p->extra_i[7] = 0;
    free_overflow(p, s);  // a plan for another cap, or one whose building failed
    const int64_t m = v.m;
    const unsigned grid = grid_for(m, 256, (int64_t)num_sms() * 32);
    const size_t sv = vsize(f->value_type);
    unsigned char *stats = nullptr, *temp = nullptr;  // lengths and the caps' statistics; positions and row lists
    CapList caps = kCaps;
    if (p->param > 0) caps.cap[0] = p->param;
    int64_t nov = 0, novf = 0, cap = kNoCap, longest = 0;
    auto up = [](size_t n) { return (n + 255) / 256 * 256; };
    auto build = [&]() -> sspmv_status {
        CapStats st[kNumCaps];
        SSPMV_TRY(dalloc(&stats, up(sizeof(st)) + (size_t)m * 4, s));
        CapStats *dst = (CapStats *)stats;
        int32_t *len = (int32_t *)(stats + up(sizeof(st)));
        SSPMV_CUDA_TRY(cudaMemsetAsync(dst, 0, sizeof(st), cu(s)));
        stored_row_lengths<<<grid, 256, 0, cu(s)>>>(m, v.C, v.chunk_ptr, v.col, len);
        SSPMV_LAUNCH_CHECK();
        cap_stats<<<grid_for(m, kBlock, (int64_t)num_sms() * 4), kBlock, 0, cu(s)>>>(m, len, caps, dst);
        SSPMV_LAUNCH_CHECK();
        SSPMV_CUDA_TRY(cudaMemcpyAsync(st, dst, sizeof(st), cudaMemcpyDeviceToHost, cu(s)));
        SSPMV_CUDA_TRY(cudaStreamSynchronize(cu(s)));
        longest = (int64_t)st[kNumCaps - 1].longest;
        const bool whole = v.sorted && m > kWholeRows && longest <= kShortRow;
        const int pick = p->param > 0 ? 0 : whole ? kNumCaps - 1 : choose_cap(st, m, f->num_nnzs);
        cap = caps.cap[pick];
        nov = (int64_t)st[pick].rows;
        novf = (int64_t)st[pick].nnz;
        if (novf > 0x7fffffff) return fail(SSPMV_NOT_SUPPORTED, "overflow of the long rows exceeds the int32 range");
        if (nov == 0) return SSPMV_OK;
        const size_t rows_at = up((size_t)m * 8), optr_at = rows_at + up((size_t)nov * 4);
        SSPMV_TRY(dalloc(&temp, optr_at + ((size_t)nov + 1) * 4, s));
        int64_t *pos = (int64_t *)temp;
        int32_t *rows = (int32_t *)(temp + rows_at), *optr = (int32_t *)(temp + optr_at);
        const size_t col_at = up((size_t)nov * 4), val_at = col_at + up((size_t)novf * 4);
        unsigned char *kept = nullptr;  // the plan's as soon as it exists (free_overflow)
        SSPMV_TRY(dalloc(&kept, val_at + (size_t)novf * sv, s));
        p->extra[0] = kept;
        p->extra_i[8] = (int64_t)col_at;
        p->extra_i[9] = (int64_t)val_at;
        int32_t *yrow = (int32_t *)kept, *ocol = (int32_t *)(kept + col_at);
        overflow_flags<<<grid, 256, 0, cu(s)>>>(m, cap, len, pos);
        SSPMV_LAUNCH_CHECK();
        SSPMV_TRY(exclusive_scan_i64(pos, pos, m, nullptr, s));
        overflow_rows<<<grid, 256, 0, cu(s)>>>(m, cap, len, pos, v.reorder, nov, (int32_t)novf, rows, yrow, optr);
        SSPMV_LAUNCH_CHECK();
        SSPMV_TRY(dispatch_value(f->value_type, [&](auto tag) -> sspmv_status {
            using V = decltype(tag);
            copy_overflow<V><<<grid_for(novf, kCopyTile), kBlock, 0, cu(s)>>>(
                nov, (int32_t)novf, v.C, rows, optr, v.chunk_ptr, v.col, (const V *)v.val, ocol, (V *)(kept + val_at));
            SSPMV_LAUNCH_CHECK();
            return SSPMV_OK;
        }));
        // no empty rows, and no split ones to wait for if all are short
        return ensure_stream_plan(p->stream, nov, novf, optr, yrow, f->value_type, s, 0, -1,
                                  longest <= kStreamWholeRow ? 0 : -1);
    };
    const sspmv_status st = build();
    dfree(stats, s);
    dfree(temp, s);
    SSPMV_TRY(st);
    p->extra_i[1] = nov;
    p->extra_i[2] = nov > 0 ? cap : kNoCap;
    p->extra_i[3] = p->param;
    p->extra_i[4] = novf;
    p->extra_i[5] = longest;
    p->extra_i[7] = 1;
    return SSPMV_OK;
}

template <typename V, int K>
sspmv_status launch_sliced(const SlicedView &v, Plan *p, V alpha, const V *x, int64_t ldx, V beta, V *y,
                           int64_t ldy, sspmv_stream_t s) {
    // Two or four FP32 right-hand sides on many rows, none very long: the thread
    // pass alone, whatever the cap (S-ELL, block rows, k = 2: 3M rows 84.5 us with
    // it, 70 so, 1M 30.4 and 27.6, but 100k 5.9 and 8.4).
    const bool whole = p && sizeof(V) == 4 && (K == 2 || K == 4) && v.m > kWholeRows && p->extra_i[5] <= kShortRow;
    const int64_t nov = p && !whole && stream_takes_strides(ldx, ldy, sizeof(V)) ? p->extra_i[1] : 0;
    StreamView lv;
    if (nov > 0) {  // the long rows first: the thread pass starts under their last wave
        const unsigned char *kept = (const unsigned char *)p->extra[0];
        lv = stream_view(p->stream, p->extra_i[4], (const int32_t *)(kept + p->extra_i[8]), kept + p->extra_i[9]);
        SSPMV_TRY((launch_stream_windows<V, K>(lv, p->stream, alpha, x, ldx, beta, y, ldy, v.cols, s)));
    }
    // A thread per row and no grid stride: a fixed grid gave the same blocks the
    // long rows at the head of every sigma slice (4M rows FP32, sigma = 4096:
    // 580 us so, 328 with blocks scheduled as they finish).
    unsigned grid = grid_for(v.m, kBlock);
    const int xvec = xrow_vec(x, ldx, sizeof(V), K);
    auto go = [&](auto kernel) {
        kernel<<<grid, kBlock, 0, cu(s)>>>((int)v.m, v.C, v.chunk_ptr, v.reorder, v.col, (const V *)v.val, x, ldx,
                                           xvec, alpha, beta, y, ldy, nov > 0 ? p->extra_i[2] : kNoCap);
        return cudaSuccess;
    };
    auto go_behind = [&](auto kernel) {
        return launch_behind(kernel, grid, kBlock, cu(s), (int)v.m, v.C, v.chunk_ptr, v.reorder, v.col,
                             (const V *)v.val, x, ldx, xvec, alpha, beta, y, ldy, p->extra_i[2]);
    };
    cudaError_t launched = cudaSuccess;
    if constexpr (K == 1) {
        const bool plain = alpha == V(1) && beta == V(0);  // y = sum
        auto slots = [&](auto tag) {
            constexpr int S = decltype(tag)::value;
            constexpr bool flat = S > 4 && sizeof(V) == 4;
            if (plain) go(sliced_spmv_kernel<V, K, S, true, flat>);
            else go(sliced_spmv_kernel<V, K, S, false, flat>);
        };
        // the widest chunk
        const int64_t w = v.nchunks > 0 ? (p->extra_i[5] + v.align - 1) / v.align * v.align : v.width;
        const bool ell = v.nchunks == 0;
        if (nov > 0) {
            launched = plain ? go_behind(sliced_spmv_kernel<V, K, 4, true, false, true, false, false, true>)
                             : go_behind(sliced_spmv_kernel<V, K, 4, false, false, true, false, false, true>);
        } else if (w <= 3 || (sizeof(V) == 8 && !ell && (w == 6 || w == 7)) || (ell && w == 4)) {
            // tested loads, where the slots left over would be read one by one
            // (S-ELL without padding, 1M rows of 3, FP64: 22.1 us so, 17.9 tested;
            // of 7 36.6 and 32.7; FP32, of 3, 17.6 and 15.5)
            bool wave = false;
            if constexpr (sizeof(V) == 8) {
                wave = w <= 2;
                if (wave && plain) go(sliced_spmv_kernel<V, K, 4, true, false, false, false, true>);
                else if (wave) go(sliced_spmv_kernel<V, K, 4, false, false, false, false, true>);
            }
            if (!wave) slots(std::integral_constant<int, 4>());
        } else if (!ell || w > 12 || (sizeof(V) == 4 && (w == 7 || w == 8))) {
            // rows of many lengths, or of more slots than registers hold at once
            // (ELL of 8 random columns, 1M rows, FP32: 35.3 us with all of them
            // in flight, 31.7 so)
            bool wave = false;
            if constexpr (sizeof(V) == 8) {
                wave = (int64_t)grid <= 8 * num_sms() && ((int64_t)grid > 6 * num_sms() || w > 32);
                if (wave && plain) go(sliced_spmv_kernel<V, K, 4, true, false, false, false, true, true>);
                else if (wave) go(sliced_spmv_kernel<V, K, 4, false, false, false, false, true, true>);
            }
            if (!wave && plain) go(sliced_spmv_kernel<V, K, 4, true, false, false, false, false, true>);
            else if (!wave) go(sliced_spmv_kernel<V, K, 4, false, false, false, false, false, true>);
        } else if (w <= 6 || (sizeof(V) == 4 && w > 10)) {  // 12 at once: 53.3 us, 6 and 6: 45.0
            slots(std::integral_constant<int, 6>());
        } else if (w <= 8) {
            if constexpr (sizeof(V) == 8) slots(std::integral_constant<int, 8>());
        } else if (w <= 10) {
            slots(std::integral_constant<int, 10>());
        } else {
            if constexpr (sizeof(V) == 8) slots(std::integral_constant<int, 12>());
        }
    } else {
        // Two FP32 right-hand sides, and any number on rows sorted by length:
        // a fixed grid striding over the rows (5-point Laplacian 1M, FP32, k = 2,
        // 18.1 us in blocks of 256 rows, 16.2 so; SELL-c-R of block rows k = 8
        // 42.2 and 36.7), otherwise blocks (banded FP32 k = 4 28.0 and 29.2,
        // FP64 k = 2 42 and 50).
        const bool stride = (K == 2 && sizeof(V) == 4) || (K > 2 && v.sorted) || (whole && !v.reorder && p->extra_i[1] > 0);
        if (nov > 0) {
            launched = go_behind(sliced_spmv_kernel<V, K, 4, false, false, true>);
        } else if (stride) {
            grid = grid_for(v.m, kBlock, (int64_t)num_sms() * 16);
            go(sliced_spmv_kernel<V, K, 4, false, false, false, true>);
        } else {
            go(sliced_spmv_kernel<V, K, 4>);
        }
    }
    SSPMV_CUDA_TRY(launched);
    SSPMV_LAUNCH_CHECK();
    return nov > 0 ? launch_split_rows<V, K>(lv, p->stream, alpha, beta, y, ldy, s) : SSPMV_OK;
}

sspmv_status spmm_sliced(const sspmv_features *f, const SlicedView &v, double alpha, int32_t k, const void *X,
                         int64_t ldx, double beta, void *Y, int64_t ldy, sspmv_stream_t s) {
    SSPMV_TRY(check_spmm_args(f, k, X, ldx, Y, ldy));
    if (v.m == 0) return SSPMV_OK;
    Plan *p = nullptr;
    if (v.nchunks > 0) {  // ELL (nchunks == 0 here) keeps every row in the thread pass
        p = get_plan(f);
        if (!p) return fail(SSPMV_OUT_OF_MEMORY, "plan allocation failed");
        SSPMV_TRY(ensure_overflow_plan(f, v, p, s));
    }
    return dispatch_value(f->value_type, [&](auto tag) -> sspmv_status {
        using V = decltype(tag);
        return for_rhs_chunks<V>(k, (const V *)X, (V *)Y, [&](int32_t step, const V *xs, V *ys) {
            const V a = (V)alpha, b = (V)beta;
            switch (step) {
            case 8: return launch_sliced<V, 8>(v, p, a, xs, ldx, b, ys, ldy, s);
            case 4: return launch_sliced<V, 4>(v, p, a, xs, ldx, b, ys, ldy, s);
            case 2: return launch_sliced<V, 2>(v, p, a, xs, ldx, b, ys, ldy, s);
            default: return launch_sliced<V, 1>(v, p, a, xs, ldx, b, ys, ldy, s);
            }
        });
    });
}

// ------------------------------------------------------------ converters --
// keys for the slice sort: position p holds row m-1-p (descending input order)
__global__ void sell_sort_keys(int64_t m, int64_t sigma, int32_t maxlen, const int32_t *__restrict__ rp,
                               uint64_t *__restrict__ keys, uint32_t *__restrict__ vals) {
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < m; p += (int64_t)gridDim.x * blockDim.x) {
        const int64_t row = m - 1 - p;
        const int32_t len = rp[row + 1] - rp[row];
        keys[p] = (uint64_t)(row / sigma) * (uint64_t)(maxlen + 1) + (uint64_t)(maxlen - len);
        vals[p] = (uint32_t)row;
    }
}

// The same order by a block per whole slices, in shared memory: slices of up to
// kSortRows rows (shorter ones several to a block).  A stable radix sort of
// 8-bit digits of (longest - length) over the block's rows in descending order,
// then of the slice where there are several; a warp ranks 32 IT consecutive
// rows, 32 at a time.  SELL-c-sigma (16384, 4) of 500k rows: 23.6 us; the
// same by the radix sort of all rows (three passes of five launches, and the
// longest row read back for the keys) 137.
constexpr int kSortThreads = 1024;
constexpr int kSortRows = 16 * kSortThreads;
constexpr int kSortSlices = 256;  // slices a block takes at most

template <int IT>
constexpr size_t sort_smem() {
    return (size_t)kSortThreads * IT * (sizeof(uint32_t) + sizeof(uint16_t)) + 32 * 256 * sizeof(uint16_t);
}

template <int IT>
__global__ void __launch_bounds__(kSortThreads) sell_sort_slices(int64_t m, int64_t sigma, int64_t seg,
                                                                 const int32_t *__restrict__ rp,
                                                                 int32_t *__restrict__ reorder) {
    constexpr unsigned kFull = 0xffffffffu;
    extern __shared__ __align__(16) unsigned char sort_smem_raw[];
    uint32_t *s_key = reinterpret_cast<uint32_t *>(sort_smem_raw);
    uint16_t *s_idx = reinterpret_cast<uint16_t *>(s_key + kSortThreads * IT);
    uint16_t *s_cnt = s_idx + kSortThreads * IT;  // [warp][digit]: the warp's rows, then their first place
    __shared__ uint32_t s_first[256];             // place of the first row of a digit
    __shared__ uint32_t s_longest;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t b0 = (int64_t)blockIdx.x * seg;
    const int n = (int)min(seg, m - b0);
    uint16_t *cnt = s_cnt + warp * 256;
    uint32_t key[IT];
    uint16_t idx[IT];
    if (threadIdx.x == 0) s_longest = 0;
    __syncthreads();
    uint32_t most = 0;
#pragma unroll
    for (int u = 0; u < IT; u++) {
        const int t = (warp * IT + u) * 32 + lane;
        idx[u] = t < n ? (uint16_t)(n - 1 - t) : 0;
        key[u] = t < n ? (uint32_t)(rp[b0 + idx[u] + 1] - rp[b0 + idx[u]]) : 0;
        most = max(most, key[u]);
    }
    most = __reduce_max_sync(kFull, most);
    if (lane == 0) atomicMax(&s_longest, most);
    __syncthreads();
    most = s_longest;
#pragma unroll
    for (int u = 0; u < IT; u++) key[u] = most - key[u];

    const int digits = (39 - __clz(most | 1)) / 8;  // of the lengths; one pass more for the slices
    for (int pass = 0; pass < digits + (seg > sigma ? 1 : 0); pass++) {
        auto digit = [&](int u) {
            return pass < digits ? (int)(key[u] >> (8 * pass)) & 0xff : (int)((uint32_t)idx[u] / (uint32_t)sigma);
        };
        for (int d = lane; d < 128; d += 32) reinterpret_cast<uint32_t *>(cnt)[d] = 0;
        __syncwarp();
        uint16_t rank[IT];
#pragma unroll
        for (int u = 0; u < IT; u++) {
            const bool valid = (warp * IT + u) * 32 + lane < n;
            const int d = valid ? digit(u) : 256;
            const unsigned peers = __match_any_sync(kFull, d);
            const int before = valid ? cnt[d] : 0;
            rank[u] = (uint16_t)(before + __popc(peers & ((1u << lane) - 1u)));
            __syncwarp();
            if (valid && lane == __ffs(peers) - 1) cnt[d] = (uint16_t)(before + __popc(peers));
            __syncwarp();
        }
        __syncthreads();
        if (threadIdx.x < 256) {
            uint32_t run = 0;
            for (int w = 0; w < 32; w++) {
                const uint32_t c = s_cnt[w * 256 + threadIdx.x];
                s_cnt[w * 256 + threadIdx.x] = (uint16_t)run;
                run += c;
            }
            s_first[threadIdx.x] = run;
        }
        __syncthreads();
        if (warp == 0) {  // exclusive scan of the 256 digits, 8 a lane
            uint32_t v[8], sum = 0;
#pragma unroll
            for (int q = 0; q < 8; q++) {
                v[q] = s_first[lane * 8 + q];
                sum += v[q];
            }
            uint32_t inc = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t up = __shfl_up_sync(kFull, inc, o);
                if (lane >= o) inc += up;
            }
            uint32_t run = inc - sum;
#pragma unroll
            for (int q = 0; q < 8; q++) {
                s_first[lane * 8 + q] = run;
                run += v[q];
            }
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < IT; u++) {
            if ((warp * IT + u) * 32 + lane < n) {
                const int d = digit(u);
                const int pos = (int)s_first[d] + cnt[d] + rank[u];
                s_key[pos] = key[u];
                s_idx[pos] = idx[u];
            }
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < IT; u++) {
            const int t = (warp * IT + u) * 32 + lane;
            if (t < n) {
                key[u] = s_key[t];
                idx[u] = s_idx[t];
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int u = 0; u < IT; u++) {
        const int t = (warp * IT + u) * 32 + lane;
        if (t < n) reorder[b0 + t] = (int32_t)(b0 + idx[u]);
    }
}

sspmv_status sort_slices(int64_t m, int64_t sigma, const int32_t *rp, int32_t *reorder, sspmv_stream_t s) {
    const int64_t seg = sigma * std::max<int64_t>(1, std::min<int64_t>(kSortSlices, 2 * kSortThreads / sigma));
    auto go = [&](auto tag) -> sspmv_status {
        constexpr int IT = decltype(tag)::value;
        SSPMV_CUDA_TRY(cudaFuncSetAttribute(sell_sort_slices<IT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            (int)sort_smem<IT>()));
        sell_sort_slices<IT><<<(unsigned)((m + seg - 1) / seg), kSortThreads, sort_smem<IT>(), cu(s)>>>(m, sigma, seg, rp,
                                                                                                      reorder);
        SSPMV_LAUNCH_CHECK();
        return SSPMV_OK;
    };
    if (seg <= 2 * kSortThreads) return go(std::integral_constant<int, 2>());
    if (seg <= 4 * kSortThreads) return go(std::integral_constant<int, 4>());
    if (seg <= 8 * kSortThreads) return go(std::integral_constant<int, 8>());
    return go(std::integral_constant<int, 16>());
}

__global__ void copy_u32_to_i32(int64_t n, const uint32_t *__restrict__ in, int32_t *__restrict__ out) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = (int32_t)in[i];
}

// chunk width = max row length in the chunk, rounded up to `align`.  Pass 1
// (thread per stored row position) folds row lengths into width[] with
// atomicMax -- one atomic per block when the block's rows lie in one chunk
// (ELL is a single chunk of all rows), one per row otherwise; width[] starts
// at zero.  Pass 2 rounds and sizes each chunk.
__global__ void chunk_row_max(int64_t m, int32_t C, const int32_t *__restrict__ rp,
                              const int32_t *__restrict__ reorder, int32_t *__restrict__ width) {
    __shared__ int s_max[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    for (int64_t base = (int64_t)blockIdx.x * blockDim.x; base < m; base += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = base + threadIdx.x;
        int len = 0;
        if (i < m) {
            const int64_t r = reorder ? reorder[i] : i;
            len = rp[r + 1] - rp[r];
        }
        const int64_t last = min(base + (int64_t)blockDim.x, m) - 1;
        if (base / C == last / C) {  // block-uniform branch
            int v = len;
            for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
            if (lane == 0) s_max[warp] = v;
            __syncthreads();
            if (threadIdx.x == 0) {
                int b = 0;
                for (int w = 0; w < nwarps; w++) b = max(b, s_max[w]);
                if (b > 0) atomicMax(width + base / C, b);
            }
            __syncthreads();
        } else if (len > 0) {
            atomicMax(width + i / C, len);
        }
    }
}

__global__ void chunk_widths(int64_t nchunks, int32_t C, int32_t align, int32_t *__restrict__ width,
                             int64_t *__restrict__ slots) {
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < nchunks;
         c += (int64_t)gridDim.x * blockDim.x) {
        const int32_t w = ((width[c] + align - 1) / align) * align;
        width[c] = w;
        slots[c] = (int64_t)w * C;
    }
}

// Copies the CSR rows into the slab, padding included: a warp per 256
// consecutive slots, eight a lane with their loads in flight together; a slot's
// chunk is the one before's or one soon after (a chunk as wide as a 38k-nonzero
// row is spread over many blocks).  Writes are consecutive; neighbouring slots
// read C rows at a time, and the warp's 256 / C slots of each row share their
// sectors.  For chunks of up to kFillChunk rows: SELL-c-sigma (16384, 4) of 500k
// power-law rows FP64 704 us with a thread per row (the rows of 256 and more by
// the block that holds them, all the longest in one block) after two fills, 94
// with a binary search for each slot, now 71 (242 MB: 36 us).
constexpr int kFillTile = 2048;
constexpr int kFillChunk = 256;

template <typename V>
__global__ void __launch_bounds__(256, 6) sliced_fill_slots(int64_t m, int32_t C, int64_t nchunks, int64_t total,
                                                         const int64_t *__restrict__ chunk_ptr,
                                                         const int32_t *__restrict__ reorder,
                                                         const int32_t *__restrict__ rp,
                                                         const int32_t *__restrict__ ci, const V *__restrict__ cv,
                                                         int32_t *__restrict__ col, V *__restrict__ val) {
    constexpr int U = kFillTile / 256;
    const int lane = threadIdx.x & 31;
    const int64_t e0 = (int64_t)blockIdx.x * kFillTile + (threadIdx.x >> 5) * (32 * U);  // the warp's slots
    if (e0 >= total) return;  // warp-uniform
    const int64_t c1 = warp_last_le(chunk_ptr, nchunks, min(e0 + 32 * U, total) - 1, lane);
    int64_t c = warp_last_le(chunk_ptr, c1 + 1, e0, lane);
    int64_t row[U];
    int32_t k[U];  // slot within the row; -1: no such row
#pragma unroll
    for (int u = 0; u < U; u++) {  // the chunk of each slot: this one's or soon after
        const int64_t e = e0 + u * 32 + lane;
        k[u] = -1;
        row[u] = 0;
        if (e < total) {
            if (c < c1 && __ldg(chunk_ptr + c + 1) <= e) {
                int64_t hi = c1;
                c++;
                while (c < hi) {
                    const int64_t mid = (c + hi + 1) >> 1;
                    if (__ldg(chunk_ptr + mid) <= e) c = mid;
                    else hi = mid - 1;
                }
            }
            const int64_t at = e - __ldg(chunk_ptr + c), kk = div_nonneg(at, C), i = c * C + (at - kk * C);
            if (i < m) {
                k[u] = (int32_t)kk;
                row[u] = i;
            }
        }
    }
    if (reorder) {
#pragma unroll
        for (int u = 0; u < U; u++) row[u] = __ldg(reorder + row[u]);
    }
    int32_t at[U];  // nonzero of the slot, -1: padding
#pragma unroll
    for (int u = 0; u < U; u++) {
        const int32_t s0 = __ldg(rp + row[u]), s1 = __ldg(rp + row[u] + 1);
        at[u] = k[u] >= 0 && k[u] < s1 - s0 ? s0 + k[u] : -1;
    }
    int32_t oc[U];
    V ov[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
        oc[u] = __ldg(ci + max(at[u], 0));
        ov[u] = __ldg(cv + max(at[u], 0));
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
        const int64_t e = e0 + u * 32 + lane;
        if (e < total) {
            col[e] = at[u] >= 0 ? oc[u] : -1;
            val[e] = at[u] >= 0 ? ov[u] : V(0);
        }
    }
}

// The same for wider chunks (ELL is one of num_rows rows) after the slab was
// filled with padding: a thread per stored row, except rows of kFillLong
// nonzeros or more, which the CTA holding them copies together
// after its short rows (one thread walking a 38k-nonzero row alone took
// milliseconds).
constexpr int64_t kFillLong = 256;

template <typename V>
__global__ void __launch_bounds__(256) sliced_fill(int64_t m, int32_t C, const int64_t *__restrict__ chunk_ptr,
                                                   const int32_t *__restrict__ reorder,
                                                   const int32_t *__restrict__ rp, const int32_t *__restrict__ ci,
                                                   const V *__restrict__ cv, int32_t *__restrict__ col,
                                                   V *__restrict__ val) {
    __shared__ int64_t s_long[256];
    __shared__ int s_count;
    for (int64_t b0 = (int64_t)blockIdx.x * blockDim.x; b0 < m; b0 += (int64_t)gridDim.x * blockDim.x) {
        if (threadIdx.x == 0) s_count = 0;
        __syncthreads();
        const int64_t i = b0 + threadIdx.x;
        if (i < m) {
            const int64_t r = reorder ? reorder[i] : i;
            const int64_t s0 = rp[r], len = rp[r + 1] - s0;
            if (len >= kFillLong) {
                s_long[atomicAdd(&s_count, 1)] = i;
            } else {
                const int64_t ic = div_nonneg(i, C);
                const int64_t base = chunk_ptr[ic] + (i - ic * C);
                for (int64_t k = 0; k < len; k++) {
                    col[base + k * C] = ci[s0 + k];
                    val[base + k * C] = cv[s0 + k];
                }
            }
        }
        __syncthreads();
        for (int t = 0; t < s_count; t++) {  // CTA-uniform
            const int64_t li = s_long[t];
            const int64_t r = reorder ? reorder[li] : li;
            const int64_t s0 = rp[r], len = rp[r + 1] - s0;
            const int64_t lc = div_nonneg(li, C);
            const int64_t base = chunk_ptr[lc] + (li - lc * C);
            for (int64_t k = threadIdx.x; k < len; k += blockDim.x) {
                col[base + k * C] = ci[s0 + k];
                val[base + k * C] = cv[s0 + k];
            }
        }
        __syncthreads();  // s_long / s_count are reused by the next round
    }
}

struct SlicedBuild {
    int32_t *reorder = nullptr;
    int32_t *width = nullptr;
    int64_t *chunk_ptr = nullptr;
    int64_t total = 0;
    int32_t *col = nullptr;
    void *val = nullptr;
    int64_t nchunks = 0;
    void release(sspmv_stream_t s) {
        dfree(reorder, s);
        dfree(width, s);
        dfree(chunk_ptr, s);
        dfree(col, s);
        dfree(val, s);
        *this = SlicedBuild();
    }
};

// sigma: 0 = no reordering (S-ELL / ELL), otherwise the slice height
// (>= num_rows for SELL-c-R).
sspmv_status build_sliced(const sspmv_csr *A, int32_t C, int32_t align, int64_t sigma, SlicedBuild &b,
                          sspmv_stream_t s) {
    const int64_t m = A->f.num_rows;
    const int32_t vt = A->f.value_type;
    b.nchunks = (m + C - 1) / C;
    const unsigned g = grid_for(m, 256, (int64_t)num_sms() * 16);
    sspmv_status st = SSPMV_OK;
    if (sigma > 0) {
        st = dalloc(&b.reorder, (size_t)m, s);
        if (st == SSPMV_OK && m > 0) {
            if (sigma <= kSortRows) {
                st = sort_slices(m, sigma, A->row_offset, b.reorder, s);
            } else {
                int32_t maxlen = 0;
                uint64_t *keys = nullptr;
                uint32_t *vals = nullptr;
                st = max_row_length(A->row_offset, m, &maxlen, s);
                if (st == SSPMV_OK) st = dalloc(&keys, (size_t)m, s);
                if (st == SSPMV_OK) st = dalloc(&vals, (size_t)m, s);
                if (st == SSPMV_OK) {
                    sell_sort_keys<<<g, 256, 0, cu(s)>>>(m, sigma, maxlen, A->row_offset, keys, vals);
                    note_launch();
                    const uint64_t nslices = (uint64_t)((m + sigma - 1) / sigma);
                    const uint64_t maxkey = (nslices - 1) * (uint64_t)(maxlen + 1) + (uint64_t)maxlen;
                    st = radix_sort_pairs(keys, vals, m, bits_for(maxkey), s);
                }
                if (st == SSPMV_OK) {
                    copy_u32_to_i32<<<g, 256, 0, cu(s)>>>(m, vals, b.reorder);
                    note_launch();
                }
                dfree(keys, s);
                dfree(vals, s);
            }
        }
        if (st != SSPMV_OK) { b.release(s); return st; }
    }
    st = dalloc(&b.width, (size_t)b.nchunks, s);
    if (st == SSPMV_OK) st = dalloc(&b.chunk_ptr, (size_t)b.nchunks + 1, s);
    if (st == SSPMV_OK && b.nchunks > 0) {
        cudaError_t e = cudaMemsetAsync(b.width, 0, (size_t)b.nchunks * 4, cu(s));
        if (e != cudaSuccess) st = fail(SSPMV_CUDA_ERROR, "width memset: %s", cudaGetErrorString(e));
        if (st == SSPMV_OK && m > 0) {
            chunk_row_max<<<grid_for(m, 256, (int64_t)num_sms() * 16), 256, 0, cu(s)>>>(m, C, A->row_offset,
                                                                                      b.reorder, b.width);
            note_launch();
        }
        if (st == SSPMV_OK) {
            chunk_widths<<<grid_for(b.nchunks, 256, (int64_t)num_sms() * 16), 256, 0, cu(s)>>>(b.nchunks, C, align,
                                                                                             b.width, b.chunk_ptr);
            note_launch();
            st = exclusive_scan_i64(b.chunk_ptr, b.chunk_ptr, b.nchunks, &b.total, s);
        }
    }
    if (st == SSPMV_OK) {
        cudaError_t e = cudaMemcpyAsync(b.chunk_ptr + b.nchunks, &b.total, 8, cudaMemcpyHostToDevice, cu(s));
        if (e != cudaSuccess) st = fail(SSPMV_CUDA_ERROR, "chunk_ptr: %s", cudaGetErrorString(e));
    }
    if (st == SSPMV_OK) st = dalloc(&b.col, (size_t)b.total, s);
    if (st == SSPMV_OK) st = dalloc((unsigned char **)&b.val, (size_t)b.total * vsize(vt), s);
    const bool by_slot = C <= kFillChunk;
    if (st == SSPMV_OK && b.total > 0 && !by_slot) {
        cudaError_t e = cudaMemsetAsync(b.col, 0xff, (size_t)b.total * 4, cu(s));
        if (e == cudaSuccess) e = cudaMemsetAsync(b.val, 0, (size_t)b.total * vsize(vt), cu(s));
        if (e != cudaSuccess) st = fail(SSPMV_CUDA_ERROR, "memset: %s", cudaGetErrorString(e));
    }
    if (st == SSPMV_OK && b.total > 0) {
        st = dispatch_value(vt, [&](auto tag) -> sspmv_status {
            using V = decltype(tag);
            if (by_slot)
                sliced_fill_slots<V><<<grid_for(b.total, kFillTile), 256, 0, cu(s)>>>(
                    m, C, b.nchunks, b.total, b.chunk_ptr, b.reorder, A->row_offset, A->col_index,
                    (const V *)A->values, b.col, (V *)b.val);
            else
                sliced_fill<V><<<g, 256, 0, cu(s)>>>(m, C, b.chunk_ptr, b.reorder, A->row_offset, A->col_index,
                                                     (const V *)A->values, b.col, (V *)b.val);
            SSPMV_LAUNCH_CHECK();
            return SSPMV_OK;
        });
    }
    if (st == SSPMV_OK) {
        cudaError_t e = cudaStreamSynchronize(cu(s));
        if (e != cudaSuccess) st = fail(SSPMV_CUDA_ERROR, "convert: %s", cudaGetErrorString(e));
    }
    if (st != SSPMV_OK) b.release(s);
    return st;
}

sspmv_status check_csr(const sspmv_csr *A) {
    if (!A) return fail(SSPMV_INVALID_ARG, "null csr");
    return check_dims(A->f.value_type, A->f.num_rows, A->f.num_cols, A->f.num_nnzs);
}

// Host copy of a slot-major slab, reordered to the reference's row-major chunks.
sspmv_status export_slab(const int64_t *d_chunk_ptr, int64_t nchunks, int32_t C, int64_t total, const int32_t *d_col,
                         const void *d_val, size_t sv, int32_t *col_out, void *val_out, sspmv_stream_t s) {
    std::vector<int64_t> cp((size_t)nchunks + 1);
    std::vector<int32_t> col((size_t)std::max<int64_t>(total, 1));
    std::vector<unsigned char> val((size_t)std::max<int64_t>(total, 1) * sv);
    SSPMV_CUDA_TRY(cudaMemcpyAsync(cp.data(), d_chunk_ptr, (size_t)(nchunks + 1) * 8, cudaMemcpyDeviceToHost, cu(s)));
    if (total > 0) {
        SSPMV_CUDA_TRY(cudaMemcpyAsync(col.data(), d_col, (size_t)total * 4, cudaMemcpyDeviceToHost, cu(s)));
        SSPMV_CUDA_TRY(cudaMemcpyAsync(val.data(), d_val, (size_t)total * sv, cudaMemcpyDeviceToHost, cu(s)));
    }
    SSPMV_CUDA_TRY(cudaStreamSynchronize(cu(s)));
    for (int64_t c = 0; c < nchunks; c++) {
        const int64_t base = cp[(size_t)c], w = (cp[(size_t)c + 1] - base) / C;
        for (int32_t r = 0; r < C; r++)
            for (int64_t k = 0; k < w; k++) {
                const int64_t src = base + k * C + r, dst = base + (int64_t)r * w + k;
                if (col_out) col_out[dst] = col[(size_t)src];
                if (val_out) std::memcpy((unsigned char *)val_out + dst * sv, val.data() + src * sv, sv);
            }
    }
    return SSPMV_OK;
}

sspmv_status d2h(void *dst, const void *src, size_t bytes, sspmv_stream_t s) {
    if (!dst || bytes == 0) return SSPMV_OK;
    SSPMV_CUDA_TRY(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, cu(s)));
    SSPMV_CUDA_TRY(cudaStreamSynchronize(cu(s)));
    return SSPMV_OK;
}

double sliced_bytes(const sspmv_features *f, int64_t nchunks, bool reorder, int32_t k, int32_t beta_nonzero) {
    const double sv = (double)vsize(f->value_type);
    return (double)f->num_nnzs * (sv + 4.0) + (double)(nchunks + 1) * 8.0 +
           (reorder ? (double)f->num_rows * 4.0 : 0.0) + (double)k * (double)f->num_cols * sv +
           (double)k * (double)f->num_rows * sv * (beta_nonzero ? 2.0 : 1.0);
}

}  // namespace

// =================================================================== ELL ===
// coo_to_ell (include/sparse_conversion.h:94-142): row counts, then each row's
// entries in COO order.  The same slab as csr_to_ell on the COO's stable
// row sort (coo_to_csr keeps each row's entries in COO order), so that is how
// it is built.  Like the reference it ignores ld (it always sets RowMajor).
extern "C" sspmv_status sspmv_coo_to_ell(const sspmv_coo *coo, int32_t ld, sspmv_ell *out, sspmv_stream_t s) {
    if (!coo || !out) return fail(SSPMV_INVALID_ARG, "null argument");
    (void)ld;
    sspmv_csr csr;
    SSPMV_TRY(sspmv_coo_to_csr(coo, &csr, s));
    const sspmv_status st = sspmv_csr_to_ell(&csr, SSPMV_ROW_MAJOR, out, s);
    sspmv_delete_csr(&csr);
    return st;
}

extern "C" sspmv_status sspmv_csr_to_ell(const sspmv_csr *csr, int32_t ld, sspmv_ell *out, sspmv_stream_t s) {
    SSPMV_TRY(check_csr(csr));
    if (!out) return fail(SSPMV_INVALID_ARG, "null output");
    if (ld != SSPMV_ROW_MAJOR && ld != SSPMV_COL_MAJOR) return fail(SSPMV_INVALID_ARG, "ld must be 0 or 1");
    const int64_t m = csr->f.num_rows;
    int32_t width = 0;
    SSPMV_TRY(max_row_length(csr->row_offset, m, &width, s));
    if ((double)m * (double)width > 4.0e9)
        return fail(SSPMV_INFEASIBLE, "ELL needs %lld x %d slots", (long long)m, width);
    // ELL == one chunk of C = m rows, alignment 1.
    SlicedBuild b;
    SSPMV_TRY(build_sliced(csr, (int32_t)std::max<int64_t>(m, 1), 1, 0, b, s));
    sspmv_ell A;
    init_features(&A.f, csr->f.value_type, m, csr->f.num_cols, csr->f.num_nnzs, 1);
    A.ld = ld;
    A.max_row_width = width;
    A.min_row_width = 0;
    A.col_index = b.col;
    A.values = b.val;
    Plan *p = get_plan(&A.f);
    p->extra[0] = b.chunk_ptr;  // {0, m*width}
    dfree(b.width, s);
    *out = A;
    return SSPMV_OK;
}

extern "C" sspmv_status sspmv_spmm_ell(double alpha, const sspmv_ell *A, int32_t k, const void *X, int64_t ldx,
                                       double beta, void *Y, int64_t ldy, sspmv_stream_t s) {
    if (!A) return fail(SSPMV_INVALID_ARG, "null matrix");
    Plan *p = get_plan(&A->f);
    SlicedView v{A->f.num_rows, (int32_t)std::max<int64_t>(A->f.num_rows, 1), (const int64_t *)p->extra[0], nullptr,
                 A->col_index, A->values, 0, A->max_row_width, A->f.num_cols, 1, false};
    return spmm_sliced(&A->f, v, alpha, k, X, ldx, beta, Y, ldy, s);
}

extern "C" sspmv_status sspmv_LeSpMV_ell(double alpha, const sspmv_ell *A, const void *x, double beta, void *y,
                                         sspmv_stream_t s) {
    return sspmv_spmm_ell(alpha, A, 1, x, 1, beta, y, 1, s);
}

extern "C" sspmv_status sspmv_ell_export(const sspmv_ell *A, int32_t *col_index, void *values, sspmv_stream_t s) {
    if (!A) return fail(SSPMV_INVALID_ARG, "null matrix");
    const int64_t m = A->f.num_rows, w = A->max_row_width, tot = m * w;
    const size_t sv = vsize(A->f.value_type);
    if (A->ld == SSPMV_COL_MAJOR) {
        SSPMV_TRY(d2h(col_index, A->col_index, (size_t)tot * 4, s));
        SSPMV_TRY(d2h(values, A->values, (size_t)tot * sv, s));
        return SSPMV_OK;
    }
    std::vector<int32_t> col((size_t)std::max<int64_t>(tot, 1));
    std::vector<unsigned char> val((size_t)std::max<int64_t>(tot, 1) * sv);
    SSPMV_TRY(d2h(col.data(), A->col_index, (size_t)tot * 4, s));
    SSPMV_TRY(d2h(val.data(), A->values, (size_t)tot * sv, s));
    for (int64_t i = 0; i < m; i++)
        for (int64_t k = 0; k < w; k++) {
            if (col_index) col_index[i * w + k] = col[(size_t)(k * m + i)];
            if (values) std::memcpy((unsigned char *)values + (i * w + k) * sv, val.data() + (k * m + i) * sv, sv);
        }
    return SSPMV_OK;
}

extern "C" sspmv_status sspmv_delete_ell(sspmv_ell *A) {
    if (!A) return SSPMV_OK;
    const DeleteScope scope;
    free_plan(&A->f, nullptr);
    if (A->f.owns) {
        dfree(A->col_index, nullptr);
        dfree(A->values, nullptr);
    }
    A->col_index = nullptr;
    A->values = nullptr;
    return SSPMV_OK;
}

extern "C" double sspmv_algorithmic_bytes_ell(const sspmv_ell *A, int32_t k, int32_t beta_nonzero) {
    return sliced_bytes(&A->f, 0, false, k, beta_nonzero) - 8.0;
}

// ================================================================= S-ELL ===
extern "C" sspmv_status sspmv_csr_to_sell(const sspmv_csr *csr, int32_t C, int32_t align, sspmv_s_ell *out,
                                          sspmv_stream_t s) {
    SSPMV_TRY(check_csr(csr));
    if (!out) return fail(SSPMV_INVALID_ARG, "null output");
    if (C == 0) C = 4;
    if (align == 0) align = default_alignment(csr->f.value_type);
    if (C < 1 || align < 1) return fail(SSPMV_INVALID_ARG, "chunkwidth and alignment must be >= 1");
    SlicedBuild b;
    SSPMV_TRY(build_sliced(csr, C, align, 0, b, s));
    sspmv_s_ell A;
    init_features(&A.f, csr->f.value_type, csr->f.num_rows, csr->f.num_cols, csr->f.num_nnzs, 1);
    A.sliceWidth = C;
    A.chunk_num = (int32_t)b.nchunks;
    A.alignment = align;
    A.row_width = b.width;
    A.chunk_ptr = b.chunk_ptr;
    A.total_slots = b.total;
    A.col_index = b.col;
    A.values = b.val;
    *out = A;
    return SSPMV_OK;
}

extern "C" sspmv_status sspmv_spmm_sell(double alpha, const sspmv_s_ell *A, int32_t k, const void *X, int64_t ldx,
                                        double beta, void *Y, int64_t ldy, sspmv_stream_t s) {
    if (!A) return fail(SSPMV_INVALID_ARG, "null matrix");
    SlicedView v{A->f.num_rows, A->sliceWidth,   A->chunk_ptr,   nullptr,
                 A->col_index,  A->values,     A->chunk_num, 0, A->f.num_cols, A->alignment, false};
    return spmm_sliced(&A->f, v, alpha, k, X, ldx, beta, Y, ldy, s);
}

extern "C" sspmv_status sspmv_LeSpMV_sell(double alpha, const sspmv_s_ell *A, const void *x, double beta, void *y,
                                          sspmv_stream_t s) {
    return sspmv_spmm_sell(alpha, A, 1, x, 1, beta, y, 1, s);
}

extern "C" sspmv_status sspmv_sell_export(const sspmv_s_ell *A, int32_t *row_width, int32_t *col_index,
                                          void *values, sspmv_stream_t s) {
    if (!A) return fail(SSPMV_INVALID_ARG, "null matrix");
    SSPMV_TRY(d2h(row_width, A->row_width, (size_t)A->chunk_num * 4, s));
    return export_slab(A->chunk_ptr, A->chunk_num, A->sliceWidth, A->total_slots, A->col_index, A->values,
                       vsize(A->f.value_type), col_index, values, s);
}

extern "C" sspmv_status sspmv_delete_sell(sspmv_s_ell *A) {
    if (!A) return SSPMV_OK;
    const DeleteScope scope;
    free_plan(&A->f, nullptr);
    if (A->f.owns) {
        dfree(A->row_width, nullptr);
        dfree(A->chunk_ptr, nullptr);
        dfree(A->col_index, nullptr);
        dfree(A->values, nullptr);
    }
    A->row_width = nullptr;
    A->chunk_ptr = nullptr;
    A->col_index = nullptr;
    A->values = nullptr;
    return SSPMV_OK;
}

extern "C" double sspmv_algorithmic_bytes_sell(const sspmv_s_ell *A, int32_t k, int32_t beta_nonzero) {
    return sliced_bytes(&A->f, A->chunk_num, false, k, beta_nonzero);
}

// ========================================================== SELL-c-sigma ===
extern "C" sspmv_status sspmv_csr_to_sell_c_sigma(const sspmv_csr *csr, int32_t sigma, int32_t C, int32_t align,
                                                  sspmv_sell_c_sigma *out, sspmv_stream_t s) {
    SSPMV_TRY(check_csr(csr));
    if (!out) return fail(SSPMV_INVALID_ARG, "null output");
    if (sigma == 0) sigma = 16384;
    if (C == 0) C = 4;
    if (align == 0) align = default_alignment(csr->f.value_type);
    if (C < 1 || align < 1 || sigma < 1) return fail(SSPMV_INVALID_ARG, "sigma, C and alignment must be >= 1");
    if (sigma % C) return fail(SSPMV_INVALID_ARG, "sigma (%d) must be a multiple of C (%d)", sigma, C);
    SlicedBuild b;
    SSPMV_TRY(build_sliced(csr, C, align, sigma, b, s));
    const int64_t m = csr->f.num_rows;
    sspmv_sell_c_sigma A;
    init_features(&A.f, csr->f.value_type, m, csr->f.num_cols, csr->f.num_nnzs, 1);
    A.sliceWidth_Sigma = sigma;
    A.chunkWidth_C = C;
    A.sliceNum = (int32_t)((m + sigma - 1) / sigma);
    A.chunk_num_per_slice = sigma / C;
    A.chunkNum = A.sliceNum * A.chunk_num_per_slice;
    A.validchunkNum = (int32_t)b.nchunks;
    A.alignment = align;
    A.reorder = b.reorder;
    A.chunk_len = b.width;
    A.chunk_ptr = b.chunk_ptr;
    A.total_slots = b.total;
    A.col_index = b.col;
    A.values = b.val;
    *out = A;
    return SSPMV_OK;
}

extern "C" sspmv_status sspmv_spmm_sell_c_sigma(double alpha, const sspmv_sell_c_sigma *A, int32_t k, const void *X,
                                                int64_t ldx, double beta, void *Y, int64_t ldy, sspmv_stream_t s) {
    if (!A) return fail(SSPMV_INVALID_ARG, "null matrix");
    SlicedView v{A->f.num_rows, A->chunkWidth_C,   A->chunk_ptr,   A->reorder,
                 A->col_index,  A->values,         A->validchunkNum, 0, A->f.num_cols, A->alignment, A->sliceWidth_Sigma >= A->f.num_rows};
    return spmm_sliced(&A->f, v, alpha, k, X, ldx, beta, Y, ldy, s);
}

extern "C" sspmv_status sspmv_LeSpMV_sell_c_sigma(double alpha, const sspmv_sell_c_sigma *A, const void *x,
                                                  double beta, void *y, sspmv_stream_t s) {
    return sspmv_spmm_sell_c_sigma(alpha, A, 1, x, 1, beta, y, 1, s);
}

extern "C" sspmv_status sspmv_sell_c_sigma_export(const sspmv_sell_c_sigma *A, int32_t *reorder, int32_t *chunk_len,
                                                  int32_t *col_index, void *values, sspmv_stream_t s) {
    if (!A) return fail(SSPMV_INVALID_ARG, "null matrix");
    SSPMV_TRY(d2h(reorder, A->reorder, (size_t)A->f.num_rows * 4, s));
    SSPMV_TRY(d2h(chunk_len, A->chunk_len, (size_t)A->validchunkNum * 4, s));
    return export_slab(A->chunk_ptr, A->validchunkNum, A->chunkWidth_C, A->total_slots, A->col_index, A->values,
                       vsize(A->f.value_type), col_index, values, s);
}

extern "C" sspmv_status sspmv_delete_sell_c_sigma(sspmv_sell_c_sigma *A) {
    if (!A) return SSPMV_OK;
    const DeleteScope scope;
    free_plan(&A->f, nullptr);
    if (A->f.owns) {
        dfree(A->reorder, nullptr);
        dfree(A->chunk_len, nullptr);
        dfree(A->chunk_ptr, nullptr);
        dfree(A->col_index, nullptr);
        dfree(A->values, nullptr);
    }
    A->reorder = A->chunk_len = A->col_index = nullptr;
    A->chunk_ptr = nullptr;
    A->values = nullptr;
    return SSPMV_OK;
}

extern "C" double sspmv_algorithmic_bytes_sell_c_sigma(const sspmv_sell_c_sigma *A, int32_t k, int32_t beta_nonzero) {
    return sliced_bytes(&A->f, A->validchunkNum, true, k, beta_nonzero);
}

// ============================================================== SELL-c-R ===
extern "C" sspmv_status sspmv_csr_to_sell_c_R(const sspmv_csr *csr, int32_t C, int32_t align, sspmv_sell_c_R *out,
                                              sspmv_stream_t s) {
    SSPMV_TRY(check_csr(csr));
    if (!out) return fail(SSPMV_INVALID_ARG, "null output");
    if (C == 0) C = 4;
    if (align == 0) align = default_alignment(csr->f.value_type);
    if (C < 1 || align < 1) return fail(SSPMV_INVALID_ARG, "C and alignment must be >= 1");
    const int64_t m = csr->f.num_rows;
    SlicedBuild b;
    SSPMV_TRY(build_sliced(csr, C, align, std::max<int64_t>(m, 1), b, s));
    sspmv_sell_c_R A;
    init_features(&A.f, csr->f.value_type, m, csr->f.num_cols, csr->f.num_nnzs, 1);
    A.chunkWidth_C = C;
    A.validchunkNum = (int32_t)b.nchunks;
    A.alignment = align;
    A.reorder = b.reorder;
    A.chunk_len = b.width;
    A.chunk_ptr = b.chunk_ptr;
    A.total_slots = b.total;
    A.col_index = b.col;
    A.values = b.val;
    *out = A;
    return SSPMV_OK;
}

extern "C" sspmv_status sspmv_spmm_sell_c_R(double alpha, const sspmv_sell_c_R *A, int32_t k, const void *X,
                                            int64_t ldx, double beta, void *Y, int64_t ldy, sspmv_stream_t s) {
    if (!A) return fail(SSPMV_INVALID_ARG, "null matrix");
    SlicedView v{A->f.num_rows, A->chunkWidth_C,   A->chunk_ptr,   A->reorder,
                 A->col_index,  A->values,         A->validchunkNum, 0, A->f.num_cols, A->alignment, true};
    return spmm_sliced(&A->f, v, alpha, k, X, ldx, beta, Y, ldy, s);
}

extern "C" sspmv_status sspmv_LeSpMV_sell_c_R(double alpha, const sspmv_sell_c_R *A, const void *x, double beta,
                                              void *y, sspmv_stream_t s) {
    return sspmv_spmm_sell_c_R(alpha, A, 1, x, 1, beta, y, 1, s);
}

extern "C" sspmv_status sspmv_sell_c_R_export(const sspmv_sell_c_R *A, int32_t *reorder, int32_t *chunk_len,
                                              int32_t *col_index, void *values, sspmv_stream_t s) {
    if (!A) return fail(SSPMV_INVALID_ARG, "null matrix");
    SSPMV_TRY(d2h(reorder, A->reorder, (size_t)A->f.num_rows * 4, s));
    SSPMV_TRY(d2h(chunk_len, A->chunk_len, (size_t)A->validchunkNum * 4, s));
    return export_slab(A->chunk_ptr, A->validchunkNum, A->chunkWidth_C, A->total_slots, A->col_index, A->values,
                       vsize(A->f.value_type), col_index, values, s);
}

extern "C" sspmv_status sspmv_delete_sell_c_R(sspmv_sell_c_R *A) {
    if (!A) return SSPMV_OK;
    const DeleteScope scope;
    free_plan(&A->f, nullptr);
    if (A->f.owns) {
        dfree(A->reorder, nullptr);
        dfree(A->chunk_len, nullptr);
        dfree(A->chunk_ptr, nullptr);
        dfree(A->col_index, nullptr);
        dfree(A->values, nullptr);
    }
    A->reorder = A->chunk_len = A->col_index = nullptr;
    A->chunk_ptr = nullptr;
    A->values = nullptr;
    return SSPMV_OK;
}

extern "C" double sspmv_algorithmic_bytes_sell_c_R(const sspmv_sell_c_R *A, int32_t k, int32_t beta_nonzero) {
    return sliced_bytes(&A->f, A->validchunkNum, true, k, beta_nonzero);
}
