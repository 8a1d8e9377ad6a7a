// bsr.cu -- BSR format on sm_103a: GPU converter, SpMV / SpMM, export.
//
// Converter (csr_to_bsr, include/sparse_conversion.h:769-926): the distinct
// (block row, block column) pairs of the nonzeros, block columns ascending in
// each block row, blocks stored row-major (r x c) and zero filled.  On the GPU
// every nonzero contributes the key block_row*nb + block_col, the keys are
// radix sorted and made unique, and values are written row by row in CSR
// order (a duplicated (row, col) keeps its last value, as the reference's
// overwrite).  r = c = 1 copies the CSR arrays, as the reference does.
//
// SpMV (LeSpMV_bsr, src/spmv_bsr.cpp:215-233): the block-stream kernel (below)
// for SpMV with r a power of two <= 32 and c <= 16 a power of two; otherwise,
// for SpMM and for kernel_flag 1, one thread per matrix row.  There the r
// threads of a block row read the r consecutive c-wide rows of each block,
// so a block (r*c values) is one contiguous read; x[bc*c .. bc*c+c) is one
// c-wide read shared by the r threads.  Columns past num_cols (the ragged
// last block column) are skipped.
#include <algorithm>
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
constexpr int kStreamBlock = 64;

__global__ void bsr_keys(int64_t m, int32_t r, int32_t c, int64_t nb, const int32_t *__restrict__ rp,
                         const int32_t *__restrict__ ci, uint64_t *__restrict__ keys, uint32_t *__restrict__ vals) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
        const uint64_t br = (uint64_t)div_nonneg(i, r);
        for (int32_t jj = rp[i]; jj < rp[i + 1]; jj++) {
            keys[jj] = br * (uint64_t)nb + (uint64_t)(ci[jj] / c);
            vals[jj] = (uint32_t)jj;
        }
    }
}

__global__ void unique_flags(int64_t n, const uint64_t *__restrict__ keys, int32_t *__restrict__ flags) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        flags[i] = (i == 0 || keys[i] != keys[i - 1]) ? 1 : 0;
}

__global__ void unique_scatter(int64_t n, const uint64_t *__restrict__ keys, const int32_t *__restrict__ pos,
                               int64_t nb, uint64_t *__restrict__ ukeys, int32_t *__restrict__ bcol) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        if (i == 0 || keys[i] != keys[i - 1]) {
            ukeys[pos[i]] = keys[i];
            bcol[pos[i]] = (int32_t)(keys[i] % (uint64_t)nb);
        }
}

// row_ptr[b] = first unique block with block row >= b
__global__ void bsr_row_ptr(int64_t mb, int64_t nb, int64_t nnzb, const uint64_t *__restrict__ ukeys,
                            int32_t *__restrict__ row_ptr) {
    for (int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; b <= mb; b += (int64_t)gridDim.x * blockDim.x) {
        const uint64_t key = (uint64_t)b * (uint64_t)nb;
        int64_t lo = 0, hi = nnzb;
        while (lo < hi) {
            int64_t mid = (lo + hi) >> 1;
            if (ukeys[mid] < key) lo = mid + 1;
            else hi = mid;
        }
        row_ptr[b] = (int32_t)lo;
    }
}

template <typename V>
__global__ void bsr_fill(int64_t m, int32_t r, int32_t c, const int32_t *__restrict__ rp, const int32_t *__restrict__ ci,
                         const V *__restrict__ cv, const int32_t *__restrict__ row_ptr, const int32_t *__restrict__ bcol,
                         V *__restrict__ data) {
    const int64_t rc = (int64_t)r * c;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t br = div_nonneg(i, r), q = i - br * r;
        const int32_t b0 = row_ptr[br], b1 = row_ptr[br + 1];
        for (int32_t jj = rp[i]; jj < rp[i + 1]; jj++) {
            const int32_t col = ci[jj], bc = col / c;
            int32_t lo = b0, hi = b1;
            while (lo < hi) {
                int32_t mid = (lo + hi) >> 1;
                if (bcol[mid] < bc) lo = mid + 1;
                else hi = mid;
            }
            data[(int64_t)lo * rc + q * c + (col - bc * c)] = cv[jj];
        }
    }
}

template <typename V, int K, int CB, bool PLAIN = false>
__global__ void __launch_bounds__(kBlock) bsr_spmv_kernel(int m, int n, int r, int cr,
                                                        const int32_t *__restrict__ row_ptr,
                                                        const int32_t *__restrict__ bcol, const V *__restrict__ data,
                                                        const V *__restrict__ x, int64_t ldx, int xvec, V alpha,
                                                        V beta, V *__restrict__ y, int64_t ldy) {
    const int c = CB > 0 ? CB : cr;
    const int64_t rc = (int64_t)r * c;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t br = div_nonneg(i, r), q = i - br * r;
        const int32_t k0 = ld_stream(row_ptr + br), k1 = ld_stream(row_ptr + br + 1);
        V s[K];
#pragma unroll
        for (int t = 0; t < K; t++) s[t] = V(0);
        for (int32_t k = k0; k < k1; k++) {
            const int64_t x0 = (int64_t)ld_x(bcol + k) * c;
            const V *blk = data + k * rc + q * c;
            if (CB > 0 && x0 + c <= n) {
                V a[CB > 0 ? CB : 1];
#pragma unroll
                for (int e = 0; e < (CB > 0 ? CB : 1); e++) a[e] = ld_stream(blk + e);
#pragma unroll
                for (int e = 0; e < (CB > 0 ? CB : 1); e++) {
                    V xr[K];
                    ld_xrow<V, K>(x, x0 + e, ldx, xvec != 0, xr);
#pragma unroll
                    for (int t = 0; t < K; t++) s[t] += a[e] * xr[t];
                }
            } else {
                for (int e = 0; e < c; e++) {
                    if (x0 + e >= n) break;
                    const V a = ld_stream(blk + e);
                    V xr[K];
                    ld_xrow<V, K>(x, x0 + e, ldx, xvec != 0, xr);
#pragma unroll
                    for (int t = 0; t < K; t++) s[t] += a * xr[t];
                }
            }
        }
        V *yp = y + i * ldy;
#pragma unroll
        for (int t = 0; t < K; t++) yp[t] = row_out(PLAIN, alpha, s[t], beta, yp + t);
    }
}

// ------------------------------------------------------- block stream --
// The thread-per-row kernel above leaves lanes idle wherever the block rows of
// a warp hold different numbers of blocks, and GB300's narrow FP64 pipe is
// paid per warp instruction, however few lanes are active (profiled on 4x4
// FP64 blocks, about one block per block row: the pipe 75-84% busy with a
// third of its lanes doing FMAs).  This kernel streams blocks instead, as the
// stream kernel (csr_stream.cu) streams nonzeros, on the same plan made of the
// block rows: r lanes (lane q of the group takes row q of a block) walk B
// consecutive blocks with all their loads in flight -- 16 bytes of a block's
// row and of x at a time -- and restart at block row ends; the groups' open
// sums are joined by one segmented scan per step of B * 32 / r blocks.  A warp
// finishes the block rows that start in its window, so one launch and no
// pieces; r must be a power of two <= 32.  With one block per group and step,
// a scan for each, block_row read per block and values one at a time: 2M rows
// of 4x4 blocks FP32 22.5 us, now 17.1 (FP64 50.8, now 34.7).  It moves 3.2
// TB/s there: a chain of two dependent loads (the block's column, then x) at 32
// warps a SM.  The next step's columns and blocks loaded before this step's
// sums measured 19.6 us (more registers, fewer warps).
// SMALL: a matrix that leaves most warps idle takes one block a group, half a step
// of them a window: more warps and the shortest chain, which is its time (4,000
// rows, 2x2 FP64, 5.6 us with four blocks a group, 2.7 so).
template <typename V, int C, bool SMALL = false>
struct BsrShape {
    static constexpr int kWords = (int)(C * sizeof(V) / 4);             // 4-byte words of a block's row
    static constexpr int B = SMALL || kWords >= 16 ? 1 : kWords <= 4 ? 4 : 16 / kWords;  // up to 16 words a lane in flight
};

// Resident CTAs per SM the register budget is set for: 2M rows of 4x4 blocks,
// FP32 at 14 / 16 / 20 CTAs 19.6 / 19.2 / 20.1 us, FP64 at 16 / 20 43.8 /
// 40.0 us; 1M rows of 8x8 FP64 at 16 / 20 (which spills) 54.9 / 57.9 us.
template <typename V, int C>
constexpr int bsr_ctas() {
    return BsrShape<V, C>::kWords > 16 ? 8 : sizeof(V) == 8 && C == 4 ? 20 : 16;
}

// C values at p: vector loads when `vec` (p aligned to min(16, C values)).
template <typename V, int C, bool STREAM>
__device__ __forceinline__ void ld_run(const V *__restrict__ p, bool vec, V (&out)[C]) {
    constexpr int kBytes = (int)(C * sizeof(V));
    if constexpr (kBytes >= 16) {
        if (vec) {
#pragma unroll
            for (int h = 0; h < kBytes / 16; h++) {
                const float4 *src = reinterpret_cast<const float4 *>(p) + h;
                const float4 t = STREAM ? __ldcs(src) : __ldg(src);
                if constexpr (sizeof(V) == 4) {
                    out[4 * h] = t.x; out[4 * h + 1] = t.y; out[4 * h + 2] = t.z; out[4 * h + 3] = t.w;
                } else {
                    out[2 * h] = __hiloint2double(__float_as_int(t.y), __float_as_int(t.x));
                    out[2 * h + 1] = __hiloint2double(__float_as_int(t.w), __float_as_int(t.z));
                }
            }
            return;
        }
    } else if constexpr (kBytes == 8 && sizeof(V) == 4) {
        if (vec) {
            const float2 *src = reinterpret_cast<const float2 *>(p);
            const float2 t = STREAM ? __ldcs(src) : __ldg(src);
            out[0] = t.x;
            out[1] = t.y;
            return;
        }
    }
#pragma unroll
    for (int e = 0; e < C; e++) out[e] = STREAM ? ld_stream(p + e) : ld_x(p + e);
}

template <typename V, int C, bool PLAIN, bool SMALL>
__global__ void __launch_bounds__(kStreamBlock, (bsr_ctas<V, C>())) bsr_stream_kernel(
    const StreamView A, int m, int n, int lr, const V *__restrict__ data, int dvec, const V *__restrict__ x, int xvec, V alpha,
    V beta, V *__restrict__ y) {
    constexpr unsigned kFull = 0xffffffffu;
    constexpr int B = BsrShape<V, C, SMALL>::B;
    constexpr bool kSeed = sizeof(V) == 8;
    const int64_t w = (int64_t)blockIdx.x * (kStreamBlock / 32) + (threadIdx.x >> 5);
    const int r = 1 << lr, NG = 32 >> lr;
    const int lane = threadIdx.x & 31, g = lane >> lr, q = lane & (r - 1);
    if (w >= A.windows) {  // warp-uniform: block rows without blocks, y = beta * y, 256 rows a warp
        const int64_t t0 = (w - A.windows) * kEmptyUnit + lane;
        int64_t i[8];
        V old[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int64_t t = t0 + 32 * u;
            i[u] = (t >> lr) < A.nempty ? ((int64_t)__ldg(A.empty + (t >> lr)) << lr) + (t & (r - 1)) : m;
        }
#pragma unroll
        for (int u = 0; u < 8; u++) old[u] = !PLAIN && beta != V(0) && i[u] < m ? y[i[u]] : V(0);
#pragma unroll
        for (int u = 0; u < 8; u++)
            if (i[u] < m) y[i[u]] = PLAIN || beta == V(0) ? V(0) : beta * old[u];
        return;
    }
    const int64_t rc = (int64_t)r * C;
    const int4 rec = __ldg(A.rec + w);
    const uint32_t eA = (uint32_t)rec.x, eB = (uint32_t)rec.y;
    int row = rec.z;
    auto put = [&](int ordinal, V sum) {
        const int64_t i = ((int64_t)(A.nzrow ? __ldg(A.nzrow + ordinal) : ordinal) << lr) + q;
        if (i < m) y[i] = row_out(PLAIN, alpha, sum, beta, y + i);
    };
    V carry = V(0);  // the open block row's sum over the earlier steps
    const unsigned before = g == 0 ? 0u : 0xffffffffu >> (32 - (g << lr));  // lanes of the groups before this one
    for (uint32_t b = eA & ~(uint32_t)(B - 1); b < eB && eA < eB; b += B * NG) {  // warp-uniform
        const uint32_t e0 = b + (uint32_t)(B * g);
        // which of the B blocks belong to the window, and which end a block row
        unsigned in = 0;
#pragma unroll
        for (int u = 0; u < B; u++) in |= (e0 + u >= eA && e0 + u < eB ? 1u : 0u) << u;
        const unsigned eb = in ? (__ldg(A.ends + (e0 >> 3)) >> (e0 & 7)) & in : 0u;
        int bc[B];
        V a[B][C], xv[B][C];
#pragma unroll
        for (int u = 0; u < B; u++) bc[u] = (in >> u) & 1u ? ld_stream(A.col + e0 + u) : 0;
#pragma unroll
        for (int u = 0; u < B; u++) {
            if ((in >> u) & 1u) {
                ld_run<V, C, true>(data + (int64_t)(e0 + u) * rc + q * C, dvec != 0, a[u]);
            } else {
#pragma unroll
                for (int e = 0; e < C; e++) a[u][e] = V(0);
            }
        }
#pragma unroll
        for (int u = 0; u < B; u++) {
            const int64_t x0 = (int64_t)bc[u] * C;
            if (((in >> u) & 1u) && x0 + C <= n) {
                ld_run<V, C, false>(x + x0, xvec != 0, xv[u]);
            } else {  // the ragged last block column: its fill is no part of the product
#pragma unroll
                for (int e = 0; e < C; e++) {
                    const bool ok = ((in >> u) & 1u) && x0 + e < n;
                    xv[u][e] = ok ? ld_x(x + x0 + e) : V(0);
                    if (!ok) a[u][e] = V(0);
                }
            }
        }
        const int mine = __popc(eb);
        int pos = 0, nend = 0;  // block rows ended in the groups before this one, and in the step
#pragma unroll
        for (int bit = 0; (1 << bit) <= B; bit++) {
            const unsigned f = __ballot_sync(kFull, q == 0 && ((mine >> bit) & 1));
            pos += __popc(f & before) << bit;
            nend += __popc(f) << bit;
        }
        const unsigned flags = __ballot_sync(kFull, mine != 0) & (before | (1u << lane));
        const int dist = flags ? g - ((31 - __clz(flags)) >> lr) : g;
        // FP64 carries the open sum through the FMAs; in FP32 the step's sum and
        // each block's are taken apart, which keeps a long chain's rounding out
        V sum = kSeed && g == 0 ? carry : V(0), head = V(0);
        bool first = true;
        int idx = row + pos;
        auto end_row = [&](V total) {
            if (first) {
                first = false;
                head = total;
            } else {
                put(idx, total);
            }
            idx++;
        };
        if constexpr (kSeed) {
#pragma unroll
            for (int u = 0; u < B; u++) {
#pragma unroll
                for (int e = 0; e < C; e++) sum = fma(a[u][e], xv[u][e], sum);
                if ((eb >> u) & 1u) {
                    end_row(sum);
                    sum = V(0);
                }
            }
        } else {
            V part[B];
#pragma unroll
            for (int u = 0; u < B; u++) {
                part[u] = V(0);
#pragma unroll
                for (int e = 0; e < C; e++) part[u] = fma(a[u][e], xv[u][e], part[u]);
            }
#pragma unroll
            for (int u = 0; u < B; u += 2) {  // by pairs of blocks
                const V next = u + 1 < B ? part[u + 1 < B ? u + 1 : u] : V(0);
                const bool end0 = (eb >> u) & 1u, end1 = u + 1 < B && ((eb >> (u + 1)) & 1u);
                if (end0) end_row(sum + part[u]);
                sum = end0 ? next : sum + (part[u] + next);
                if (end1) {
                    end_row(sum);
                    sum = V(0);
                }
            }
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {  // segmented inclusive scan of the groups' open sums
            if (!__any_sync(kFull, dist >= o)) break;
            const V up = __shfl_up_sync(kFull, sum, o << lr);
            if (dist >= o) sum += up;
        }
        const V cin = __shfl_up_sync(kFull, sum, r);
        if (mine) {
            if (g > 0) head += cin;
            if (!kSeed && pos == 0) head += carry;
            put(row + pos, head);
        }
        const V open = __shfl_sync(kFull, sum, ((NG - 1) << lr) + q);
        carry = kSeed || nend > 0 ? open : carry + open;
        row += nend;
    }
}

// out[0]: lane slots the thread-per-row kernel spends (every warp of 32 rows,
// 32 / r block rows, runs as many block iterations as its longest block row);
// out[1]: block rows without blocks, and tiles[b].x the block's with, for the
// stream plan.
__global__ void __launch_bounds__(kBlock) bsr_row_kernel_slots(int64_t mb, int64_t rows, int lr,
                                                               const int32_t *__restrict__ row_ptr,
                                                               unsigned long long *__restrict__ out,
                                                               int2 *__restrict__ tiles) {
    __shared__ int s_empty[kBlock / 32];
    const int64_t per = 32 >> lr;
    const int64_t w0 = (int64_t)blockIdx.x * rows / per, w1 = min(w0 + rows / per, (mb + per - 1) / per);
    unsigned long long acc = 0;
    int empty = 0;
    for (int64_t w = w0 + threadIdx.x; w < w1; w += kBlock) {
        int32_t mx = 0;
        const int64_t b1 = min(mb, (w + 1) * per);
        for (int64_t b = w * per; b < b1; b++) {
            const int32_t len = row_ptr[b + 1] - row_ptr[b];
            mx = max(mx, len);
            empty += len == 0;
        }
        acc += (unsigned long long)mx * (unsigned long long)per;
    }
    acc = warp_sum(acc);
    empty = warp_sum(empty);
    if ((threadIdx.x & 31) == 0) {
        if (acc) atomicAdd(out, acc);
        s_empty[threadIdx.x >> 5] = empty;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    for (int w = 1; w < kBlock / 32; w++) empty += s_empty[w];
    if (empty) atomicAdd(out + 1, (unsigned long long)empty);
    tiles[blockIdx.x] = make_int2((int)(min(rows, mb - blockIdx.x * rows) - empty), 0);
}

int log2_exact(int64_t v) {
    int l = 0;
    while ((int64_t(1) << l) < v) l++;
    return (int64_t(1) << l) == v ? l : -1;
}

// The block-stream kernel pays a segmented scan per step (about twice the
// FP64 work of a thread whose lanes are all busy); the thread-per-row kernel
// pays for its idle lanes.  The stream kernel is chosen when the thread
// kernel's lane slots exceed the blocks' by this factor.  Thread per row
// against stream, 1M rows: even rows, 4x4 FP64 (banded) 58.7 / 89.0 us;
// uneven rows, 4x4 FP32 (2M) 27.2 / 19.2.
constexpr double kStreamWaste = 2.0;

// extra_i[2], decided once and published in one word: bits 0-1, 1 = block-stream
// kernel, 2 = thread-per-row kernel; above them the block rows without blocks.
// extra[3]: for the block-stream kernel, the tiles' counts until its plan is built.
sspmv_status choose_bsr_kernel(const sspmv_bsr *A, Plan *p, sspmv_stream_t s) {
    if (p->extra_i[2]) return SSPMV_OK;
    std::lock_guard<PlanMutex> guard(plan_mutex());
    if (p->extra_i[2]) return SSPMV_OK;
    const int lr = log2_exact(A->blockDim_r);
    const int64_t rows = stream_tile_rows(A->mb), tiles = (A->mb + rows - 1) / rows;
    unsigned long long *d = nullptr, h[2] = {0, 0};
    SSPMV_TRY(dalloc(&d, 2 + (size_t)tiles, s));  // the sums, then the tiles
    int2 *tile = (int2 *)(d + 2);
    auto body = [&]() -> sspmv_status {
        SSPMV_CUDA_TRY(cudaMemsetAsync(d, 0, sizeof(h), cu(s)));
        bsr_row_kernel_slots<<<(unsigned)tiles, kBlock, 0, cu(s)>>>(A->mb, rows, lr, A->row_ptr, d, tile);
        SSPMV_LAUNCH_CHECK();
        SSPMV_CUDA_TRY(cudaMemcpyAsync(h, d, sizeof(h), cudaMemcpyDeviceToHost, cu(s)));
        SSPMV_CUDA_TRY(cudaStreamSynchronize(cu(s)));
        return SSPMV_OK;
    };
    const sspmv_status st = body();
    const bool stream = st == SSPMV_OK && (double)h[0] > kStreamWaste * (double)A->nnzb;
    if (stream) p->extra[3] = d;
    else dfree(d, s);
    if (st != SSPMV_OK) return st;
    p->extra_i[2] = ((int64_t)h[1] << 2) | (stream ? 1 : 2);
    return SSPMV_OK;
}

template <typename V, int C>
sspmv_status launch_bsr_stream(const sspmv_bsr *A, Plan *p, V alpha, const V *x, V beta, V *y, sspmv_stream_t s) {
    // windows of whole steps less a block row's overhang; never split
    const int lr = log2_exact(A->blockDim_r), groups = 32 >> lr, step = BsrShape<V, C>::B * groups;
    const int64_t mean = A->mb > 0 ? (A->nnzb + A->mb - 1) / A->mb : 1;
    const int slack = (int)std::min<int64_t>(step / 4, mean + 1);
    const int warps = bsr_ctas<V, C>() * (kStreamBlock / 32);
    const int64_t slots = (int64_t)num_sms() * warps;
    // one wave of half steps, of one block a group or of B: a window and what its
    // last block row goes on past it in one step (100k rows, 4x4 FP32, 4.4 us in
    // windows of whole steps, 3.7 so)
    const bool small = A->nnzb <= slots * std::max(1, groups / 2) && step > groups;
    const bool half = !small && A->nnzb <= slots * std::max(1, step / 2);
    const int window = small   ? std::max(1, groups / 2)
                       : half  ? std::max(1, step / 2)
                               : step * window_steps(A->nnzb, step, step - slack, warps) - slack;
    if (!p->stream.window) {
        std::lock_guard<PlanMutex> guard(plan_mutex());
        const unsigned long long *d = (const unsigned long long *)p->extra[3];
        SSPMV_TRY(ensure_stream_plan(p->stream, A->mb, A->nnzb, A->row_ptr, nullptr, A->f.value_type, s,
                                     window, 0x7fffffff, d ? p->extra_i[2] >> 2 : -1,
                                     d ? (const int2 *)(d + 2) : nullptr));
        dfree(p->extra[3], s);
        p->extra[3] = nullptr;
    }
    const StreamView v = stream_view(p->stream, A->nnzb, A->block_colindex, A->block_data);
    const size_t run = std::min<size_t>(16, C * sizeof(V));
    const int xvec = reinterpret_cast<uintptr_t>(x) % run == 0 ? 1 : 0;
    const int dvec = reinterpret_cast<uintptr_t>(A->block_data) % run == 0 ? 1 : 0;
    auto go = [&](auto kernel) {
        kernel<<<grid_for(v.windows + empty_units((int64_t)v.nempty << lr), kStreamBlock / 32), kStreamBlock, 0, cu(s)>>>(
            v, (int)A->f.num_rows, (int)A->f.num_cols, lr, (const V *)A->block_data, dvec, x, xvec, alpha, beta, y);
    };
    const bool plain = alpha == V(1) && beta == V(0);  // y = sum
    if (small && plain) go(bsr_stream_kernel<V, C, true, true>);
    else if (small) go(bsr_stream_kernel<V, C, false, true>);
    else if (plain) go(bsr_stream_kernel<V, C, true, false>);
    else go(bsr_stream_kernel<V, C, false, false>);
    SSPMV_LAUNCH_CHECK();
    return SSPMV_OK;
}

// The block-stream kernel takes SpMV (k = 1, unit strides) for r a power of
// two <= 32 and c in {1, 2, 4, 8, 16}: with kernel_flag 2 always, with
// kernel_flag 0 when the block rows are uneven enough (choose_bsr_kernel);
// kernel_flag 1 is the thread-per-row kernel.
template <typename V>
bool try_bsr_stream(const sspmv_bsr *A, V alpha, const V *x, V beta, V *y, sspmv_stream_t s, sspmv_status *st) {
    if (A->f.kernel_flag == 1 || A->nnzb > 0x7fffffff || A->nnzb == 0) return false;
    const int lr = log2_exact(A->blockDim_r);
    if (lr < 0 || lr > 5) return false;
    if (A->blockDim_c != 1 && A->blockDim_c != 2 && A->blockDim_c != 4 && A->blockDim_c != 8 && A->blockDim_c != 16)
        return false;
    Plan *p = get_plan(&A->f);
    if (!p) {
        *st = fail(SSPMV_OUT_OF_MEMORY, "plan allocation failed");
        return true;
    }
    if (A->f.kernel_flag != 2) {
        *st = choose_bsr_kernel(A, p, s);
        if (*st != SSPMV_OK) return true;
        if ((p->extra_i[2] & 3) != 1) return false;
    }
    switch (A->blockDim_c) {
    case 1: *st = launch_bsr_stream<V, 1>(A, p, alpha, x, beta, y, s); return true;
    case 2: *st = launch_bsr_stream<V, 2>(A, p, alpha, x, beta, y, s); return true;
    case 4: *st = launch_bsr_stream<V, 4>(A, p, alpha, x, beta, y, s); return true;
    case 8: *st = launch_bsr_stream<V, 8>(A, p, alpha, x, beta, y, s); return true;
    case 16: *st = launch_bsr_stream<V, 16>(A, p, alpha, x, beta, y, s); return true;
    default: return false;
    }
}

template <typename V, int K, int CB>
sspmv_status launch_bsr_c(const sspmv_bsr *A, V alpha, const V *x, int64_t ldx, V beta, V *y, int64_t ldy,
                          sspmv_stream_t s) {
    const unsigned grid = grid_for(A->f.num_rows, kBlock, (int64_t)num_sms() * 16);
    auto go = [&](auto kernel) {
        kernel<<<grid, kBlock, 0, cu(s)>>>((int)A->f.num_rows, (int)A->f.num_cols, (int)A->blockDim_r,
                                           (int)A->blockDim_c, A->row_ptr, A->block_colindex,
                                           (const V *)A->block_data, x, ldx, xrow_vec(x, ldx, sizeof(V), K), alpha,
                                           beta, y, ldy);
    };
    if (K == 1 && alpha == V(1) && beta == V(0)) go(bsr_spmv_kernel<V, K, CB, K == 1>);  // y = sum
    else go(bsr_spmv_kernel<V, K, CB>);
    SSPMV_LAUNCH_CHECK();
    return SSPMV_OK;
}

template <typename V, int K>
sspmv_status launch_bsr(const sspmv_bsr *A, V alpha, const V *x, int64_t ldx, V beta, V *y, int64_t ldy,
                        sspmv_stream_t s) {
    switch (A->blockDim_c) {
    case 1: return launch_bsr_c<V, K, 1>(A, alpha, x, ldx, beta, y, ldy, s);
    case 2: return launch_bsr_c<V, K, 2>(A, alpha, x, ldx, beta, y, ldy, s);
    case 4: return launch_bsr_c<V, K, 4>(A, alpha, x, ldx, beta, y, ldy, s);
    case 8: return launch_bsr_c<V, K, 8>(A, alpha, x, ldx, beta, y, ldy, s);
    case 16: return launch_bsr_c<V, K, 16>(A, alpha, x, ldx, beta, y, ldy, s);
    default: return launch_bsr_c<V, K, 0>(A, alpha, x, ldx, beta, y, ldy, s);
    }
}

}  // namespace

extern "C" sspmv_status sspmv_csr_to_bsr(const sspmv_csr *csr, int32_t r, int32_t c, sspmv_bsr *out,
                                         sspmv_stream_t s) {
    if (!csr || !out) return fail(SSPMV_INVALID_ARG, "null argument");
    SSPMV_TRY(check_dims(csr->f.value_type, csr->f.num_rows, csr->f.num_cols, csr->f.num_nnzs));
    if (r == 0) r = 16;
    if (c == 0) c = default_alignment(csr->f.value_type);
    if (r < 1 || c < 1) return fail(SSPMV_INVALID_ARG, "block dimensions must be >= 1");
    const int64_t m = csr->f.num_rows, n = csr->f.num_cols, nnz = csr->f.num_nnzs;
    const int32_t vt = csr->f.value_type;
    const size_t sv = vsize(vt);
    sspmv_bsr A;
    init_features(&A.f, vt, m, n, nnz, 1);
    A.blockDim_r = r;
    A.blockDim_c = c;
    A.blockNNZ = (int64_t)r * c;
    A.mb = (m + r - 1) / r;
    A.nb = (n + c - 1) / c;
    A.row_ptr = nullptr;
    A.block_colindex = nullptr;
    A.block_data = nullptr;
    const unsigned g = grid_for(std::max<int64_t>(m, 1), 256, (int64_t)num_sms() * 16);
    sspmv_status st = SSPMV_OK;
    if (r == 1 && c == 1) {  // include/sparse_conversion.h:784-815: copies of the CSR arrays
        A.nnzb = nnz;
        st = dalloc(&A.row_ptr, (size_t)m + 1, s);
        if (st == SSPMV_OK) st = dalloc(&A.block_colindex, (size_t)nnz, s);
        if (st == SSPMV_OK) st = dalloc((unsigned char **)&A.block_data, (size_t)nnz * sv, s);
        if (st == SSPMV_OK) {
            cudaError_t e = cudaMemcpyAsync(A.row_ptr, csr->row_offset, ((size_t)m + 1) * 4, cudaMemcpyDeviceToDevice, cu(s));
            if (e == cudaSuccess && nnz)
                e = cudaMemcpyAsync(A.block_colindex, csr->col_index, (size_t)nnz * 4, cudaMemcpyDeviceToDevice, cu(s));
            if (e == cudaSuccess && nnz)
                e = cudaMemcpyAsync(A.block_data, csr->values, (size_t)nnz * sv, cudaMemcpyDeviceToDevice, cu(s));
            if (e == cudaSuccess) e = cudaStreamSynchronize(cu(s));
            if (e != cudaSuccess) st = fail(SSPMV_CUDA_ERROR, "csr_to_bsr copy: %s", cudaGetErrorString(e));
        }
    } else {
        uint64_t *keys = nullptr, *ukeys = nullptr;
        uint32_t *vals = nullptr;
        int32_t *pos = nullptr;
        int32_t nnzb = 0;
        st = dalloc(&keys, (size_t)nnz, s);
        if (st == SSPMV_OK) st = dalloc(&vals, (size_t)nnz, s);
        if (st == SSPMV_OK) st = dalloc(&pos, (size_t)nnz, s);
        if (st == SSPMV_OK && nnz > 0) {
            bsr_keys<<<g, 256, 0, cu(s)>>>(m, r, c, A.nb, csr->row_offset, csr->col_index, keys, vals);
            note_launch();
            st = radix_sort_pairs(keys, vals, nnz, bits_for((uint64_t)(A.mb * A.nb)), s);
            if (st == SSPMV_OK) {
                unique_flags<<<grid_for(nnz, 256, (int64_t)num_sms() * 16), 256, 0, cu(s)>>>(nnz, keys, pos);
                note_launch();
                st = exclusive_scan_i32(pos, pos, nnz, &nnzb, s);
            }
        }
        A.nnzb = nnzb;
        if (st == SSPMV_OK) st = dalloc(&ukeys, (size_t)nnzb, s);
        if (st == SSPMV_OK) st = dalloc(&A.block_colindex, (size_t)nnzb, s);
        if (st == SSPMV_OK) st = dalloc(&A.row_ptr, (size_t)A.mb + 1, s);
        if (st == SSPMV_OK) st = dalloc((unsigned char **)&A.block_data, (size_t)nnzb * A.blockNNZ * sv, s);
        if (st == SSPMV_OK) {
            cudaMemsetAsync(A.block_data, 0, (size_t)nnzb * A.blockNNZ * sv, cu(s));
            if (nnz > 0) {
                unique_scatter<<<grid_for(nnz, 256, (int64_t)num_sms() * 16), 256, 0, cu(s)>>>(nnz, keys, pos, A.nb,
                                                                                            ukeys, A.block_colindex);
                note_launch();
            }
            bsr_row_ptr<<<grid_for(A.mb + 1, 256), 256, 0, cu(s)>>>(A.mb, A.nb, nnzb, ukeys, A.row_ptr);
            note_launch();
            if (m > 0)
                st = dispatch_value(vt, [&](auto tag) -> sspmv_status {
                    using V = decltype(tag);
                    bsr_fill<V><<<g, 256, 0, cu(s)>>>(m, r, c, csr->row_offset, csr->col_index, (const V *)csr->values,
                                                      A.row_ptr, A.block_colindex, (V *)A.block_data);
                    SSPMV_LAUNCH_CHECK();
                    return SSPMV_OK;
                });
            cudaError_t e = cudaStreamSynchronize(cu(s));
            if (st == SSPMV_OK && e != cudaSuccess) st = fail(SSPMV_CUDA_ERROR, "csr_to_bsr: %s", cudaGetErrorString(e));
        }
        dfree(keys, s);
        dfree(vals, s);
        dfree(pos, s);
        dfree(ukeys, s);
    }
    if (st != SSPMV_OK) {
        dfree(A.row_ptr, s);
        dfree(A.block_colindex, s);
        dfree(A.block_data, s);
        return st;
    }
    *out = A;
    return SSPMV_OK;
}

extern "C" sspmv_status sspmv_csr_count_blocks(const sspmv_csr *csr, int32_t r, int32_t c, int64_t *nnzb,
                                               sspmv_stream_t s) {
    if (!csr || !nnzb) return fail(SSPMV_INVALID_ARG, "null argument");
    if (r < 1 || c < 1) return fail(SSPMV_INVALID_ARG, "block dimensions must be >= 1");
    const int64_t m = csr->f.num_rows, n = csr->f.num_cols, nnz = csr->f.num_nnzs;
    *nnzb = 0;
    if (nnz == 0) return SSPMV_OK;
    const int64_t mb = (m + r - 1) / r, nb = (n + c - 1) / c;
    uint64_t *keys = nullptr;
    uint32_t *vals = nullptr;
    int32_t *pos = nullptr;
    sspmv_status st = dalloc(&keys, (size_t)nnz, s);
    if (st == SSPMV_OK) st = dalloc(&vals, (size_t)nnz, s);
    if (st == SSPMV_OK) st = dalloc(&pos, (size_t)nnz, s);
    if (st == SSPMV_OK) {
        bsr_keys<<<grid_for(m, 256, (int64_t)num_sms() * 16), 256, 0, cu(s)>>>(m, r, c, nb, csr->row_offset,
                                                                                csr->col_index, keys, vals);
        note_launch();
        st = radix_sort_pairs(keys, vals, nnz, bits_for((uint64_t)(mb * nb)), s);
    }
    int32_t total = 0;
    if (st == SSPMV_OK) {
        unique_flags<<<grid_for(nnz, 256, (int64_t)num_sms() * 16), 256, 0, cu(s)>>>(nnz, keys, pos);
        note_launch();
        st = exclusive_scan_i32(pos, pos, nnz, &total, s);
    }
    dfree(keys, s);
    dfree(vals, s);
    dfree(pos, s);
    if (st == SSPMV_OK) *nnzb = total;
    return st;
}

extern "C" sspmv_status sspmv_spmm_bsr(double alpha, const sspmv_bsr *A, int32_t k, const void *X, int64_t ldx,
                                       double beta, void *Y, int64_t ldy, sspmv_stream_t s) {
    if (!A) return fail(SSPMV_INVALID_ARG, "null matrix");
    SSPMV_TRY(check_spmm_args(&A->f, k, X, ldx, Y, ldy));
    if (A->f.num_rows == 0) return SSPMV_OK;
    return dispatch_value(A->f.value_type, [&](auto tag) -> sspmv_status {
        using V = decltype(tag);
        return for_rhs_chunks<V>(k, (const V *)X, (V *)Y, [&](int32_t step, const V *xs, V *ys) {
            const V a = (V)alpha, b = (V)beta;
            if (step == 1 && ldx == 1 && ldy == 1) {
                sspmv_status st = SSPMV_OK;
                if (try_bsr_stream<V>(A, a, xs, b, ys, s, &st)) return st;
            }
            switch (step) {
            case 8: return launch_bsr<V, 8>(A, a, xs, ldx, b, ys, ldy, s);
            case 4: return launch_bsr<V, 4>(A, a, xs, ldx, b, ys, ldy, s);
            case 2: return launch_bsr<V, 2>(A, a, xs, ldx, b, ys, ldy, s);
            default: return launch_bsr<V, 1>(A, a, xs, ldx, b, ys, ldy, s);
            }
        });
    });
}

extern "C" sspmv_status sspmv_LeSpMV_bsr(double alpha, const sspmv_bsr *A, const void *x, double beta, void *y,
                                         sspmv_stream_t s) {
    return sspmv_spmm_bsr(alpha, A, 1, x, 1, beta, y, 1, s);
}

extern "C" sspmv_status sspmv_bsr_export(const sspmv_bsr *A, int32_t *row_ptr, int32_t *block_colindex,
                                         void *block_data, sspmv_stream_t s) {
    if (!A) return fail(SSPMV_INVALID_ARG, "null matrix");
    const bool one = A->blockDim_r == 1 && A->blockDim_c == 1;
    const size_t nrp = (size_t)(one ? A->f.num_rows : A->mb) + 1;
    if (row_ptr) SSPMV_CUDA_TRY(cudaMemcpyAsync(row_ptr, A->row_ptr, nrp * 4, cudaMemcpyDeviceToHost, cu(s)));
    if (block_colindex && A->nnzb)
        SSPMV_CUDA_TRY(cudaMemcpyAsync(block_colindex, A->block_colindex, (size_t)A->nnzb * 4, cudaMemcpyDeviceToHost, cu(s)));
    if (block_data && A->nnzb)
        SSPMV_CUDA_TRY(cudaMemcpyAsync(block_data, A->block_data, (size_t)A->nnzb * A->blockNNZ * vsize(A->f.value_type),
                                       cudaMemcpyDeviceToHost, cu(s)));
    SSPMV_CUDA_TRY(cudaStreamSynchronize(cu(s)));
    return SSPMV_OK;
}

extern "C" sspmv_status sspmv_delete_bsr(sspmv_bsr *A) {
    if (!A) return SSPMV_OK;
    const DeleteScope scope;
    free_plan(&A->f, nullptr);
    if (A->f.owns) {
        dfree(A->row_ptr, nullptr);
        dfree(A->block_colindex, nullptr);
        dfree(A->block_data, nullptr);
    }
    A->row_ptr = A->block_colindex = nullptr;
    A->block_data = nullptr;
    return SSPMV_OK;
}

extern "C" double sspmv_algorithmic_bytes_bsr(const sspmv_bsr *A, int32_t k, int32_t beta_nonzero) {
    const double sv = (double)vsize(A->f.value_type);
    return (double)A->f.num_nnzs * sv + (double)A->nnzb * 4.0 + (double)(A->mb + 1) * 4.0 +
           (double)k * (double)A->f.num_cols * sv + (double)k * (double)A->f.num_rows * sv * (beta_nonzero ? 2.0 : 1.0);
}
