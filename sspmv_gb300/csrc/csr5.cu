// csr5.cu -- CSR5 format on sm_103a: GPU converter, SpMV / SpMM, export.
//
// Format (Liu & Vinter, ICS'15; reference struct include/sparse_format.h:141-
// 166): the nonzeros are cut into tiles of sigma x omega; tile t's elements
// are stored transposed (element of lane x, position i at t*sigma*omega +
// i*omega + x) unless the tile lies inside one row ("fast track", tile_ptr
// words equal) or is the last tile.  tile_ptr[t] = row holding the tile's
// first nonzero, bit 31 set when the tile meets an empty row.  Each lane's
// first descriptor word holds y_offset (rows started in earlier lanes),
// seg_offset and one bit per position where a row starts; tiles with empty
// rows map segment numbers to rows through tile_desc_offset.
//
// Converter (csr_to_csr5, include/sparse_conversion.h:939-1379, csr5_utils.h):
// every step runs per tile or per row on the GPU and reproduces the
// reference's arrays bit for bit (tile_ptr[_p] left 0 as the reference does;
// tile_desc_offset slots the reference never writes are 0).
//
// SpMV (LeSpMV_csr5, src/spmv_csr5.cpp:439-457, which the reference builds for
// double with AVX-512 only): a lane per tile column, 32 / omega tiles per step
// of a warp, so that a warp's step is 32 sigma consecutive nonzeros, lane l
// the sigma at l sigma (c5_window).  Row ends come from the stream kernel's
// plan (csr_stream.cu: one bit per nonzero, a record per window), not from
// the tile descriptors, and one segmented scan joins the lanes of all tiles of
// a step; rows that cross a window are left in pieces and finished by the
// split-row kernel in window order.  Deterministic.  Unlike the reference,
// beta is applied to every row (the reference drops it on rows that lie inside
// one tile, src/spmv_csr5.cpp:287-288).
#include <algorithm>
#include <cstring>
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

struct Geom {
    int32_t sigma, omega, byo, bso, np, p;
};

// ------------------------------------------------------------ converter --
__global__ void c5_tile_ptr(int32_t p, int32_t tile, int32_t m, int32_t nnz, const int32_t *__restrict__ rp,
                            uint32_t *__restrict__ tp) {
    int32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= p) return;
    int64_t b = (int64_t)t * tile;
    if (b > nnz) b = nnz;
    int32_t start = 0, stop = m;
    while (stop >= start) {
        int32_t med = (stop + start) / 2;
        if (b >= rp[med]) start = med + 1;
        else stop = med - 1;
    }
    tp[t] = (uint32_t)(start - 1);
}

__global__ void c5_dirty(int32_t p, const int32_t *__restrict__ rp, const uint32_t *__restrict__ tin,
                         uint32_t *__restrict__ tout) {
    int32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= p) return;
    uint32_t start = tin[t] & 0x7FFFFFFFu, stop = tin[t + 1] & 0x7FFFFFFFu;
    uint32_t v = tin[t];
    if (start != stop) {
        for (uint32_t r = start; r <= stop; r++)
            if (rp[r] == rp[r + 1]) {
                v = start | 0x80000000u;
                break;
            }
    }
    tout[t] = v;
}

__global__ void c5_bits(int32_t m, int32_t p, Geom g, const int32_t *__restrict__ rp, uint32_t *__restrict__ td) {
    const int32_t tile = g.sigma * g.omega, bao = g.byo + g.bso;
    for (int32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < m; r += gridDim.x * blockDim.x) {
        const int32_t ptr = rp[r];
        const int32_t pid = ptr / tile;
        if (pid < p - 1) {
            const int32_t lx = (ptr / g.sigma) % g.omega;
            const int32_t glid = ptr % g.sigma + bao;
            atomicOr(td + (size_t)pid * g.omega * g.np + (size_t)(glid / 32) * g.omega + lx, 1u << (31 - glid % 32));
        }
    }
}

// include/sparse_conversion.h:1113-1213, one thread per tile
__global__ void c5_offsets_pack(int32_t p, Geom g, const uint32_t *__restrict__ tp, uint32_t *__restrict__ td,
                                int32_t *__restrict__ tdo_ptr) {
    int32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= p - 1) return;
    const bool with_empty = (tp[t] >> 31) & 1u;
    const uint32_t rs = tp[t] & 0x7FFFFFFFu, re = tp[t + 1] & 0x7FFFFFFFu;
    if (rs == re) return;
    const int32_t bao = g.byo + g.bso, omega = g.omega, sigma = g.sigma;
    uint32_t *d = td + (size_t)t * omega * g.np;
    int32_t segn[33], present[33];
    for (int32_t l = 0; l <= omega; l++) {
        segn[l] = 0;
        present[l] = 0;
    }
    present[omega] = 1;
    for (int32_t lane = 0; lane < omega; lane++) {
        int32_t stop = 0, ly = 0, pres = lane == 0;
        uint32_t bitflag = (d[lane] << bao) | ((uint32_t)pres << 31);
        const int32_t start = !((bitflag >> 31) & 1u);
        pres |= (int32_t)((bitflag >> 31) & 1u);
        for (int32_t i = 1; i < sigma; i++) {
            if ((!ly && i == 32 - bao) || (ly && (i - (32 - bao)) % 32 == 0)) {
                ly++;
                bitflag = d[(size_t)ly * omega + lane];
            }
            const int32_t ni = !ly ? i : i - (32 - bao);
            stop += (int32_t)((bitflag >> (31 - ni % 32)) & 1u);
            pres |= (int32_t)((bitflag >> (31 - ni % 32)) & 1u);
        }
        const int32_t sg = stop - start + pres;
        segn[lane] = sg > 0 ? sg : 0;
        present[lane] = pres;
    }
    int32_t run = 0;
    for (int32_t l = 0; l <= omega; l++) {
        const int32_t v = segn[l];
        segn[l] = run;
        run += v;
    }
    if (with_empty) tdo_ptr[t] = segn[omega];
    for (int32_t lane = 0; lane < omega; lane++) {
        int32_t yo = segn[lane], ss = 0, nx = lane + 1;
        if (present[lane])
            while (!present[nx] && nx < omega) {
                ss++;
                nx++;
            }
        yo = lane ? yo - 1 : 0;
        d[lane] = d[lane] | ((uint32_t)yo << (32 - g.byo)) | ((uint32_t)ss << (32 - bao));
    }
}

__device__ int32_t c5_rel_row(const int32_t *rp, int32_t rs, int32_t re, int32_t idx) {
    int32_t start = 0, stop = re - rs - 1;
    while (stop >= start) {
        const int32_t med = (stop + start) / 2;
        if (idx >= rp[rs + 1 + med]) start = med + 1;
        else stop = med - 1;
    }
    return start - 1;
}

// include/sparse_conversion.h:1254-1358, one thread per tile with empty rows
__global__ void c5_desc_offsets(int32_t p, Geom g, const int32_t *__restrict__ rp, const uint32_t *__restrict__ tp,
                                const uint32_t *__restrict__ td, const int32_t *__restrict__ tdo_ptr,
                                int32_t *__restrict__ tdo) {
    int32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= p - 1 || !((tp[t] >> 31) & 1u)) return;
    const int32_t rs = (int32_t)(tp[t] & 0x7FFFFFFFu), re = (int32_t)(tp[t + 1] & 0x7FFFFFFFu);
    const int32_t omega = g.omega, sigma = g.sigma, bao = g.byo + g.bso, bbf = 32 - bao;
    const int32_t optr = tdo_ptr[t];
    const uint32_t *d0 = td + (size_t)t * omega * g.np;
    for (int32_t lane = 0; lane < omega; lane++) {
        int32_t ly = 0;
        uint32_t d = d0[lane];
        int32_t yo = (int32_t)(d >> (32 - g.byo));
        d <<= bao;
        d = lane ? d : (d | 0x80000000u);
        if (((d >> 31) & 1u) && lane) {
            tdo[optr + yo] = c5_rel_row(rp, rs, re, t * omega * sigma + lane * sigma);
            yo++;
        }
        for (int32_t i = 1; i < sigma; i++) {
            if ((!ly && i == bbf) || (ly && !(31 & (i - bbf)))) {
                ly++;
                d = d0[(size_t)ly * omega + lane];
            }
            const int32_t ni = 31 & (!ly ? i : i - bbf);
            if ((d >> (31 - ni)) & 1u) {
                tdo[optr + yo] = c5_rel_row(rp, rs, re, t * omega * sigma + lane * sigma + i);
                yo++;
            }
        }
    }
}

template <typename T>
__global__ void c5_transpose(int64_t nnz, int32_t p, int32_t sigma, int32_t omega, const uint32_t *__restrict__ tp,
                             const T *__restrict__ in, T *__restrict__ out) {
    const int64_t tile = (int64_t)sigma * omega;
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < nnz; k += (int64_t)gridDim.x * blockDim.x) {
        const int64_t t = div_nonneg(k, (int)tile);
        if (t >= p - 1 || tp[t] == tp[t + 1]) {
            out[k] = in[k];
        } else {
            const int64_t q = k - t * tile, y = div_nonneg(q, omega), x = q - y * omega;  // destination (y, x)
            out[k] = in[t * tile + x * sigma + y];
        }
    }
}

// ------------------------------------------------------------------ SpMV --
struct C5Shape {
    int32_t sigma, omega, tiles;  // tile tiles - 1 (and what follows) is stored in CSR order
};

// One window (rows that cross its ends are split), one warp.  A tile inside
// one row is stored untransposed: its elements all belong to that row, so the
// lanes add them up in the transposed order all the same.
//
// Bound like the stream kernel by the x gathers and the shuffles queued behind
// them.  An earlier form read the tile pointer and descriptors before the
// columns' addresses were known, scanned each tile on its own and left pieces
// per tile, with a row pass for the last tile and a fix-up over all tiles:
// power-law 1M FP64 (sigma 16, omega 8) 139 us, now 95.
template <typename V, int K, int SIG, bool PLAIN>
__device__ __forceinline__ void c5_window(const StreamView &A, const C5Shape g, const V *__restrict__ x, int64_t ldx,
                                          int xvec, V alpha, V beta, V *__restrict__ y, int64_t ldy, const int64_t w,
                                          V *__restrict__ tail_val, V *__restrict__ head_val) {
    constexpr unsigned kFull = 0xffffffffu;
    constexpr bool kSeed = sizeof(V) == 8;  // as the stream kernel
    // nonzeros of a lane in flight together: for one FP64 right-hand side four
    // with 18 CTAs per SM (uniform 3M x 32, sigma 32: 367 us; eight with 14: 388)
    constexpr int kB = (K == 1 && sizeof(V) == 8) || K * sizeof(V) > 16 ? 4 : 8;
    const int lane = threadIdx.x & 31;
    const int sigma = SIG > 0 ? SIG : g.sigma;
    const V *val = static_cast<const V *>(A.val);
    const int64_t tile = (int64_t)sigma * g.omega;
    const int xl = lane & (g.omega - 1);
    const int4 rec = __ldg(A.rec + w);
    int row = rec.z;
    bool head_split = rec.w & 1;
    auto y_of = [&](int ordinal) {
        return y + (int64_t)(A.nzrow ? __ldg(A.nzrow + ordinal) : ordinal) * ldy;
    };
    auto put = [&](int ordinal, const V(&sum)[K]) {
        V *yp = y_of(ordinal);
#pragma unroll
        for (int q = 0; q < K; q++) yp[q] = row_out(PLAIN, alpha, sum[q], beta, yp + q);
    };
    V carry[K];  // the open row's sum over the earlier steps
#pragma unroll
    for (int q = 0; q < K; q++) carry[q] = V(0);
    bool later = false;
    const int64_t wend = min((w + 1) * (int64_t)A.window, (int64_t)A.nnz);
    for (int64_t b = w * (int64_t)A.window; b < wend; b += 32 * (int64_t)sigma) {  // warp-uniform
        const int64_t e0 = b + (int64_t)lane * sigma;  // this lane's nonzeros e0 .. e0 + sigma - 1
        const int64_t t = e0 / tile;
        const bool csr_order = t >= (int64_t)g.tiles - 1;
        const int64_t p0 = csr_order ? e0 : t * tile + xl;
        const int64_t step = csr_order ? 1 : g.omega;
        const int nv = (int)max((int64_t)0, min((int64_t)sigma, (int64_t)A.nnz - e0));
        // row ends of the lane, 8 at a time: bits e0 + i .. e0 + i + 7
        auto ends8 = [&](int i) -> unsigned {
            if (i >= nv) return 0u;
            const int64_t e = e0 + i;
            unsigned v = A.ends[e >> 3];
            if (SIG == 0 && (e & 7)) v |= e + 8 - (e & 7) < (int64_t)A.nnz ? (unsigned)A.ends[(e >> 3) + 1] << 8 : 0u;
            v >>= e & 7;
            const int n = nv - i;
            return v & (n >= 8 ? 0xffu : (1u << n) - 1u);
        };
        int mine = 0;
        if constexpr (SIG > 0) {
#pragma unroll
            for (int i = 0; i < sigma; i += 8) mine += __popc(ends8(i));
        } else {
            for (int i = 0; i < sigma; i += 8) mine += __popc(ends8(i) & (sigma - i < 8 ? (1u << (sigma - i)) - 1u : 0xffu));
        }
        int pos = 0, nend = 0;  // rows ended in the lanes before this one, and in the step
        const unsigned before = (1u << lane) - 1u;
        for (int bit = 0; (1 << bit) <= sigma; bit++) {
            const unsigned m = __ballot_sync(kFull, (mine >> bit) & 1);
            pos += __popc(m & before) << bit;
            nend += __popc(m) << bit;
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
        for (int i = 0; i < sigma; i += kB) {
            int c[kB];
            V a[kB], xv[kB][K];
#pragma unroll
            for (int u = 0; u < kB; u++) {
                c[u] = 0;
                a[u] = V(0);
                if (i + u < nv) {
                    c[u] = ld_stream(A.col + p0 + (i + u) * step);
                    a[u] = ld_stream(val + p0 + (i + u) * step);
                }
            }
#pragma unroll
            for (int u = 0; u < kB; u++) {
                if (i + u < nv) {
                    ld_xrow<V, K>(x, c[u], ldx, xvec != 0, xv[u]);
                } else {
#pragma unroll
                    for (int q = 0; q < K; q++) xv[u][q] = V(0);
                }
            }
            const unsigned eb = ends8(i);
#pragma unroll
            for (int u = 0; u < kB; u++) {
                if (SIG == 0 && i + u >= sigma) break;
#pragma unroll
                for (int q = 0; q < K; q++) sum[q] = fma(a[u], xv[u][q], sum[q]);
                if ((eb >> u) & 1u) {
                    if (first) {
                        first = false;
#pragma unroll
                        for (int q = 0; q < K; q++) head[q] = sum[q];
                    } else {
                        put(idx, sum);
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
        V cin[K];
#pragma unroll
        for (int q = 0; q < K; q++) cin[q] = __shfl_up_sync(kFull, sum[q], 1);
        if (mine) {
            if (lane > 0) {
#pragma unroll
                for (int q = 0; q < K; q++) head[q] += cin[q];
            }
            if (!kSeed && pos == 0 && later) {
#pragma unroll
                for (int q = 0; q < K; q++) head[q] += carry[q];
            }
            if (head_split && pos == 0) {
                V *hp = head_val + w * kMaxK;
#pragma unroll
                for (int q = 0; q < K; q++) hp[q] = head[q];
            } else {
                put(row + pos, head);
            }
        }
#pragma unroll
        for (int q = 0; q < K; q++) {
            const V last = __shfl_sync(kFull, sum[q], 31);
            carry[q] = kSeed || nend > 0 ? last : carry[q] + last;
        }
        if (nend > 0) head_split = false;
        row += nend;
        later = true;
    }
    if ((rec.w & 2) && lane == 0) {
        V *cp = tail_val + w * kMaxK;
#pragma unroll
        for (int q = 0; q < K; q++) cp[q] = carry[q];
    }
}

constexpr int kC5Block = 64;
template <typename V, int K, int SIG>
constexpr int c5_min_ctas() {
    return K == 1 ? (sizeof(V) == 8 ? 18 : SIG == 16 ? 20 : 18) : K * sizeof(V) <= 16 ? 10 : 8;
}

template <typename V, int K, int SIG, bool PLAIN>
__global__ void __launch_bounds__(kC5Block, (c5_min_ctas<V, K, SIG>())) csr5_kernel(
    const StreamView A, const C5Shape g, const V *__restrict__ x, int64_t ldx, int xvec, V alpha, V beta,
    V *__restrict__ y, int64_t ldy, V *__restrict__ tail_val, V *__restrict__ head_val) {
    const int64_t w = (int64_t)blockIdx.x * (kC5Block / 32) + (threadIdx.x >> 5);
    let_next_start();
    if (w >= A.windows) {  // rows without nonzeros
        scale_empty_rows<V, K>(A, w - A.windows, PLAIN ? V(0) : beta, y, (uint64_t)ldy * sizeof(V), false);
        return;
    }
    c5_window<V, K, SIG, PLAIN>(A, g, x, ldx, xvec, alpha, beta, y, ldy, w, tail_val, head_val);
}

// Nonzeros per window: whole steps of 32 sigma.  Where these pass the 32-bit
// range one window covers the matrix, whose nonzeros are fewer.
int c5_window_size(int64_t nnz, int sigma, int warps_per_sm) {
    const int64_t step = 32 * (int64_t)sigma;
    if (step > INT32_MAX / 5) return (int)std::min<int64_t>(step, INT32_MAX);
    return (int)step * window_steps(nnz, (int)step, (int)step, warps_per_sm);
}

template <typename V, int K>
__global__ void csr5_no_nonzeros(int64_t m, V beta, V *__restrict__ y, int64_t ldy) {
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < m; r += (int64_t)gridDim.x * blockDim.x)
#pragma unroll
        for (int q = 0; q < K; q++) y[r * ldy + q] = beta == V(0) ? V(0) : beta * y[r * ldy + q];
}

template <typename V, int K>
sspmv_status csr5_pass(const sspmv_csr5 *A, Plan *pl, V alpha, const V *x, int64_t ldx, V beta, V *y, int64_t ldy,
                       sspmv_stream_t s) {
    const int64_t m = A->f.num_rows, nnz = A->f.num_nnzs;
    if (nnz == 0) {
        csr5_no_nonzeros<V, K><<<grid_for(m, kBlock, (int64_t)num_sms() * 16), kBlock, 0, cu(s)>>>(m, beta, y, ldy);
        SSPMV_LAUNCH_CHECK();
        return SSPMV_OK;
    }
    if (A->_p > 1 && A->omega != 4 && A->omega != 8 && A->omega != 16 && A->omega != 32)
        return fail(SSPMV_NOT_SUPPORTED, "CSR5 SpMV supports omega in {4, 8, 16, 32}");
    // A single tile is in CSR order whatever its shape: steps of 16 a lane
    // (with the format's sigma one of more nonzeros than the matrix would leave
    // them all to one lane).
    const C5Shape g = A->_p > 1 ? C5Shape{A->sigma, A->omega, A->_p} : C5Shape{16, 32, 1};
    const int ctas = A->f.value_type == SSPMV_F64 ? c5_min_ctas<double, 1, 16>() : c5_min_ctas<float, 1, 16>();
    SSPMV_TRY(ensure_stream_plan(pl->stream, m, nnz, A->row_offset, nullptr, A->f.value_type, s,
                                 c5_window_size(nnz, g.sigma, ctas * (kC5Block / 32)), 0));
    const StreamView v = stream_view(pl->stream, nnz, A->col_index, A->values);
    const unsigned grid = grid_for(v.windows + empty_units(v.nempty), kC5Block / 32);
    V *tv = (V *)pl->stream.tail_val, *hv = (V *)pl->stream.head_val;
    auto go = [&](auto kernel) {
        kernel<<<grid, kC5Block, 0, cu(s)>>>(v, g, x, ldx, xrow_vec(x, ldx, sizeof(V), K), alpha, beta, y, ldy, tv, hv);
    };
    const bool plain = alpha == V(1) && beta == V(0);  // y = sum
    if (g.sigma == 16) {
        if (plain) go(csr5_kernel<V, K, 16, true>);
        else go(csr5_kernel<V, K, 16, false>);
    } else if (g.sigma == 32) {
        if (plain) go(csr5_kernel<V, K, 32, true>);
        else go(csr5_kernel<V, K, 32, false>);
    } else {
        go(csr5_kernel<V, K, 0, false>);
    }
    SSPMV_LAUNCH_CHECK();
    return launch_split_rows<V, K>(v, pl->stream, alpha, beta, y, ldy, s);
}

}  // namespace

extern "C" sspmv_status sspmv_csr_to_csr5(const sspmv_csr *csr, int32_t sigma, int32_t omega, sspmv_csr5 *out,
                                          sspmv_stream_t s) {
    if (!csr || !out) return fail(SSPMV_INVALID_ARG, "null argument");
    SSPMV_TRY(check_dims(csr->f.value_type, csr->f.num_rows, csr->f.num_cols, csr->f.num_nnzs));
    if (sigma == 0) sigma = 16;
    if (omega == 0) omega = default_alignment(csr->f.value_type);
    if (sigma < 1 || omega < 1 || omega > 32) return fail(SSPMV_INVALID_ARG, "sigma >= 1, 1 <= omega <= 32 required");
    const int64_t m = csr->f.num_rows, nnz = csr->f.num_nnzs;
    const int32_t vt = csr->f.value_type;
    const size_t sv = vsize(vt);
    sspmv_csr5 A;
    std::memset(&A, 0, sizeof(A));
    init_features(&A.f, vt, m, csr->f.num_cols, nnz, 1);
    A.sigma = sigma;
    A.omega = omega;
    // include/sparse_conversion.h:977-996
    int32_t base = 2;
    A.bit_y_offset = 1;
    while (base < sigma * omega) { base *= 2; A.bit_y_offset++; }
    base = 2;
    A.bit_scansum_offset = 1;
    while (base < omega) { base *= 2; A.bit_scansum_offset++; }
    if (A.bit_y_offset + A.bit_scansum_offset > 31) return fail(SSPMV_INVALID_ARG, "CSR5 omega too large for bit fields");
    A.num_packets = (A.bit_y_offset + A.bit_scansum_offset + sigma + 31) / 32;
    A._p = (int32_t)((nnz + (int64_t)sigma * omega - 1) / ((int64_t)sigma * omega));
    const int32_t p = A._p;
    Geom g{sigma, omega, A.bit_y_offset, A.bit_scansum_offset, A.num_packets, p};
    uint32_t *tp_tmp = nullptr;
    sspmv_status st = dalloc(&A.row_offset, (size_t)m + 1, s);
    if (st == SSPMV_OK) st = dalloc(&A.col_index, (size_t)nnz, s);
    if (st == SSPMV_OK) st = dalloc((unsigned char **)&A.values, (size_t)nnz * sv, s);
    if (st == SSPMV_OK) st = dalloc(&A.tile_ptr, (size_t)p + 1, s);
    if (st == SSPMV_OK) st = dalloc(&tp_tmp, (size_t)p + 1, s);
    if (st == SSPMV_OK) st = dalloc(&A.tile_desc, (size_t)p * omega * A.num_packets, s);
    if (st == SSPMV_OK) st = dalloc(&A.tile_desc_offset_ptr, (size_t)p + 1, s);
    if (st == SSPMV_OK) {
        cudaMemcpyAsync(A.row_offset, csr->row_offset, ((size_t)m + 1) * 4, cudaMemcpyDeviceToDevice, cu(s));
        cudaMemsetAsync(tp_tmp, 0, ((size_t)p + 1) * 4, cu(s));
        cudaMemsetAsync(A.tile_ptr, 0, ((size_t)p + 1) * 4, cu(s));
        cudaMemsetAsync(A.tile_desc, 0, (size_t)std::max<int64_t>((int64_t)p * omega * A.num_packets, 1) * 4, cu(s));
        cudaMemsetAsync(A.tile_desc_offset_ptr, 0, ((size_t)p + 1) * 4, cu(s));
        if (p > 0) {
            c5_tile_ptr<<<grid_for(p, 256), 256, 0, cu(s)>>>(p, sigma * omega, (int32_t)m, (int32_t)nnz, csr->row_offset,
                                                             tp_tmp);
            c5_dirty<<<grid_for(p, 256), 256, 0, cu(s)>>>(p, csr->row_offset, tp_tmp, A.tile_ptr);
            c5_bits<<<grid_for(m, 256, (int64_t)num_sms() * 16), 256, 0, cu(s)>>>((int32_t)m, p, g, csr->row_offset,
                                                                                  A.tile_desc);
            c5_offsets_pack<<<grid_for(p, 128), 128, 0, cu(s)>>>(p, g, A.tile_ptr, A.tile_desc, A.tile_desc_offset_ptr);
            for (int i = 0; i < 4; i++) note_launch();
            cudaError_t e = cudaGetLastError();
            if (e != cudaSuccess) st = fail(SSPMV_CUDA_ERROR, "csr_to_csr5: %s", cudaGetErrorString(e));
            int32_t total = 0;
            if (st == SSPMV_OK) st = exclusive_scan_i32(A.tile_desc_offset_ptr, A.tile_desc_offset_ptr, p + 1, &total, s);
            A.num_offsets = total;
            uint32_t last = 0;
            if (st == SSPMV_OK) {
                e = cudaMemcpyAsync(&last, A.tile_ptr + p - 1, 4, cudaMemcpyDeviceToHost, cu(s));
                if (e == cudaSuccess) e = cudaStreamSynchronize(cu(s));
                if (e != cudaSuccess) st = fail(SSPMV_CUDA_ERROR, "csr_to_csr5: %s", cudaGetErrorString(e));
            }
            A.tail_partition_start = (int32_t)(last & 0x7FFFFFFFu);
        }
    }
    if (st == SSPMV_OK) st = dalloc(&A.tile_desc_offset, (size_t)A.num_offsets, s);
    if (st == SSPMV_OK && A.num_offsets > 0) {
        cudaMemsetAsync(A.tile_desc_offset, 0, (size_t)A.num_offsets * 4, cu(s));
        c5_desc_offsets<<<grid_for(p, 128), 128, 0, cu(s)>>>(p, g, csr->row_offset, A.tile_ptr, A.tile_desc,
                                                             A.tile_desc_offset_ptr, A.tile_desc_offset);
        note_launch();
    }
    if (st == SSPMV_OK && nnz > 0) {
        const unsigned gn = grid_for(nnz, 256, (int64_t)num_sms() * 16);
        c5_transpose<int32_t><<<gn, 256, 0, cu(s)>>>(nnz, p, sigma, omega, A.tile_ptr, csr->col_index, A.col_index);
        note_launch();
        st = dispatch_value(vt, [&](auto tag) -> sspmv_status {
            using V = decltype(tag);
            c5_transpose<V><<<gn, 256, 0, cu(s)>>>(nnz, p, sigma, omega, A.tile_ptr, (const V *)csr->values,
                                                   (V *)A.values);
            SSPMV_LAUNCH_CHECK();
            return SSPMV_OK;
        });
    }
    if (st == SSPMV_OK) {
        cudaError_t e = cudaStreamSynchronize(cu(s));
        if (e != cudaSuccess) st = fail(SSPMV_CUDA_ERROR, "csr_to_csr5: %s", cudaGetErrorString(e));
    }
    dfree(tp_tmp, s);
    if (st != SSPMV_OK) {
        dfree(A.row_offset, s);
        dfree(A.col_index, s);
        dfree(A.values, s);
        dfree(A.tile_ptr, s);
        dfree(A.tile_desc, s);
        dfree(A.tile_desc_offset_ptr, s);
        dfree(A.tile_desc_offset, s);
        return st;
    }
    *out = A;
    return SSPMV_OK;
}

extern "C" sspmv_status sspmv_spmm_csr5(double alpha, const sspmv_csr5 *A, int32_t k, const void *X, int64_t ldx,
                                        double beta, void *Y, int64_t ldy, sspmv_stream_t s) {
    if (!A) return fail(SSPMV_INVALID_ARG, "null matrix");
    SSPMV_TRY(check_spmm_args(&A->f, k, X, ldx, Y, ldy));
    if (A->f.num_rows == 0) return SSPMV_OK;
    Plan *pl = get_plan(&A->f);
    if (!pl) return fail(SSPMV_OUT_OF_MEMORY, "plan allocation failed");
    return dispatch_value(A->f.value_type, [&](auto tag) -> sspmv_status {
        using V = decltype(tag);
        return for_rhs_chunks<V>(k, (const V *)X, (V *)Y, [&](int32_t step, const V *xs, V *ys) {
            const V a = (V)alpha, b = (V)beta;
            switch (step) {
            case 8: return csr5_pass<V, 8>(A, pl, a, xs, ldx, b, ys, ldy, s);
            case 4: return csr5_pass<V, 4>(A, pl, a, xs, ldx, b, ys, ldy, s);
            case 2: return csr5_pass<V, 2>(A, pl, a, xs, ldx, b, ys, ldy, s);
            default: return csr5_pass<V, 1>(A, pl, a, xs, ldx, b, ys, ldy, s);
            }
        });
    });
}

extern "C" sspmv_status sspmv_LeSpMV_csr5(double alpha, const sspmv_csr5 *A, const void *x, double beta, void *y,
                                          sspmv_stream_t s) {
    return sspmv_spmm_csr5(alpha, A, 1, x, 1, beta, y, 1, s);
}

extern "C" sspmv_status sspmv_csr5_export(const sspmv_csr5 *A, uint32_t *tile_ptr, uint32_t *tile_desc,
                                          int32_t *tile_desc_offset_ptr, int32_t *tile_desc_offset, int32_t *col_index,
                                          void *values, sspmv_stream_t s) {
    if (!A) return fail(SSPMV_INVALID_ARG, "null matrix");
    auto cp = [&](void *dst, const void *src, size_t bytes) -> sspmv_status {
        if (dst && bytes) SSPMV_CUDA_TRY(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, cu(s)));
        return SSPMV_OK;
    };
    const size_t p = (size_t)A->_p;
    SSPMV_TRY(cp(tile_ptr, A->tile_ptr, (p + 1) * 4));
    SSPMV_TRY(cp(tile_desc, A->tile_desc, p * A->omega * A->num_packets * 4));
    SSPMV_TRY(cp(tile_desc_offset_ptr, A->tile_desc_offset_ptr, (p + 1) * 4));
    SSPMV_TRY(cp(tile_desc_offset, A->tile_desc_offset, (size_t)A->num_offsets * 4));
    SSPMV_TRY(cp(col_index, A->col_index, (size_t)A->f.num_nnzs * 4));
    SSPMV_TRY(cp(values, A->values, (size_t)A->f.num_nnzs * vsize(A->f.value_type)));
    SSPMV_CUDA_TRY(cudaStreamSynchronize(cu(s)));
    return SSPMV_OK;
}

extern "C" sspmv_status sspmv_delete_csr5(sspmv_csr5 *A) {
    if (!A) return SSPMV_OK;
    const DeleteScope scope;
    free_plan(&A->f, nullptr);
    if (A->f.owns) {
        dfree(A->row_offset, nullptr);
        dfree(A->col_index, nullptr);
        dfree(A->values, nullptr);
        dfree(A->tile_ptr, nullptr);
        dfree(A->tile_desc, nullptr);
        dfree(A->tile_desc_offset_ptr, nullptr);
        dfree(A->tile_desc_offset, nullptr);
    }
    A->row_offset = A->col_index = A->tile_desc_offset_ptr = A->tile_desc_offset = nullptr;
    A->tile_ptr = A->tile_desc = nullptr;
    A->values = nullptr;
    return SSPMV_OK;
}

extern "C" double sspmv_algorithmic_bytes_csr5(const sspmv_csr5 *A, int32_t k, int32_t beta_nonzero) {
    const double sv = (double)vsize(A->f.value_type);
    return (double)A->f.num_nnzs * (sv + 4.0) + (double)(A->f.num_rows + 1) * 4.0 + (double)(A->_p + 1) * 4.0 +
           (double)A->_p * A->omega * A->num_packets * 4.0 + (double)A->num_offsets * 4.0 +
           (double)k * (double)A->f.num_cols * sv + (double)k * (double)A->f.num_rows * sv * (beta_nonzero ? 2.0 : 1.0);
}
