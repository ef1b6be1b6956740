// sigma = H x over full-row storage (both triangles, diagonal kept apart), and the
// dispatch to the tiled upper-triangle kernels (tiles.cu).
//
// Replaces SparseMatUpperTri::matrix_vector_prod (src/var/sparse.rs:64-78).  With
// both triangles stored every output is a private warp reduction: one warp per row,
// the column/value streams read once with evict-first loads so that the gathered
// vector x stays resident in L2.  Upper-triangle storage (the reference's own layout,
// half the bytes) goes through the tiled kernels.
#include <algorithm>
#include <type_traits>

#include "bits.cuh"
#include "internal.cuh"

namespace risq {

namespace {

constexpr unsigned FULL = 0xffffffffu;

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
    return v;
}

// VK 0: FP64 values, FP64 vectors.  VK 1: FP32 values, FP32 vectors (FP32 sums).
// VK 2: FP32 value + FP32 remainder, FP64 vectors.
//
// One warp per row, consecutive warps on consecutive rows.  What bounds it is the latency
// of the column stream (HBM) followed by the gather of x (L1 / L2), so the loop is
// software pipelined: the next 256 elements' (192 with remainders) columns and values (of
// this row, or the first ones of the warp's next row) are in flight while this chunk's x
// are gathered.
// Measured, CUDA events: 200,003 rows, 2.0e8 elements, FP32: 420 us with four loads per
// lane and no pipelining, 365 us here (4.4 TB/s of stream); 131,611 rows, 1.2e8
// elements, FP64: 264 -> 253 us (5.6 TB/s); 6,943 rows: 13.9 -> 11.5 us; FP32 + remainder
// 327 -> 286 us, with six elements a lane (eight need more than the 64 registers of four
// CTAs: 311), kept as they are stored until x is there (added on load, the chunk waited for
// its own loads: 387).  Larger blocks, and contiguous runs of rows per block, were slower
// (1.1x and 1.3-2x).

template <int VK, typename X>
__global__ void __launch_bounds__(256, 4) k_spmv(int64_t N, const int64_t* __restrict__ row_start,
                                                 const int32_t* __restrict__ row_len, const int32_t* __restrict__ cols,
                                                 const double* __restrict__ v64, const float* __restrict__ v32,
                                                 const float* __restrict__ vlo, const double* __restrict__ diag,
                                                 const X* __restrict__ x, X* __restrict__ y,
                                                 const int* __restrict__ stop) {
    if (stop && *stop) return;
    using A = typename std::conditional<VK == 1, float, double>::type;
    using R = typename std::conditional<VK == 2, float2, A>::type;  // a value as it is stored
    constexpr int SPMV_U = VK == 2 ? 6 : 8;  // elements per lane in one chunk
    const int lane = threadIdx.x & 31;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    int64_t p = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    if (p >= N) return;
    // a chunk's columns (-1: past the row's end) and values
    auto load = [&](int64_t s, int k0, int len, int (&c)[SPMV_U], R (&a)[SPMV_U]) {
#pragma unroll
        for (int j = 0; j < SPMV_U; j++) {
            const int k = k0 + lane + 32 * j;
            c[j] = -1;
            a[j] = R{};
            if (k < len) {
                c[j] = __ldcs(cols + s + k);
                if constexpr (VK == 0) a[j] = __ldcs(v64 + s + k);
                else if constexpr (VK == 2) a[j] = make_float2(__ldcs(v32 + s + k), __ldcs(vlo + s + k));
                else a[j] = __ldcs(v32 + s + k);
            }
        }
    };
    auto value = [](R r) -> A {
        if constexpr (VK == 2) return (double)r.x + (double)r.y;
        else return r;
    };
    int64_t s = row_start[p], s_next = 0;
    int len = row_len[p], len_next = 0;
    if (p + nwarps < N) {
        s_next = row_start[p + nwarps];
        len_next = row_len[p + nwarps];
    }
    int c[SPMV_U], cn[SPMV_U];
    R a[SPMV_U], an[SPMV_U];
    load(s, 0, len, c, a);
    int k0 = 0;
    A acc = 0;
    for (;;) {
        const bool more = k0 + 32 * SPMV_U < len;
        const int kn = more ? k0 + 32 * SPMV_U : 0;
        load(more ? s : s_next, kn, more ? len : len_next, cn, an);
        A xv[SPMV_U];
#pragma unroll
        for (int j = 0; j < SPMV_U; j++) xv[j] = c[j] >= 0 ? (A)__ldg(x + c[j]) : (A)0;
#pragma unroll
        for (int j = 0; j < SPMV_U; j++)
            if (c[j] >= 0) acc += value(a[j]) * xv[j];
        if (!more) {
            acc = warp_sum(acc);
            if (lane == 0) y[p] = (X)(diag[p] * (double)x[p] + (double)acc);
            acc = 0;
            p += nwarps;
            if (p >= N) break;
            s = s_next;
            len = len_next;
            len_next = 0;
            if (p + nwarps < N) {
                s_next = row_start[p + nwarps];
                len_next = row_len[p + nwarps];
            }
        }
        k0 = kn;
#pragma unroll
        for (int j = 0; j < SPMV_U; j++) {
            c[j] = cn[j];
            a[j] = an[j];
        }
    }
}

// The same for sets of more rows than the chip holds warps whose rows hold few elements: a row
// is then a chain of three latencies (its start, its columns, x) and k_spmv's chunks mostly
// empty.  A warp takes NR rows at once, U elements a lane of each; every row's sums are formed
// in the order of k_spmv.  Measured, 100,000 rows, FP64, us: 2 elements a row 24.0 (k_spmv
// 41.8), 60: 30.4 (44.1), 84: 34.5 (44.5) with two rows and one element; 113: 38.5 (47.4) with
// one row and four (54 with two and one).  Rows of 300 and more: k_spmv is the faster one.
constexpr int64_t ROWS_TWO = 96, ROWS_ONE = 192;  // elements a row, on average, up to which

template <int VK, typename X, int NR, int U>
__global__ void __launch_bounds__(256) k_spmv_short(int64_t N, const int64_t* __restrict__ row_start,
                                                    const int32_t* __restrict__ row_len, const int32_t* __restrict__ cols,
                                                    const double* __restrict__ v64, const float* __restrict__ v32,
                                                    const float* __restrict__ vlo, const double* __restrict__ diag,
                                                    const X* __restrict__ x, X* __restrict__ y,
                                                    const int* __restrict__ stop) {
    if (stop && *stop) return;
    using A = typename std::conditional<VK == 1, float, double>::type;
    const int lane = threadIdx.x & 31;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t p0 = ((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5) * NR; p0 < N; p0 += nwarps * NR) {
        int64_t s[NR];
        int len[NR], most = 0;
        A acc[NR];
#pragma unroll
        for (int r = 0; r < NR; r++) {
            s[r] = 0;
            len[r] = 0;
            acc[r] = 0;
            if (p0 + r < N) {
                s[r] = row_start[p0 + r];
                len[r] = row_len[p0 + r];
            }
            most = max(most, len[r]);
        }
        for (int k0 = lane; k0 < most; k0 += 32 * U) {
            int c[NR][U];
            A a[NR][U], xv[NR][U];
#pragma unroll
            for (int r = 0; r < NR; r++)
#pragma unroll
                for (int j = 0; j < U; j++) {
                    const int k = k0 + 32 * j;
                    c[r][j] = -1;
                    a[r][j] = 0;
                    if (k < len[r]) {
                        c[r][j] = __ldcs(cols + s[r] + k);
                        if constexpr (VK == 0) a[r][j] = __ldcs(v64 + s[r] + k);
                        else if constexpr (VK == 2) a[r][j] = (double)__ldcs(v32 + s[r] + k) + (double)__ldcs(vlo + s[r] + k);
                        else a[r][j] = __ldcs(v32 + s[r] + k);
                    }
                }
#pragma unroll
            for (int r = 0; r < NR; r++)
#pragma unroll
                for (int j = 0; j < U; j++) xv[r][j] = c[r][j] >= 0 ? (A)__ldg(x + c[r][j]) : (A)0;
#pragma unroll
            for (int r = 0; r < NR; r++)
#pragma unroll
                for (int j = 0; j < U; j++)
                    if (c[r][j] >= 0) acc[r] += a[r][j] * xv[r][j];
        }
#pragma unroll
        for (int r = 0; r < NR; r++) acc[r] = warp_sum(acc[r]);
#pragma unroll
        for (int r = 0; r < NR; r++)
            if (lane == r && p0 + r < N) y[p0 + r] = (X)(diag[p0 + r] * (double)x[p0 + r] + (double)acc[r]);
    }
}

// FP64 sigma that recomputes every stored element from the two determinants and
// the integrals (Slater-Condon in FP64, bitwise the values a FP64 build stores),
// reading only the int32 column stream from HBM.  SMEM: the packed integral tables
// are staged in shared memory (n <= 20 fits in 227 KB).
template <int W, bool SMEM>
__global__ void __launch_bounds__(1024, 1) k_spmv_otf(int64_t N, const uint64_t* __restrict__ up,
                                                      const uint64_t* __restrict__ dn,
                                                      const int64_t* __restrict__ row_start,
                                                      const int32_t* __restrict__ row_len,
                                                      const int32_t* __restrict__ cols,
                                                      const double* __restrict__ diag, Ints Ig, uint32_t n1,
                                                      uint32_t n2, const double* __restrict__ x,
                                                      double* __restrict__ y, const int* __restrict__ stop) {
    if (stop && *stop) return;
    extern __shared__ double sm[];
    if constexpr (SMEM) {
        for (uint32_t k = threadIdx.x; k < n1; k += blockDim.x) sm[k] = Ig.h1[k];
        for (uint32_t k = threadIdx.x; k < n2; k += blockDim.x) sm[n1 + k] = Ig.h2[k];
        __syncthreads();
    }
    const IntsShared Is{sm, sm + n1, Ig.nuc};
    const int lane = threadIdx.x & 31;
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t p = warp; p < N; p += nwarps) {
        Bits<W> a, b;
#pragma unroll
        for (int k = 0; k < W; k++) { a.w[k] = __ldg(up + k * N + p); b.w[k] = __ldg(dn + k * N + p); }
        const int64_t s = row_start[p];
        const int len = row_len[p];
        double acc = 0.0;
        for (int k = lane; k < len; k += 32) {
            const int q = __ldcs(cols + s + k);
            Bits<W> aq, bq;
#pragma unroll
            for (int w = 0; w < W; w++) { aq.w[w] = __ldg(up + w * N + q); bq.w[w] = __ldg(dn + w * N + q); }
            double v;
            if constexpr (SMEM) v = sc_pair<W, IntsShared>(Is, a, b, aq, bq);
            else v = sc_pair<W, Ints>(Ig, a, b, aq, bq);
            acc += v * __ldg(x + q);
        }
        acc = warp_sum(acc);
        if (lane == 0) y[p] = diag[p] * x[p] + acc;
    }
}

template <int W>
int launch_otf(risqgpu* h, const double* x, double* y) {
    const int64_t n = (int64_t)h->N;
    Ints I{h->d_h1, h->d_h2, h->nuc};
    const size_t smem = sizeof(double) * (h->n1 + h->n2);
    int max_smem = 0;
    cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, h->device);
    if (smem <= (size_t)max_smem) {
        RQ_TRY((allow_smem(h, k_spmv_otf<W, true>, smem)));
        k_spmv_otf<W, true><<<num_sms(h), 1024, smem, h->stream>>>(n, h->d_up, h->d_dn, h->d_row_start, h->d_row_len,
                                                                   h->d_cols, h->d_diag, I, (uint32_t)h->n1,
                                                                   (uint32_t)h->n2, x, y, h->stop_flag);
    } else {
        int occ = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_spmv_otf<W, false>, 1024, 0);
        k_spmv_otf<W, false><<<num_sms(h) * std::max(occ, 1), 1024, 0, h->stream>>>(
            n, h->d_up, h->d_dn, h->d_row_start, h->d_row_len, h->d_cols, h->d_diag, I, (uint32_t)h->n1,
            (uint32_t)h->n2, x, y, h->stop_flag);
    }
    return check_launch(h, "sigma otf");
}

__global__ void k_permute_in(const double* __restrict__ x, const int32_t* __restrict__ orig, int64_t n,
                             double* __restrict__ xi) {
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x)
        xi[p] = x[orig[p]];
}
__global__ void k_permute_out(const double* __restrict__ yi, const int32_t* __restrict__ orig, int64_t n,
                              double* __restrict__ y) {
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x)
        y[orig[p]] = yi[p];
}

// Second-order self-energy of every determinant over the stored matrix:
// S_i = -sum_{j != i} H_ij^2 / max(H_jj - E, gmin).  VK as in k_spmv (0 FP64 values,
// 1 FP32, 2 FP32 + remainder).  One warp per row, private sum.
template <int VK>
__global__ void __launch_bounds__(256) k_self_energy(int64_t N, const int64_t* __restrict__ row_start,
                                                     const int32_t* __restrict__ row_len,
                                                     const int32_t* __restrict__ cols, const double* __restrict__ v64,
                                                     const float* __restrict__ v32, const float* __restrict__ vlo,
                                                     const double* __restrict__ diag, double energy, double gmin,
                                                     double* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t p = warp; p < N; p += nwarps) {
        const int64_t s = row_start[p];
        const int len = row_len[p];
        double acc = 0.0;
        for (int k = lane; k < len; k += 32) {
            const int c = cols[s + k];
            double v;
            if constexpr (VK == 0) v = v64[s + k];
            else if constexpr (VK == 2) v = (double)v32[s + k] + (double)vlo[s + k];
            else v = (double)v32[s + k];
            acc += v * v / fmax(diag[c] - energy, gmin);
        }
        acc = warp_sum(acc);
        if (lane == 0) out[p] = -acc;
    }
}

}  // namespace

int sigma_device(risqgpu* h, const void* x, void* y, int kind) {
    if (!h->built) { h->err = "sigma before build"; return RISQGPU_ERR_INVALID; }
    const int64_t n = (int64_t)h->N;
    if (h->upper) return sigma_tiles(h, x, y, kind);
    if (h->precision == RISQGPU_MATRIX_FREE) {
        if (kind != 0) {
            h->err = "a matrix-free build has only the FP64 sigma";
            return RISQGPU_ERR_INVALID;
        }
        return sigma_matrix_free(h, (const double*)x, (double*)y);
    }
    // every warp of the chip resident, no more of them than rows
    const int64_t chip = (int64_t)num_sms(h) * 32, nnz = (int64_t)h->nnz_full;
    const bool two = n > chip && nnz <= ROWS_TWO * n, one = !two && n > chip && nnz <= ROWS_ONE * n;
    const int64_t ctas = two ? (n + 15) / 16 : (n + 7) / 8;
    const int grid = (int)std::min<int64_t>(ctas, (int64_t)num_sms(h) * (two || one ? 8 : 4));
    auto go = [&](auto kern, const double* v64, const float* v32, const float* vlo, auto* xv, auto* yv) {
        kern<<<grid, 256, 0, h->stream>>>(n, h->d_row_start, h->d_row_len, h->d_cols, v64, v32, vlo, h->d_diag, xv, yv,
                                          h->stop_flag);
    };
    if (kind == 0) {
        const double* xd = (const double*)x;
        double* yd = (double*)y;
        if (h->precision == RISQGPU_FP64)
            go(two ? k_spmv_short<0, double, 2, 1> : one ? k_spmv_short<0, double, 1, 4> : k_spmv<0, double>, h->d_val64, nullptr,
               nullptr, xd, yd);
        else if (h->precision == RISQGPU_MIXED)
            go(two ? k_spmv_short<2, double, 2, 1> : one ? k_spmv_short<2, double, 1, 4> : k_spmv<2, double>, nullptr, h->d_val32,
               h->d_val_lo, xd, yd);
        else  // FP32 or columns-only storage: exact FP64 elements recomputed on the fly
            return h->W == 1 ? launch_otf<1>(h, xd, yd) : launch_otf<2>(h, xd, yd);
    } else {
        if (h->precision == RISQGPU_FP64 || h->precision == RISQGPU_COLS) {
            h->err = "FP32 sigma needs an FP32 or MIXED build";
            return RISQGPU_ERR_INVALID;
        }
        go(two ? k_spmv_short<1, float, 2, 1> : one ? k_spmv_short<1, float, 1, 4> : k_spmv<1, float>, nullptr, h->d_val32, nullptr,
           (const float*)x, (float*)y);
    }
    return check_launch(h, "sigma");
}

int permute_in(risqgpu* h, const double* x, double* xi) {
    const int64_t n = (int64_t)h->N;
    const int g = std::max(1, (int)std::min<int64_t>((n + 255) / 256, 148 * 16));
    k_permute_in<<<g, 256, 0, h->stream>>>(x, h->d_orig, n, xi);
    return check_launch(h, "permute in");
}

int permute_out(risqgpu* h, const double* yi, double* y) {
    const int64_t n = (int64_t)h->N;
    const int g = std::max(1, (int)std::min<int64_t>((n + 255) / 256, 148 * 16));
    k_permute_out<<<g, 256, 0, h->stream>>>(yi, h->d_orig, n, y);
    return check_launch(h, "permute out");
}

int sigma_host(risqgpu* h, const double* x, double* y, int nvec) {
    if (!h->built) { h->err = "sigma before build"; return RISQGPU_ERR_INVALID; }
    if (nvec < 1) { h->err = "nvec < 1"; return RISQGPU_ERR_INVALID; }
    const int64_t n = (int64_t)h->N;
    double *dx = nullptr, *dxi = nullptr, *dyi = nullptr;
    ScopedFree<3> release(dx, dxi, dyi);
    RQ_TRY(dalloc(h, dx, n));
    RQ_TRY(dalloc(h, dxi, n));
    RQ_TRY(dalloc(h, dyi, n));
    for (int c = 0; c < nvec; c++) {
        RQ_CUDA(h, cudaMemcpyAsync(dx, x + (size_t)c * n, sizeof(double) * n, cudaMemcpyHostToDevice, h->stream));
        RQ_TRY(permute_in(h, dx, dxi));
        RQ_TRY(sigma_device(h, dxi, dyi, 0));
        RQ_TRY(permute_out(h, dyi, dx));
        RQ_CUDA(h, cudaMemcpyAsync(y + (size_t)c * n, dx, sizeof(double) * n, cudaMemcpyDeviceToHost, h->stream));
    }
    return sync(h, "sigma_host");
}

int self_energy_impl(risqgpu* h, double energy, double gmin, double* out) {
    if (!h->built) { h->err = "self energy before build"; return RISQGPU_ERR_INVALID; }
    if (h->precision == RISQGPU_COLS || h->precision == RISQGPU_MATRIX_FREE) {
        h->err = "self energy needs stored values (not COLS or MATRIX_FREE)";
        return RISQGPU_ERR_INVALID;
    }
    if (!(gmin > 0.0)) { h->err = "gmin must be positive"; return RISQGPU_ERR_INVALID; }
    const int64_t n = (int64_t)h->N;
    double *si = nullptr, *sc = nullptr;
    ScopedFree<2> release(si, sc);
    RQ_TRY(dalloc(h, si, n));
    RQ_TRY(dalloc(h, sc, n));
    RQ_CUDA(h, cudaMemsetAsync(si, 0, sizeof(double) * n, h->stream));
    if (h->tiled) {
        RQ_TRY(tiles_self_energy(h, energy, gmin, si));
        RQ_TRY(permute_out(h, si, sc));
        RQ_CUDA(h, cudaMemcpyAsync(out, sc, sizeof(double) * n, cudaMemcpyDeviceToHost, h->stream));
        return sync(h, "self energy");
    }
    const int grid = num_sms(h) * 8;
    if (h->precision == RISQGPU_FP64)
        k_self_energy<0><<<grid, 256, 0, h->stream>>>(n, h->d_row_start, h->d_row_len, h->d_cols, h->d_val64, nullptr,
                                                      nullptr, h->d_diag, energy, gmin, si);
    else if (h->precision == RISQGPU_MIXED)
        k_self_energy<2><<<grid, 256, 0, h->stream>>>(n, h->d_row_start, h->d_row_len, h->d_cols, nullptr, h->d_val32,
                                                      h->d_val_lo, h->d_diag, energy, gmin, si);
    else
        k_self_energy<1><<<grid, 256, 0, h->stream>>>(n, h->d_row_start, h->d_row_len, h->d_cols, nullptr, h->d_val32,
                                                      nullptr, h->d_diag, energy, gmin, si);
    RQ_TRY(check_launch(h, "self energy"));
    RQ_TRY(permute_out(h, si, sc));
    RQ_CUDA(h, cudaMemcpyAsync(out, sc, sizeof(double) * n, cudaMemcpyDeviceToHost, h->stream));
    return sync(h, "self energy");
}

}  // namespace risq
