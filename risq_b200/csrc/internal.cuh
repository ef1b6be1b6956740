// Internal state of a risqgpu handle and shared host helpers.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <string>
#include <utility>
#include <vector>

#include "../../include/risqgpu.h"
#include "tiles.cuh"

namespace risq {

// A failed CUDA call inside a handle method: record and return.
#define RQ_CUDA(h, call)                                                                         \
    do {                                                                                         \
        cudaError_t e_ = (call);                                                                 \
        if (e_ != cudaSuccess) {                                                                 \
            (h)->err = std::string(#call) + ": " + cudaGetErrorString(e_);                       \
            return e_ == cudaErrorMemoryAllocation ? RISQGPU_ERR_OOM : RISQGPU_ERR_CUDA;         \
        }                                                                                        \
    } while (0)

#define RQ_TRY(call)                 \
    do {                             \
        int s_ = (call);             \
        if (s_ != RISQGPU_OK) return s_; \
    } while (0)

struct MlpWeights {
    int n_in = 0, hidden = 0;
    // device copies: bf16 weights as raw u16 + fp32 biases
    uint16_t *w1 = nullptr, *w2 = nullptr, *w3 = nullptr;
    float *b1 = nullptr, *b2 = nullptr, *b3 = nullptr;
    float4 fnorm = {0.f, 1.f, 0.f, 1.f};  // (mu_e, 1/sd_e, mu_h, 1/sd_h)
    bool loaded = false;
};

}  // namespace risq

struct risqgpu {
    int device = 0;
    cudaStream_t stream = nullptr;        // stream all work is issued on
    cudaStream_t own_stream = nullptr;    // the handle's own stream
    double sigma_ms_acc = 0.0;            // event time of sigma launches inside Davidson
    bool time_sigma = false;
    std::string err;
    // device memory held by this handle through dalloc, and the caller's bound on it
    // (0 = none; risqgpu_set_memory_limit)
    size_t mem_used = 0;
    size_t mem_limit = 0;

    // integrals (reference packed layout)
    int norb = 0;
    double nuc = 0.0;
    size_t n1 = 0, n2 = 0;
    double* d_h1 = nullptr;
    double* d_h2 = nullptr;
    std::vector<double> h_h1, h_h2;  // host copies (excitation tables, diagonal of HF)

    // determinant set, internal order = sorted by (up, dn)
    int W = 1;        // 64-bit words per spin string
    size_t N = 0;     // determinants
    size_t nsh = 0;   // n_stored_h of the pending build
    int n_up = 0, n_dn = 0;
    uint64_t* d_up = nullptr;    // SoA [W][N]
    uint64_t* d_dn = nullptr;    // SoA [W][N]
    uint64_t* d_up_b = nullptr;  // alpha strings in beta-group order, SoA [W][N]
    int32_t* d_orig = nullptr;   // internal -> caller index
    int32_t* d_inv = nullptr;    // caller -> internal index
    double* d_diag = nullptr;    // H_ii, internal order

    // alpha groups over the internal order
    int32_t G_a = 0;
    int32_t* d_ga = nullptr;        // group of each det
    int32_t* d_ga_start = nullptr;  // G_a + 1
    // beta groups: order_b lists internal indices sorted by (dn, up)
    int32_t G_b = 0;
    int32_t* d_gb = nullptr;        // group of each det (internal index)
    int32_t* d_gb_start = nullptr;  // G_b + 1 (positions in order_b)
    int32_t* d_order_b = nullptr;
    int32_t* d_pos_b = nullptr;     // position of each det in order_b
    // single-excitation partners between alpha groups
    int32_t* d_pa_start = nullptr;  // G_a + 1
    int32_t* d_pa_list = nullptr;
    size_t n_pa = 0;
    // open-addressing table (alpha group, beta string) -> internal index, one-word
    // strings only (norb <= 64); 2^ht_bits slots {beta lo, beta hi, group, index},
    // index -1 = empty
    int4* d_ht = nullptr;
    int ht_bits = 0;
    bool grouped = false;  // the groups and the table above are complete (the set was accepted)

    // sparse H: both triangles, rows in internal order, diagonal separate
    int precision = -1;   // value storage: FP64, FP32, MIXED, COLS or MATRIX_FREE
    bool upper = false;   // only pairs with q > p (internal order) are stored
    bool built = false;
    int64_t* d_row_start = nullptr;  // N + 1 (segment starts; capacity per row)
    int32_t* d_row_len = nullptr;    // stored elements per row
    int32_t* d_cols = nullptr;
    double* d_val64 = nullptr;
    float* d_val32 = nullptr;
    float* d_val_lo = nullptr;  // FP64 - FP32 remainder (MIXED)
    size_t cap = 0;             // allocated element slots
    uint64_t nnz_full = 0;
    uint64_t nnz_upper = 0;
    // matrix-free storage: the sigma's row counter and the builder's singles threshold
    int* d_mf_counter = nullptr;
    double mf_thr = 0.0;

    // Tiled upper-triangle storage (upper builds), see tiles.cu.  Rows are cut into panels
    // of 2^tile_rb consecutive rows and columns into windows of 2^tile_cb; panels into
    // blocks of 2^tile_kb rows.  A dense (panel, window) tile holds its blocks' rows in
    // groups of 32; the pairs of sparse tiles are the panel's leftovers.
    bool tiled = false;
    bool tile_list = false;           // as pair lists, see tiles_list.cuh
    int tile_rb = 0, tile_cb = 0, tile_kb = 0;
    int64_t n_panels = 0;
    int64_t n_tiles = 0;
    uint64_t n_dense_el = 0;          // stored pairs in dense tiles
    int64_t* d_panel_tile = nullptr;  // n_panels + 1: first tile of each panel
    int64_t n_units = 0;              // sigma work units, large ones first
    risq::SigmaUnit* d_units = nullptr;
    int32_t* d_tile_win = nullptr;    // window of each tile
    int32_t* d_tile_blk = nullptr;    // n_tiles + 1: first block record of each tile
    float2* d_tile_bound = nullptr;   // largest row sum of |H| in each tile, bound on its column sums
    risq::TileBlock* d_tile_blocks = nullptr;
    int64_t* d_tile_off = nullptr;    // pair lists: first pair and pairs of each tile; the codes,
    int32_t* d_tile_len = nullptr;    // a panel's leftovers after its tiles (values: d_val64, ...)
    uint32_t* d_el_idx = nullptr;
    std::vector<risq::TileChunk> chunks;  // the element arrays, chunk of panels by chunk
    risq::TileChunk* d_chunk_tab = nullptr;
    int64_t* d_left_off = nullptr;    // per panel: first leftover, their number; then their
    int32_t* d_left_len = nullptr;    // columns, rows in the panel and values
    uint32_t* d_left_col = nullptr;
    uint16_t* d_left_row = nullptr;
    float* d_left32 = nullptr;
    float* d_left_lo = nullptr;
    int64_t* d_row_left = nullptr;    // FP64 values: N, first leftover of each row (columns in
    int32_t* d_row_nleft = nullptr;   // d_left_col), and their number
    double* d_left64 = nullptr;
    double h_row_abs_max = 0.0;       // bound on sum_q |H_pq| (both triangles) of any row, for the fixed-point scale
    // sigma work space, allocated with the matrix: the accumulator (N int64; FP32 values: N
    // more, row sums from entry (N + 1) / 2 on, where the columns are summed in FP32), max |x| per
    // run of entries, and the scalars of k_sigma_prep
    long long* d_acc = nullptr;
    double* d_wmax = nullptr;
    double* d_sig_scalars = nullptr;

    // Row-block partition for several GPUs (risqgpu_set_partition): this handle builds
    // and applies the row panels [part_p_lo, part_p_hi) of the tiled layout; partial
    // sums are added across the ranks by the caller's all-reduce.
    bool reproducible = false;  // FP32 sigma in fixed point too (risqgpu_set_reproducible)
    int part_rank = 0, part_n = 1;
    risqgpu_allreduce_fn part_reduce = nullptr;
    void* part_user = nullptr;
    unsigned long long* d_agree = nullptr;  // while a partitioned build runs: see part_agree
    int64_t part_p_lo = 0, part_p_hi = 0;

    // previous build kept for an incremental extension
    size_t prev_N = 0;
    int32_t* d_prev_orig = nullptr;
    int64_t* d_prev_row_start = nullptr;
    int32_t* d_prev_row_len = nullptr;
    int32_t* d_prev_cols = nullptr;
    double* d_prev_val64 = nullptr;
    float* d_prev_val32 = nullptr;
    float* d_prev_val_lo = nullptr;
    int prev_precision = -1;

    // host copy of the caller-order determinants (incremental prefix check)
    std::vector<uint64_t> h_dets;

    risq::MlpWeights mlp;
    // Davidson search space and restart size (0 = the reference's nroots + 10 and nroots)
    int dav_space = 0;
    int dav_keep = 0;

    // large blocks of a matrix that went, for the build that follows; whether freed ones join
    // them; and whether large buffers take no more than they need
    std::vector<std::pair<void*, size_t>> parked;
    bool parking = false;
    bool exact = false;

    // page-locked results of a Davidson iteration, and the device flag that a sigma looks at
    // before it starts (null, or set by a solve that has ended)
    double* pinned = nullptr;
    const int* stop_flag = nullptr;

    // variational wavefunction of the last risqgpu_variational run (caller order)
    std::vector<uint64_t> wf_dets;
    std::vector<double> wf_coeffs, wf_diag;
    double wf_energy = 0.0;
    std::vector<risqgpu_var_iter> var_log;
    // result of the last risqgpu_find_new_dets
    std::vector<uint64_t> pend_dets;
    std::vector<double> pend_diag;
};

namespace risq {

// Make the handle's device current for the duration of a call.
struct DeviceGuard {
    int prev = -1;
    explicit DeviceGuard(int dev) {
        cudaGetDevice(&prev);
        if (prev != dev) cudaSetDevice(dev);
    }
    ~DeviceGuard() {
        int cur = -1;
        cudaGetDevice(&cur);
        if (prev >= 0 && cur != prev) cudaSetDevice(prev);
    }
};

// Device memory of the handles.  Every buffer comes from dalloc and goes back through
// dfree; a ledger records each one's handle and size (mem_used, with what a block is larger
// than was asked for).  A handle without a memory bound takes its buffers from memory that
// the process keeps per device (capi.cu): a build or a solve makes and drops 50 to 90 buffers,
// and with cudaMalloc / cudaFree those cost more than its kernels (131,611 determinants:
// 11.4 ms of a 20 ms build; 551,147: 49 of 113 ms).  At most POOL_KEEP bytes of idle large
// blocks (a sixteenth of the device) and a pool of at most SMALL_KEEP bytes, or what is in
// use of it, are kept; all are given back when the last handle on the device goes, when a
// caller asks (risqgpu_release_memory), and before any allocation is reported as failed.  A
// handle with a memory bound allocates from the device directly, so that what it holds is
// what its bound counts.
//
// The large blocks of a matrix that goes because another set or build follows stay with the
// handle (`parked`) until that build returns: unmapping and mapping them again took from 0.1
// to 2.5 s for 120 GB on a host whose GPUs are shared.
constexpr size_t POOL_KEEP = (size_t)6 << 30, SMALL_KEEP = (size_t)2 << 30;
int mem_alloc(risqgpu* h, void** p, size_t bytes, bool device = false);  // RISQGPU status; sets h->err
void mem_free(void* p);
void drop_parked(risqgpu* h, bool reuse);  // to the idle blocks, or to the device
int pool_acquire(int device);  // one call per handle made on the device
void pool_release(int device);  // one call per handle destroyed, after its buffers
void pool_trim(int device);
size_t pool_idle(int device);  // idle bytes kept

// While it lives, large blocks that the handle frees are parked.
struct Parking {
    risqgpu* h;
    explicit Parking(risqgpu* h_) : h(h_) { h->parking = true; }
    ~Parking() { h->parking = false; }
};

// Free a device pointer (ignores null) and reset it.  Stream-ordered: work already issued
// on the handle's stream may still use the buffer.
template <typename T>
inline void dfree(T*& p) {
    if (p) mem_free((void*)p);
    p = nullptr;
}

template <typename T>
inline int dalloc(risqgpu* h, T*& p, size_t count) {
    dfree(p);
    if (count == 0) count = 1;
    return mem_alloc(h, (void**)&p, count * sizeof(T));
}

// A buffer that the ranks' reduce function is given: with a partition from cudaMalloc, since a
// caller's own all-reduce may open it in another process or reach it from another GPU, which
// memory of a private pool does not allow.
template <typename T>
inline int dalloc_reduced(risqgpu* h, T*& p, size_t count) {
    dfree(p);
    return mem_alloc(h, (void**)&p, (count ? count : 1) * sizeof(T), h->part_n > 1);
}

// Device bytes that new allocations may take: free device memory and what is kept idle or
// parked, bounded by the handle's limit.  The device is asked only when the latter does not
// cover `need`: on a host whose GPUs are shared cudaMemGetInfo was seen to take from 0.1 to
// 75 ms (a build of 551,147 determinants: 47 ms).
inline size_t mem_available(risqgpu* h, size_t need) {
    size_t idle = pool_idle(h->device);
    for (const auto& b : h->parked) idle += b.second;
    if (!h->mem_limit && idle >= need) return idle;
    size_t fr = 0, tot = 0;
    if (cudaMemGetInfo(&fr, &tot) != cudaSuccess) {
        cudaGetLastError();
        fr = 0;
    }
    fr += idle;
    if (h->mem_limit) fr = std::min(fr, h->mem_limit > h->mem_used ? h->mem_limit - h->mem_used : (size_t)0);
    return fr;
}

// Frees the device pointers it was given when it goes out of scope, so that every
// early return of a function releases its work buffers.
template <int K>
struct ScopedFree {
    void** slots[K];
    template <typename... T>
    explicit ScopedFree(T*&... p) : slots{reinterpret_cast<void**>(&p)...} {
        static_assert(sizeof...(T) == K, "ScopedFree<K> takes K pointers");
    }
    ~ScopedFree() {
        for (void** s : slots) dfree(*s);
    }
    ScopedFree(const ScopedFree&) = delete;
    ScopedFree& operator=(const ScopedFree&) = delete;
};

// Lets a kernel take `bytes` of dynamic shared memory.  The permission belongs to the kernel, in
// the whole process: it is always the device's most, so that a thread with a smaller set does
// not take it from another between that one's call and its launch.
template <typename K>
inline int allow_smem(risqgpu* h, K kern, size_t bytes) {
    if (bytes <= ((size_t)40 << 10)) return RISQGPU_OK;  // needs none (48 KB with the static part)
    cudaFuncAttributes a;
    int most = 0;
    cudaError_t e = cudaFuncGetAttributes(&a, kern);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, h->device);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)a.sharedSizeBytes);
    if (e != cudaSuccess) {
        cudaGetLastError();
        h->err = std::string("shared memory of a kernel: ") + cudaGetErrorString(e);
        return RISQGPU_ERR_CUDA;
    }
    return RISQGPU_OK;
}

inline int check_launch(risqgpu* h, const char* what) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        h->err = std::string(what) + ": " + cudaGetErrorString(e);
        return RISQGPU_ERR_CUDA;
    }
    return RISQGPU_OK;
}

inline int sync(risqgpu* h, const char* what) {
    cudaError_t e = cudaStreamSynchronize(h->stream);
    if (e != cudaSuccess) {
        h->err = std::string(what) + ": " + cudaGetErrorString(e);
        return RISQGPU_ERR_CUDA;
    }
    return RISQGPU_OK;
}

inline int num_sms(risqgpu* h) {
    int v = 148;
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, h->device);
    return v;
}

// builder pieces (build_h.cu)
int set_dets_impl(risqgpu* h, const uint64_t* dets, size_t n, size_t nsh, const double* diag);
int build_h_impl(risqgpu* h, int precision, int builder, risqgpu_hstats* st);
int export_upper_impl(risqgpu* h, int64_t* rowptr, int64_t* cols, double* vals, size_t cap, double* diag);
int ham_elements_impl(risqgpu* h, const uint64_t* d1, const uint64_t* d2, size_t n, double* out, bool diag_only);
void free_csr(risqgpu* h);
void free_dets(risqgpu* h);

// sigma (sigma.cu).  kind: 0 = FP64 values (or FP32 hi + lo in MIXED storage) on
// FP64 vectors, 1 = FP32 values on FP32 vectors.
int sigma_device(risqgpu* h, const void* x, void* y, int kind);
int sigma_host(risqgpu* h, const double* x, double* y, int nvec);
// One FP64 vector between the caller's determinant order and the internal (sorted)
// order, on the handle's stream: xi[p] = x[orig[p]] / y[orig[p]] = yi[p].
int permute_in(risqgpu* h, const double* x, double* xi);
int permute_out(risqgpu* h, const double* yi, double* y);

// tiled upper-triangle storage (tiles.cu)
int tile_shape(int64_t N, int& rb, int& cb, int& kb);
int tile_shape64(int64_t N, int64_t pairs, int& rb, int& cb);
int tile_shape_list(int64_t N, int& rb, int& cb);
int sigma_tiles(risqgpu* h, const void* x, void* y, int kind);
// FP64 sigma of a matrix-free build (build_h.cu), internal order
int sigma_matrix_free(risqgpu* h, const double* x, double* y);
// Sum `count` int64 values in place across the partition's ranks (the caller's all-reduce,
// on the handle's stream).
int part_allreduce(risqgpu* h, void* buf_dev, size_t count);
// The ranks' common result of a step that each took for itself: out of memory anywhere is
// out of memory everywhere, so that all go on to the same collectives.
int part_agree(risqgpu* h, int rc);
int tiles_coo(risqgpu* h, int32_t* p, int32_t* q, double* v);
int tiles_self_energy(risqgpu* h, double energy, double gmin, double* out);
int tiles_rows(risqgpu* h, const uint32_t* mark, int64_t* out_r, int64_t* out_c, double* out_v,
               unsigned long long* count, unsigned long long cap);
int export_rows_impl(risqgpu* h, const int64_t* rows, size_t k, int64_t* out_r, int64_t* out_c, double* out_v,
                     size_t cap, size_t* count);
void free_tiles(risqgpu* h);
// Turns the bins that a build's search pass counted and its fill pass filled, chunk by
// chunk of whole panels, into the tiled arrays.
struct TileBuilder {
    risqgpu* h = nullptr;
    int64_t n_blocks = 0;
    std::vector<PanelCount> counts;                 // per panel, by candidates
    std::vector<PanelBase> base;                    // per panel, and the end
    unsigned long long* left_cur = nullptr;         // per panel: next leftover
    unsigned long long* sums = nullptr;             // row bounds per panel, column bounds per window
    unsigned long long* counters = nullptr;
    std::vector<int32_t> panel_chunk;
    int64_t left = 0;                               // leftovers there is room for
    int64_t stored = 0;                             // pairs, after finish
    int plan(risqgpu* h, const uint32_t* hist, const int64_t* bin_off, int64_t n_blocks);
    int begin(int64_t p_lo, int64_t p_hi, int precision, const uint32_t* hist, const int64_t* bin_off,
              unsigned long long* cur);
    int chunk(int64_t p_lo, int64_t p_hi, int64_t chunk_el0, const unsigned long long* cur, const uint32_t* code,
              const float* vin, const float* lin);
    int finish();
    int make_units();
    ~TileBuilder();
};

// The FP64 upper triangle's conversion, from CSR rows, chunk by chunk of whole panels.
struct Tiles64Builder {
    risqgpu* h = nullptr;
    unsigned long long* row_abs = nullptr;          // N: sum_q |H_pq| over both triangles, units of 2^-32
    unsigned long long* absmax = nullptr;
    unsigned long long* counters = nullptr;
    struct Chunk {                                  // what a chunk of panels adds to the arrays
        int64_t p_lo, p_hi, tiles, left;
        TileBlock* blocks;
        int32_t* win;
        float2* bound;
        uint32_t* lcol;
        double* lval;
    };
    std::vector<Chunk> parts;
    std::vector<int64_t> panel_tile;
    int64_t tiles = 0, left = 0, stored = 0;
    int begin(risqgpu* h);
    int chunk(int64_t p_lo, int64_t p_hi, const int64_t* row_start, int64_t base, const int32_t* row_len,
              const int32_t* cols, const double* vin, uint32_t* code, double* val, int64_t cap);
    int gather();
    int finish();
    ~Tiles64Builder();
};

// The upper triangle as pair lists (tiles_list.cuh), from CSR rows, chunk by chunk of panels.
struct TileListBuilder {
    risqgpu* h = nullptr;
    int precision = 0;
    unsigned long long* row_abs = nullptr;          // N: sum_q |H_pq| over both triangles, units of 2^-32
    unsigned long long* absmax = nullptr;
    struct Part {                                   // the tiles of a chunk
        int64_t tiles;
        int32_t* win;
        int64_t* off;
        int32_t* len;
        float2* bound;
    };
    std::vector<Part> parts;
    std::vector<int64_t> panel_tile;
    int64_t tiles = 0, dense = 0, stored = 0, cap = 0;
    int begin(risqgpu* h, int precision, int64_t cap);
    int chunk(int64_t p_lo, int64_t p_hi, const int64_t* row_start, int64_t base, const int32_t* row_len,
              const int32_t* cols, const double* v64, const float* v32, const float* vlo);
    int gather();
    int finish();
    ~TileListBuilder();
};

// davidson (davidson.cu)
int davidson_impl(risqgpu* h, int nroots, const double* init, int ninit, double tol, double etol, int max_iter,
                  int mode, int precond, double* evals, double* evecs, risqgpu_dstats* st);
int set_mlp_impl(risqgpu* h, int n_in, int hidden, const float* w1, const float* b1, const float* w2,
                 const float* b2, const float* w3, const float* b3, const float* feat_norm);
void free_mlp(risqgpu* h);
int precond_factors_impl(risqgpu* h, double energy, float* out);
int self_energy_impl(risqgpu* h, double energy, double gmin, double* out);

}  // namespace risq
