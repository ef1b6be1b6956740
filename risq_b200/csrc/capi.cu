// extern "C" entry points of librisqgpu.so (declared in include/risqgpu.h).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <new>
#include <unordered_map>
#include <vector>

#include "internal.cuh"

namespace risq {

namespace {

// Where a buffer came from.  Below POOL_LARGE: the device's stream-ordered pool.  From there
// on: whole blocks, kept for reuse when they are freed, in sizes that differ by a sixteenth of
// their power of two, so that one set's matrix fits the blocks another one left; a pool that
// cuts small buffers, or the first of two large ones, from a freed matrix's hole has to map
// new memory for the rest (131,611 determinants, three handles in turn: 13 ms a build,
// against 8 here).  Those of handles with a memory bound, and what ranks reduce: the device.
enum Source { FROM_DEVICE, FROM_POOL, FROM_BLOCKS };
constexpr size_t POOL_LARGE = (size_t)64 << 20;

struct Buffer {
    risqgpu* h;
    size_t bytes;   // counted against the handle
    Source source;
    size_t held;    // of its block
};
std::mutex g_ledger_mu;
std::unordered_map<void*, Buffer> g_ledger;

struct Block {  // an idle block: free once `done` has passed on the stream it was used on
    void* p;
    size_t bytes;
    cudaEvent_t done;
};
struct Pool {
    cudaMemPool_t small = nullptr;
    std::vector<Block> blocks;  // oldest first
    size_t idle = 0;            // bytes of blocks
    size_t keep = 0;            // most of them
    int users = 0;
};
std::mutex g_pool_mu;
std::unordered_map<int, Pool> g_pools;

size_t block_size(size_t bytes) {
    size_t unit = POOL_LARGE;
    while (unit * 2 <= bytes) unit *= 2;
    unit = std::min(unit / 16, (size_t)64 << 20);
    return (bytes + unit - 1) / unit * unit;
}

// Whether a block may serve a request: at most an eighth more, or hardly any where the build
// counts on every byte.
bool fits(size_t block, size_t bytes, bool exact) {
    return block >= bytes && block - bytes <= bytes / (exact ? 64 : 8);
}

void drop_oldest(Pool& P) {  // cudaFree waits for the work that uses the block
    const Block b = P.blocks.front();
    P.blocks.erase(P.blocks.begin());
    P.idle -= b.bytes;
    cudaFree(b.p);
    cudaEventDestroy(b.done);
}

bool pool_bytes(cudaMemPool_t pool, uint64_t& reserved, uint64_t& used) {
    if (pool && cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &reserved) == cudaSuccess &&
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) == cudaSuccess)
        return true;
    cudaGetLastError();
    return false;
}

// Hands a block that work on h's stream may still use to the device's idle ones.
void keep_block(risqgpu* h, void* p, size_t bytes) {
    DeviceGuard g(h->device);
    std::lock_guard<std::mutex> lk(g_pool_mu);
    Pool& P = g_pools[h->device];
    Block k{p, bytes, nullptr};
    if (bytes > P.keep || cudaEventCreateWithFlags(&k.done, cudaEventDisableTiming) != cudaSuccess ||
        cudaEventRecord(k.done, h->stream) != cudaSuccess) {
        cudaGetLastError();
        if (k.done) cudaEventDestroy(k.done);
        cudaFree(p);
        return;
    }
    P.blocks.push_back(k);
    P.idle += bytes;
    while (P.idle > P.keep) drop_oldest(P);
}

}  // namespace

int pool_acquire(int device) {
    std::lock_guard<std::mutex> lk(g_pool_mu);
    Pool& P = g_pools[device];
    if (!P.small) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        if (cudaMemPoolCreate(&P.small, &props) != cudaSuccess) {
            cudaGetLastError();
            P.small = nullptr;
            return RISQGPU_ERR_CUDA;
        }
        // above this size the pool itself returns what is idle, at each wait
        size_t fr = 0, tot = 0;
        cudaMemGetInfo(&fr, &tot);
        uint64_t small = std::min(SMALL_KEEP, tot / 32);
        cudaMemPoolSetAttribute(P.small, cudaMemPoolAttrReleaseThreshold, &small);
        P.keep = std::min(POOL_KEEP, tot / 16);
    }
    P.users++;
    return RISQGPU_OK;
}

void pool_trim(int device) {
    std::lock_guard<std::mutex> lk(g_pool_mu);
    auto it = g_pools.find(device);
    if (it == g_pools.end()) return;
    while (!it->second.blocks.empty()) drop_oldest(it->second);
    if (it->second.small) cudaMemPoolTrimTo(it->second.small, 0);
}

void pool_release(int device) {
    bool last = false;
    {
        std::lock_guard<std::mutex> lk(g_pool_mu);
        auto it = g_pools.find(device);
        if (it != g_pools.end()) last = --it->second.users == 0;
    }
    if (last) pool_trim(device);
}

size_t pool_idle(int device) {
    std::lock_guard<std::mutex> lk(g_pool_mu);
    auto it = g_pools.find(device);
    if (it == g_pools.end()) return 0;
    uint64_t reserved = 0, used = 0;
    size_t idle = it->second.idle;
    if (pool_bytes(it->second.small, reserved, used) && reserved > used) idle += (size_t)(reserved - used);
    return idle;
}

void drop_parked(risqgpu* h, bool reuse) {
    for (const auto& b : h->parked) {
        if (reuse) keep_block(h, b.first, b.second);
        else cudaFree(b.first);
    }
    h->parked.clear();
}

int mem_alloc(risqgpu* h, void** p, size_t bytes, bool device) {
    *p = nullptr;
    if (h->mem_limit && h->mem_used + bytes > h->mem_limit) {
        h->err = "allocation of " + std::to_string(bytes) + " bytes exceeds the handle's device memory limit (" +
                 std::to_string(h->mem_used) + " of " + std::to_string(h->mem_limit) + " bytes in use)";
        return RISQGPU_ERR_OOM;
    }
    Buffer b{h, bytes, FROM_DEVICE, bytes};
    cudaMemPool_t small = nullptr;
    if (!h->mem_limit && !device) {
        b.source = bytes < POOL_LARGE ? FROM_POOL : FROM_BLOCKS;
        if (b.source == FROM_BLOCKS) {
            // the smallest block that fits: of the handle's previous matrix, then of the idle ones
            b.held = h->exact ? bytes : block_size(bytes);
            auto best = h->parked.end();
            for (auto k = h->parked.begin(); k != h->parked.end(); ++k)
                if (fits(k->second, bytes, h->exact) && (best == h->parked.end() || k->second < best->second)) best = k;
            if (best != h->parked.end()) {
                *p = best->first;
                b.held = best->second;
                h->parked.erase(best);
            }
        }
        if (!*p) {
            std::lock_guard<std::mutex> lk(g_pool_mu);
            Pool& P = g_pools[h->device];
            small = P.small;
            auto best = P.blocks.end();
            if (b.source == FROM_BLOCKS)
                for (auto k = P.blocks.begin(); k != P.blocks.end(); ++k)
                    if (fits(k->bytes, bytes, h->exact) && (best == P.blocks.end() || k->bytes < best->bytes)) best = k;
            if (best != P.blocks.end()) {
                cudaStreamWaitEvent(h->stream, best->done, 0);
                cudaEventDestroy(best->done);
                *p = best->p;
                b.held = best->bytes;
                P.idle -= best->bytes;
                P.blocks.erase(best);
            }
        }
    }
    if (!*p) {
        auto take = [&]() {
            return b.source == FROM_POOL ? cudaMallocFromPoolAsync(p, b.held, small, h->stream) : cudaMalloc(p, b.held);
        };
        cudaError_t e = take();
        if (e == cudaErrorMemoryAllocation) {
            // idle memory may be all that is missing
            cudaGetLastError();
            cudaStreamSynchronize(h->stream);
            drop_parked(h, false);
            pool_trim(h->device);
            b.held = bytes;
            e = take();
        }
        if (e != cudaSuccess) {
            *p = nullptr;
            cudaGetLastError();
            h->err = "device allocation of " + std::to_string(bytes) + " bytes: " + cudaGetErrorString(e);
            return e == cudaErrorMemoryAllocation ? RISQGPU_ERR_OOM : RISQGPU_ERR_CUDA;
        }
    }
    b.bytes = b.held;
    std::lock_guard<std::mutex> lk(g_ledger_mu);
    g_ledger[*p] = b;
    h->mem_used += b.bytes;
    return RISQGPU_OK;
}

void mem_free(void* p) {
    Buffer b;
    {
        std::lock_guard<std::mutex> lk(g_ledger_mu);
        auto it = g_ledger.find(p);
        if (it == g_ledger.end()) return;
        b = it->second;
        b.h->mem_used -= b.bytes;
        g_ledger.erase(it);
    }
    if (b.source == FROM_DEVICE) cudaFree(p);
    else if (b.source == FROM_POOL) cudaFreeAsync(p, b.h->stream);
    else if (b.h->parking) b.h->parked.emplace_back(p, b.held);
    else keep_block(b.h, p, b.held);
}

}  // namespace risq

using namespace risq;

namespace {

size_t combine_2_host(long p, long q) {
    long i = p < 0 ? -p : p, j = q < 0 ? -q : q;
    return i > j ? (size_t)((i * (i - 1)) / 2 + j) : (size_t)((j * (j - 1)) / 2 + i);
}

}  // namespace

extern "C" {

const char* risqgpu_version(void) { return "risq_b200 0.1 (sm_100a)"; }

int risqgpu_device_count(void) {
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

int risqgpu_create(int norb, const double* one_body, size_t n1, const double* two_body, size_t n2, double e_nuc,
                   int device, risqgpu_t** out) {
    if (!out) return RISQGPU_ERR_INVALID;
    *out = nullptr;
    if (norb < 1 || norb > 128 || !one_body || !two_body) return RISQGPU_ERR_INVALID;
    size_t e1 = combine_2_host(norb + 1, norb + 1);
    size_t c2n = combine_2_host(norb + 1, norb + 1);
    size_t e2 = combine_2_host((long)c2n, (long)c2n);
    if (n1 != e1 || n2 != e2) return RISQGPU_ERR_INVALID;
    int ndev = risqgpu_device_count();
    if (ndev == 0) return RISQGPU_ERR_NO_DEVICE;
    if (device < 0 || device >= ndev) return RISQGPU_ERR_INVALID;
    risqgpu* h = new (std::nothrow) risqgpu();
    if (!h) return RISQGPU_ERR_OOM;
    h->device = device;
    DeviceGuard g(device);
    h->norb = norb;
    h->W = norb > 64 ? 2 : 1;
    h->nuc = e_nuc;
    h->n1 = n1;
    h->n2 = n2;
    int rc = RISQGPU_OK;
    if (pool_acquire(device) != RISQGPU_OK) {
        delete h;
        return RISQGPU_ERR_CUDA;
    }
    if (cudaStreamCreateWithFlags(&h->own_stream, cudaStreamNonBlocking) != cudaSuccess) rc = RISQGPU_ERR_CUDA;
    h->stream = h->own_stream;
    if (!rc) rc = dalloc(h, h->d_h1, n1);
    if (!rc) rc = dalloc(h, h->d_h2, n2);
    // on the handle's stream, which the buffers belong to
    if (!rc && (cudaMemcpyAsync(h->d_h1, one_body, n1 * sizeof(double), cudaMemcpyHostToDevice, h->stream) != cudaSuccess ||
                cudaMemcpyAsync(h->d_h2, two_body, n2 * sizeof(double), cudaMemcpyHostToDevice, h->stream) != cudaSuccess ||
                cudaStreamSynchronize(h->stream) != cudaSuccess))
        rc = RISQGPU_ERR_CUDA;
    if (!rc) {
        h->h_h1.assign(one_body, one_body + n1);
        h->h_h2.assign(two_body, two_body + n2);
    }
    if (rc) {
        risqgpu_destroy(h);
        return rc;
    }
    *out = h;
    return RISQGPU_OK;
}

void risqgpu_destroy(risqgpu_t* h) {
    if (!h) return;
    DeviceGuard g(h->device);
    if (h->stream) cudaStreamSynchronize(h->stream);
    h->stream = h->own_stream;  // the frees are ordered on the handle's own stream
    free_dets(h);
    drop_parked(h, true);
    free_mlp(h);
    dfree(h->d_h1);
    dfree(h->d_h2);
    if (h->pinned) cudaFreeHost(h->pinned);
    if (h->own_stream) {
        cudaStreamSynchronize(h->own_stream);
        cudaStreamDestroy(h->own_stream);
    }
    pool_release(h->device);
    delete h;
}

const char* risqgpu_last_error(const risqgpu_t* h) { return h ? h->err.c_str() : "null handle"; }

int risqgpu_set_dets(risqgpu_t* h, const uint64_t* dets, size_t n, size_t n_stored_h, const double* diag) {
    if (!h) return RISQGPU_ERR_INVALID;
    DeviceGuard g(h->device);
    h->err.clear();
    const int rc = set_dets_impl(h, dets, n, n_stored_h, diag);
    if (rc) drop_parked(h, true);  // no build will follow
    return rc;
}

int risqgpu_build_h(risqgpu_t* h, int precision, int builder, risqgpu_hstats* stats) {
    if (!h) return RISQGPU_ERR_INVALID;
    DeviceGuard g(h->device);
    if (stats) std::memset(stats, 0, sizeof(*stats));
    return build_h_impl(h, precision, builder, stats);
}

int risqgpu_nnz(const risqgpu_t* h, uint64_t* nnz_upper, uint64_t* nnz_full) {
    if (!h) return RISQGPU_ERR_INVALID;
    if (nnz_upper) *nnz_upper = h->nnz_upper;
    if (nnz_full) *nnz_full = h->nnz_full;
    return h->built ? RISQGPU_OK : RISQGPU_ERR_INVALID;
}

int risqgpu_export_upper(risqgpu_t* h, int64_t* rowptr, int64_t* cols, double* vals, size_t cap, double* diag) {
    if (!h || !rowptr || (!cols && cap) || (!vals && cap)) return RISQGPU_ERR_INVALID;
    DeviceGuard g(h->device);
    return export_upper_impl(h, rowptr, cols, vals, cap, diag);
}

int risqgpu_export_rows(risqgpu_t* h, const int64_t* rows, size_t k, int64_t* out_row, int64_t* out_col,
                        double* out_val, size_t cap, size_t* count) {
    if (!h || !count || (k && !rows) || (cap && (!out_row || !out_col || !out_val))) return RISQGPU_ERR_INVALID;
    DeviceGuard g(h->device);
    *count = 0;
    return export_rows_impl(h, rows, k, out_row, out_col, out_val, cap, count);
}

int risqgpu_sigma(risqgpu_t* h, const double* x, double* y, int nvec) {
    if (!h || !x || !y) return RISQGPU_ERR_INVALID;
    DeviceGuard g(h->device);
    if (nvec >= 1 && h->built) {
        const size_t n = h->N * (size_t)nvec;
        for (size_t i = 0; i < n; i++)
            if (!std::isfinite(x[i])) {
                h->err = "x holds a non-finite value at index " + std::to_string(i);
                return RISQGPU_ERR_INVALID;
            }
    }
    return sigma_host(h, x, y, nvec);
}

int risqgpu_sigma_device(risqgpu_t* h, const void* x_dev, void* y_dev, int dtype) {
    if (!h || !x_dev || !y_dev || (dtype != 0 && dtype != 1)) return RISQGPU_ERR_INVALID;
    DeviceGuard g(h->device);
    int rc = sigma_device(h, x_dev, y_dev, dtype);
    if (rc) return rc;
    return sync(h, "sigma_device");
}

int risqgpu_davidson(risqgpu_t* h, int nroots, const double* init, int ninit, double tol, double etol, int max_iter,
                     int mode, int precond, double* evals, double* evecs, risqgpu_dstats* stats) {
    if (!h || !evals || max_iter < 1 || mode < 0 || mode > 2 || (precond != 0 && precond != 1))
        return RISQGPU_ERR_INVALID;
    DeviceGuard g(h->device);
    if (stats) std::memset(stats, 0, sizeof(*stats));
    return davidson_impl(h, nroots, init, ninit, tol, etol, max_iter, mode, precond, evals, evecs, stats);
}

int risqgpu_sparse_optimize(risqgpu_t* h, const double* init_coeffs, double coeff_eps, double energy_eps,
                            int max_iter, int precision, int mode, int precond, double* energy, double* coeffs,
                            risqgpu_hstats* hstats, risqgpu_dstats* dstats) {
    if (!h || !energy || !coeffs || max_iter < 1) return RISQGPU_ERR_INVALID;
    DeviceGuard g(h->device);
    if (hstats) std::memset(hstats, 0, sizeof(*hstats));
    if (dstats) std::memset(dstats, 0, sizeof(*dstats));
    int rc = build_h_impl(h, precision, RISQGPU_BUILDER_AUTO, hstats);
    if (rc) return rc;
    double e = 0.0;
    std::vector<double> v(h->N);
    rc = davidson_impl(h, 1, init_coeffs, init_coeffs ? 1 : 0, coeff_eps, energy_eps, max_iter, mode, precond, &e,
                       v.data(), dstats);
    if (rc == RISQGPU_ERR_NOT_CONVERGED) {
        h->err = "Davidson Algorithm did not converge!";
        return rc;  // energy and coefficients are left unchanged (var/davidson.rs:109-111)
    }
    if (rc) return rc;
    *energy = e;
    std::memcpy(coeffs, v.data(), sizeof(double) * h->N);
    return RISQGPU_OK;
}

int risqgpu_set_subspace(risqgpu_t* h, int max_space, int keep) {
    if (!h || max_space < 0 || keep < 0 || max_space > 56 || (max_space > 0 && keep > max_space / 2)) {
        if (h) h->err = "max_space must lie in [0, 56] and keep in [0, max_space / 2]";
        return RISQGPU_ERR_INVALID;
    }
    h->dav_space = max_space;
    h->dav_keep = keep;
    return RISQGPU_OK;
}

int risqgpu_set_partition(risqgpu_t* h, int rank, int nranks, risqgpu_allreduce_fn reduce, void* user) {
    if (!h) return RISQGPU_ERR_INVALID;
    if (nranks < 1 || rank < 0 || rank >= nranks || (nranks > 1 && !reduce)) {
        h->err = "partition needs 0 <= rank < nranks and, for nranks > 1, a reduce function";
        return RISQGPU_ERR_INVALID;
    }
    h->part_rank = rank;
    h->part_n = nranks;
    h->part_reduce = nranks > 1 ? reduce : nullptr;
    h->part_user = user;
    return RISQGPU_OK;
}

int risqgpu_set_reproducible(risqgpu_t* h, int on) {
    if (!h) return RISQGPU_ERR_INVALID;
    h->reproducible = on != 0;
    return RISQGPU_OK;
}

int risqgpu_set_memory_limit(risqgpu_t* h, size_t bytes) {
    if (!h) return RISQGPU_ERR_INVALID;
    h->mem_limit = bytes;
    if (bytes) {
        // the caller shares the device: hand back what no buffer uses
        DeviceGuard g(h->device);
        cudaStreamSynchronize(h->stream);
        drop_parked(h, false);
        pool_trim(h->device);
    }
    return RISQGPU_OK;
}

int risqgpu_memory_used(const risqgpu_t* h, size_t* used, size_t* limit) {
    if (!h) return RISQGPU_ERR_INVALID;
    if (used) *used = h->mem_used;
    if (limit) *limit = h->mem_limit;
    return RISQGPU_OK;
}

int risqgpu_release_memory(risqgpu_t* h) {
    if (!h) return RISQGPU_ERR_INVALID;
    DeviceGuard g(h->device);
    RQ_TRY(sync(h, "release memory"));
    drop_parked(h, false);
    pool_trim(h->device);
    return RISQGPU_OK;
}

int risqgpu_set_stream(risqgpu_t* h, void* stream) {
    if (!h) return RISQGPU_ERR_INVALID;
    DeviceGuard g(h->device);
    if (cudaStreamSynchronize(h->stream) != cudaSuccess) return RISQGPU_ERR_CUDA;
    h->stream = stream ? (cudaStream_t)stream : h->own_stream;
    return RISQGPU_OK;
}

int risqgpu_ham_diag(risqgpu_t* h, const uint64_t* dets, size_t n, double* out) {
    if (!h || (n && (!dets || !out))) return RISQGPU_ERR_INVALID;
    DeviceGuard g(h->device);
    return ham_elements_impl(h, dets, nullptr, n, out, true);
}

int risqgpu_ham_off_diag(risqgpu_t* h, const uint64_t* d1, const uint64_t* d2, size_t n, double* out) {
    if (!h || (n && (!d1 || !d2 || !out))) return RISQGPU_ERR_INVALID;
    DeviceGuard g(h->device);
    return ham_elements_impl(h, d1, d2, n, out, false);
}

int risqgpu_set_precond_mlp(risqgpu_t* h, int n_in, int hidden, const float* w1, const float* b1, const float* w2,
                            const float* b2, const float* w3, const float* b3, const float* feat_norm) {
    if (!h) return RISQGPU_ERR_INVALID;
    DeviceGuard g(h->device);
    return set_mlp_impl(h, n_in, hidden, w1, b1, w2, b2, w3, b3, feat_norm);
}

int risqgpu_precond_factors(risqgpu_t* h, double energy, float* out) {
    if (!h || !out) return RISQGPU_ERR_INVALID;
    DeviceGuard g(h->device);
    return precond_factors_impl(h, energy, out);
}

int risqgpu_self_energy(risqgpu_t* h, double energy, double gmin, double* out) {
    if (!h || !out) return RISQGPU_ERR_INVALID;
    DeviceGuard g(h->device);
    return self_energy_impl(h, energy, gmin, out);
}

}  // extern "C"
