// HCI selection on the device: find_new_dets / iterate_excites (src/wf/mod.rs:1418-1631).
//
// The reference walks the determinants in order and, for each, the heat-bath
// sorted excitation lists (src/excite/init.rs:81-280) until |H| < eps / |c|,
// pushing every excited determinant that is not yet in the variational space
// or in the output (first occurrence wins, with the diagonal updated from that
// parent, src/wf/det.rs:271-420), and finally push_and_spin_flipped's each new
// determinant (src/wf/mod.rs:99-116).  Here one warp expands one determinant;
// the candidates of each determinant are written at a prefix-sum offset in the
// same order the reference visits them, so a candidate's index in the buffer is
// its position in the reference's sequence.  "First occurrence wins" then
// becomes a stable sort by configuration keeping the first of each run, and the
// spin-flip pushes become a second stable unique over [flip(d), d] pairs.
// Membership in the current space goes through the handle's determinant table.
#include <cub/cub.cuh>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "bits.cuh"
#include "det_table.cuh"
#include "internal.cuh"
#include "select.cuh"

namespace risq {

namespace {

constexpr unsigned FULL = 0xffffffffu;

inline int grid_of(risqgpu* h, int64_t n, int block = 256) {
    int64_t g = (n + block - 1) / block;
    int64_t cap = (int64_t)num_sms(h) * 16;
    return (int)std::max<int64_t>(1, std::min(g, cap));
}

// Membership in the handle's determinant set, which is sorted by (up, dn).  One-word
// strings: the alpha string's group by binary search over the unique alpha strings, then
// one probe of the determinant table (most excited strings are in no group, which ends the
// test there); two-word strings, and sets without groups (`alpha` null: the set was refused
// after it was sorted): binary search over the determinants.
template <int W>
struct SortedSet {
    const uint64_t* __restrict__ up;
    const uint64_t* __restrict__ dn;
    int64_t N;
    const uint64_t* __restrict__ alpha;  // unique alpha strings, ascending (one-word strings), or null
    int32_t G;
    DetTable table;
    // lexicographic compare of (up, dn) with the most significant word of up first
    __device__ __forceinline__ int cmp(int64_t p, const Bits<W>& a, const Bits<W>& b) const {
#pragma unroll
        for (int k = W - 1; k >= 0; k--) {
            uint64_t x = __ldg(up + k * N + p);
            if (x != a.w[k]) return x < a.w[k] ? -1 : 1;
        }
#pragma unroll
        for (int k = W - 1; k >= 0; k--) {
            uint64_t x = __ldg(dn + k * N + p);
            if (x != b.w[k]) return x < b.w[k] ? -1 : 1;
        }
        return 0;
    }
    // group of an alpha string, -1 if the set has none
    __device__ __forceinline__ int group(uint64_t a) const {
        int lo = 0, hi = G;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            const uint64_t x = __ldg(alpha + mid);
            if (x == a) return mid;
            if (x < a) lo = mid + 1;
            else hi = mid;
        }
        return -1;
    }
    __device__ __forceinline__ bool contains(const Bits<W>& a, const Bits<W>& b) const {
        if (W == 1 && alpha) {
            const int g = group(a.w[0]);
            return g >= 0 && table.find(g, b.w[0]) >= 0;
        }
        int64_t lo = 0, hi = N;
        while (lo < hi) {
            int64_t mid = (lo + hi) >> 1;
            int c = cmp(mid, a, b);
            if (c == 0) return true;
            if (c < 0) lo = mid + 1;
            else hi = mid;
        }
        return false;
    }
};

__global__ void k_unique_alpha(const uint64_t* __restrict__ up, const int32_t* __restrict__ ga_start, int32_t G,
                               uint64_t* __restrict__ alpha) {
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < G; g += gridDim.x * blockDim.x) alpha[g] = up[ga_start[g]];
}

struct Tables {  // heat-bath lists on the device (see select.cuh)
    const int32_t* __restrict__ opp_off;   // n*n + 1
    const int32_t* __restrict__ same_off;  // n*n + 1
    const int32_t* __restrict__ sing_off;  // n + 1
    const uint8_t* __restrict__ r;
    const uint8_t* __restrict__ s;
    const double* __restrict__ habs;
    int norb;
    double max_opp, max_same, max_sing;
};

// Excitation codes: kind (0 opp, 1 same-up, 2 same-dn, 3 single-up, 4 single-dn) in
// bits 28..30 and four 7-bit orbitals i, j, r, s.
__device__ __forceinline__ uint32_t ecode(int kind, int i, int j, int r, int s) {
    return ((uint32_t)kind << 28) | ((uint32_t)i << 21) | ((uint32_t)j << 14) | ((uint32_t)r << 7) | (uint32_t)s;
}

// One warp per determinant (caller order).  FILL = false: count the candidates of each
// determinant; FILL = true: write them at off[d].  Lane l looks at the head of list
// c0 + l, and the warp then goes through each list that has an entry above eps, 32
// consecutive entries at a time, so that loads and tests are shared by the lanes (a list
// per lane read its entries uncoalesced and waited for the longest: 3.3 ms for the fill of
// 30,011 determinants at eps 1e-3, against 0.9 here).  Candidates keep the order in which
// the reference visits them: by list, then by entry.
template <int W, bool FILL>
__global__ void __launch_bounds__(256) k_expand(const uint64_t* __restrict__ aos, const double* __restrict__ coeff,
                                                int64_t N, double eps, int singles_on, Tables T, Bits<W> valence,
                                                Ints I, SortedSet<W> set, int* __restrict__ row_counter,
                                                int64_t* __restrict__ cnt, const int64_t* __restrict__ off,
                                                uint64_t* __restrict__ out_cfg, int32_t* __restrict__ out_parent,
                                                uint32_t* __restrict__ out_code, int64_t M, int cache) {
    // cache: entries per warp for the alpha groups of this determinant's single excitations
    // (i-th valence electron, orbital), looked up when first met; 0 when they do not fit
    extern __shared__ int32_t s_group[];
    int32_t* const my_group = s_group + (threadIdx.x >> 5) * cache;
    const int lane = threadIdx.x & 31;
    const int n = T.norb;
    for (;;) {
        int d = 0;
        if (lane == 0) d = atomicAdd(row_counter, 1);
        d = __shfl_sync(FULL, d, 0);
        if (d >= N) break;
        Bits<W> up, dn;
#pragma unroll
        for (int k = 0; k < W; k++) { up.w[k] = aos[(int64_t)d * 4 + k]; dn.w[k] = aos[(int64_t)d * 4 + 2 + k]; }
        const double local_eps = eps / fabs(coeff[d]);
        const int64_t base = FILL ? off[d] : 0;
        int64_t count = 0;
        int own_group = -1;  // this determinant's alpha group
        if (W == 1 && set.alpha) own_group = set.group(up.w[0]);

        // One list [lo, hi): test(r, s, a2, b2) says whether the entry is a candidate and
        // fills in its strings.
        auto walk = [&](int lo, int hi, uint32_t code0, auto&& test) {
            for (int k0 = lo; k0 < hi; k0 += 32) {
                const int k = k0 + lane;
                const bool above = k < hi && !(T.habs[k] < local_eps);
                int r = 0, s = 0;
                Bits<W> a2, b2;
                bool keep = false;
                if (above) {
                    r = T.r[k];
                    s = T.s[k];
                    keep = test(r, s, a2, b2);
                }
                const unsigned m = __ballot_sync(FULL, keep);
                if (FILL && keep) {
                    const int64_t pos = base + count + __popc(m & ((1u << lane) - 1u));
#pragma unroll
                    for (int q = 0; q < W; q++) {
                        out_cfg[q * M + pos] = a2.w[q];
                        out_cfg[(W + q) * M + pos] = b2.w[q];
                    }
                    out_parent[pos] = d;
                    out_code[pos] = code0 | ((uint32_t)r << 7) | (uint32_t)s;
                }
                count += __popc(m);
                if (!__all_sync(FULL, above)) break;
            }
        };

        // (1) opposite-spin doubles (mod.rs:1487-1534)
        if (T.max_opp >= local_eps) {
            const Bits<W> vu = up & valence, vd = dn & valence;
            const int nu = vu.popc(), nd = vd.popc();
            const int npair = nu * nd;
            __syncwarp();
            if (W == 1 && cache)
                for (int k = lane; k < nu * n; k += 32) my_group[k] = -2;
            __syncwarp();
            for (int c0 = 0; c0 < npair; c0 += 32) {
                const int pidx = c0 + lane;
                int i = 0, j = 0, ii = 0, lo = 0, hi = 0;
                if (pidx < npair) {
                    Bits<W> t = vu;
                    ii = pidx / nd;
                    for (int k = 0; k < ii; k++) t.pop_lowest();
                    i = t.ctz();
                    Bits<W> u = vd;
                    for (int k = 0; k < pidx % nd; k++) u.pop_lowest();
                    j = u.ctz();
                    lo = T.opp_off[i * n + j];
                    hi = T.opp_off[i * n + j + 1];
                }
                unsigned todo = __ballot_sync(FULL, lo < hi && !(T.habs[lo] < local_eps));
                while (todo) {
                    const int src = __ffs(todo) - 1;
                    todo &= todo - 1;
                    const int wi = __shfl_sync(FULL, i, src), wj = __shfl_sync(FULL, j, src);
                    const int wii = __shfl_sync(FULL, ii, src);
                    walk(__shfl_sync(FULL, lo, src), __shfl_sync(FULL, hi, src), ecode(0, wi, wj, 0, 0),
                         [&](int r, int s, Bits<W>& a2, Bits<W>& b2) -> bool {
                             if (up.test(r) || dn.test(s)) return false;
                             a2 = up;
                             b2 = dn;
                             a2.clear(wi); a2.set(r);
                             b2.clear(wj); b2.set(s);
                             if (W == 1 && cache) {
                                 int g = my_group[wii * n + r];
                                 if (g == -2) my_group[wii * n + r] = g = set.group(a2.w[0]);
                                 return g < 0 || set.table.find(g, b2.w[0]) < 0;
                             }
                             return !set.contains(a2, b2);
                         });
                }
            }
        }
        // (2) same-spin doubles (mod.rs:1536-1580)
        if (T.max_same >= local_eps) {
            for (int sp = 0; sp < 2; sp++) {
                const Bits<W> x = sp == 0 ? up : dn;
                const Bits<W> vx = x & valence;
                const int nv = vx.popc();
                const int npair = nv * (nv - 1) / 2;
                for (int c0 = 0; c0 < npair; c0 += 32) {
                    const int pidx = c0 + lane;
                    int i = 0, j = 0, lo = 0, hi = 0;
                    if (pidx < npair) {
                        // bit_pairs order: (a, b) with a < b, a-major
                        int a = 0, rem = pidx;
                        while (rem >= nv - 1 - a) { rem -= nv - 1 - a; a++; }
                        int b = a + 1 + rem;
                        Bits<W> t = vx;
                        for (int k = 0; k < a; k++) t.pop_lowest();
                        i = t.ctz();
                        for (int k = a; k < b; k++) t.pop_lowest();
                        j = t.ctz();
                        lo = T.same_off[i * n + j];
                        hi = T.same_off[i * n + j + 1];
                    }
                    unsigned todo = __ballot_sync(FULL, lo < hi && !(T.habs[lo] < local_eps));
                    while (todo) {
                        const int src = __ffs(todo) - 1;
                        todo &= todo - 1;
                        const int wi = __shfl_sync(FULL, i, src), wj = __shfl_sync(FULL, j, src);
                        walk(__shfl_sync(FULL, lo, src), __shfl_sync(FULL, hi, src), ecode(1 + sp, wi, wj, 0, 0),
                             [&](int r, int s, Bits<W>& a2, Bits<W>& b2) -> bool {
                                 if (x.test(r) || x.test(s)) return false;
                                 Bits<W> nx = x;
                                 nx.clear(wi); nx.clear(wj); nx.set(r); nx.set(s);
                                 a2 = sp == 0 ? nx : up;
                                 b2 = sp == 0 ? dn : nx;
                                 if (W == 1 && set.alpha && sp == 1)
                                     return set.table.find(own_group, nx.w[0]) < 0;
                                 return !set.contains(a2, b2);
                             });
                    }
                }
            }
        }
        // (3) singles, only at the target eps (mod.rs:1582-1628)
        if (singles_on && T.max_sing >= local_eps) {
            for (int sp = 0; sp < 2; sp++) {
                const Bits<W> x = sp == 0 ? up : dn;
                const Bits<W> other = sp == 0 ? dn : up;
                Bits<W> vx = x & valence;
                while (!vx.is_zero()) {
                    const int i = vx.ctz();
                    vx.pop_lowest();
                    walk(T.sing_off[i], T.sing_off[i + 1], ecode(3 + sp, i, 0, 0, 0),
                         [&](int r, int, Bits<W>& a2, Bits<W>& b2) -> bool {
                             if (x.test(r)) return false;
                             Bits<W> nx = x;
                             nx.clear(i); nx.set(r);
                             a2 = sp == 0 ? nx : up;
                             b2 = sp == 0 ? dn : nx;
                             if (set.contains(a2, b2)) return false;
                             return fabs(sc_single<W>(I, x, nx, other)) > local_eps;
                         });
                }
            }
        }
        if (!FILL && lane == 0) cnt[d] = count;
    }
}

// Diagonal of a new determinant from its parent's (Det::new_diag_*, src/wf/det.rs:271-420).
template <int W>
__device__ double new_diag(const Ints& I, const Bits<W>& up, const Bits<W>& dn, double pdiag, uint32_t code) {
    const int kind = (code >> 28) & 7;
    const int p = (code >> 21) & 127, q = (code >> 14) & 127, r = (code >> 7) & 127, s = code & 127;
    if (kind == 0) {  // new_diag_opp
        double nd = pdiag + one_body(I, r, r) + one_body(I, s, s) - one_body(I, p, p) - one_body(I, q, q);
        nd += direct(I, r, s, r, s) - direct(I, p, q, p, q);
        Bits<W> t = up;
        while (!t.is_zero()) {
            int i = t.ctz();
            t.pop_lowest();
            if (i == p) continue;
            nd += dpe(I, i, r, i, r) - dpe(I, i, p, i, p);
            nd += direct(I, i, s, i, s) - direct(I, i, q, i, q);
        }
        t = dn;
        while (!t.is_zero()) {
            int i = t.ctz();
            t.pop_lowest();
            if (i == q) continue;
            nd += dpe(I, i, s, i, s) - dpe(I, i, q, i, q);
            nd += direct(I, i, r, i, r) - direct(I, i, p, i, p);
        }
        return nd;
    }
    if (kind == 1 || kind == 2) {  // new_diag_same
        const bool alpha = kind == 1;
        double nd = pdiag + one_body(I, r, r) + one_body(I, s, s) - one_body(I, p, p) - one_body(I, q, q);
        nd += dpe(I, r, s, r, s) - dpe(I, p, q, p, q);
        Bits<W> t = alpha ? up : dn;
        while (!t.is_zero()) {
            int i = t.ctz();
            t.pop_lowest();
            if (i == p || i == q) continue;
            nd += dpe(I, i, r, i, r) + dpe(I, i, s, i, s) - dpe(I, i, p, i, p) - dpe(I, i, q, i, q);
        }
        t = alpha ? dn : up;
        while (!t.is_zero()) {
            int i = t.ctz();
            t.pop_lowest();
            nd += direct(I, i, r, i, r) + direct(I, i, s, i, s) - direct(I, i, p, i, p) - direct(I, i, q, i, q);
        }
        return nd;
    }
    // new_diag_sing
    const bool alpha = kind == 3;
    double nd = pdiag + one_body(I, r, r) - one_body(I, p, p);
    Bits<W> t = alpha ? up : dn;
    while (!t.is_zero()) {
        int i = t.ctz();
        t.pop_lowest();
        if (i == p) continue;
        nd += dpe(I, i, r, i, r) - dpe(I, i, p, i, p);
    }
    t = alpha ? dn : up;
    while (!t.is_zero()) {
        int i = t.ctz();
        t.pop_lowest();
        nd += direct(I, i, r, i, r) - direct(I, i, p, i, p);
    }
    return nd;
}

// Kept candidate k (generation order): its diagonal, and the [flip(d), d] pair
// entries at 2k and 2k+1 (a flip equal to d is the same configuration twice).
template <int W>
__global__ void k_finish(const int64_t* __restrict__ kept, int64_t K, const uint64_t* __restrict__ cfg, int64_t M,
                         const int32_t* __restrict__ parent, const uint32_t* __restrict__ code,
                         const uint64_t* __restrict__ aos, const double* __restrict__ pdiag_caller, Ints I,
                         uint64_t* __restrict__ pair_cfg, double* __restrict__ pair_diag) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < K; k += (int64_t)gridDim.x * blockDim.x) {
        const int64_t c = kept[k];
        const int32_t par = parent[c];
        Bits<W> pu, pd, u, dd;
#pragma unroll
        for (int q = 0; q < W; q++) {
            pu.w[q] = aos[(int64_t)par * 4 + q];
            pd.w[q] = aos[(int64_t)par * 4 + 2 + q];
            u.w[q] = cfg[q * M + c];
            dd.w[q] = cfg[(W + q) * M + c];
        }
        const double dg = new_diag<W>(I, pu, pd, pdiag_caller[par], code[c]);
        const int64_t e0 = 2 * k, e1 = 2 * k + 1, L = 2 * K;
#pragma unroll
        for (int q = 0; q < W; q++) {
            pair_cfg[q * L + e0] = dd.w[q];        // flip: up <- dn
            pair_cfg[(W + q) * L + e0] = u.w[q];
            pair_cfg[q * L + e1] = u.w[q];
            pair_cfg[(W + q) * L + e1] = dd.w[q];
        }
        pair_diag[e0] = dg;
        pair_diag[e1] = dg;
    }
}

// head[t] = 1 where the sorted (by configuration) entry t starts a run
template <int W>
__global__ void k_heads(const uint64_t* __restrict__ cfg, int64_t M, const int64_t* __restrict__ perm, int64_t n,
                        int32_t* __restrict__ head) {
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
        bool same = t > 0;
        if (t > 0) {
            const int64_t a = perm[t], b = perm[t - 1];
            for (int q = 0; q < 2 * W; q++) same = same && cfg[q * M + a] == cfg[q * M + b];
        }
        head[t] = same ? 0 : 1;
    }
}

template <int W>
__global__ void k_not_in_set(const uint64_t* __restrict__ cfg, int64_t M, SortedSet<W> set,
                             int32_t* __restrict__ keep) {
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < M; t += (int64_t)gridDim.x * blockDim.x) {
        Bits<W> a, b;
        for (int q = 0; q < W; q++) { a.w[q] = cfg[q * M + t]; b.w[q] = cfg[(W + q) * M + t]; }
        keep[t] = set.contains(a, b) ? 0 : 1;
    }
}

__global__ void k_iota64(int64_t* p, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        p[i] = i;
}

__global__ void k_gather_word(const uint64_t* __restrict__ src, const int64_t* __restrict__ perm, int64_t n,
                              uint64_t* __restrict__ key) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        key[i] = src[perm[i]];
}

// Stable LSD sort of an int64 permutation by a (2W)-word configuration
// (dn words first, then up words: up is the most significant).
template <int W>
int sort_by_cfg(risqgpu* h, const uint64_t* cfg, int64_t M, int64_t* perm, int64_t n) {
    if (n <= 1) return RISQGPU_OK;
    uint64_t *k0 = nullptr, *k1 = nullptr;
    int64_t* v1 = nullptr;
    char* tmp = nullptr;
    ScopedFree<4> release(k0, k1, v1, tmp);
    RQ_TRY(dalloc(h, k0, n));
    RQ_TRY(dalloc(h, k1, n));
    RQ_TRY(dalloc(h, v1, n));
    size_t tb = 0;
    {
        cub::DoubleBuffer<uint64_t> dk(k0, k1);
        cub::DoubleBuffer<int64_t> dv(perm, v1);
        cub::DeviceRadixSort::SortPairs(nullptr, tb, dk, dv, (int)n, 0, 64, h->stream);
    }
    RQ_TRY(dalloc(h, tmp, tb));
    int64_t* cur = perm;
    int64_t* alt = v1;
    // (row of cfg, significant bits) from least to most significant: dn words, then up words
    std::vector<std::pair<int, int>> words;
    for (int k = 0; k < W; k++) words.push_back({W + k, std::min(64, h->norb - 64 * k)});
    for (int k = 0; k < W; k++) words.push_back({k, std::min(64, h->norb - 64 * k)});
    for (const auto& wb : words) {
        if (wb.second <= 0) continue;
        k_gather_word<<<grid_of(h, n), 256, 0, h->stream>>>(cfg + (int64_t)wb.first * M, cur, n, k0);
        cub::DoubleBuffer<uint64_t> dk(k0, k1);
        cub::DoubleBuffer<int64_t> dv(cur, alt);
        cub::DeviceRadixSort::SortPairs(tmp, tb, dk, dv, (int)n, 0, wb.second, h->stream);
        if (dv.Current() != cur) std::swap(cur, alt);
    }
    if (cur != perm) RQ_CUDA(h, cudaMemcpyAsync(perm, cur, sizeof(int64_t) * n, cudaMemcpyDeviceToDevice, h->stream));
    RQ_TRY(check_launch(h, "sort_by_cfg"));
    return sync(h, "sort_by_cfg");
}

// Select flagged elements of `in` (keeping order) into `out`; returns the count.
int compact_i64(risqgpu* h, const int64_t* in, const int32_t* flags, int64_t n, int64_t* out, int64_t& nout) {
    int64_t* dn = nullptr;
    char* tmp = nullptr;
    ScopedFree<2> release(dn, tmp);
    RQ_TRY(dalloc(h, dn, 1));
    size_t tb = 0;
    cub::DeviceSelect::Flagged(nullptr, tb, in, flags, out, dn, (int)n, h->stream);
    RQ_TRY(dalloc(h, tmp, tb));
    cub::DeviceSelect::Flagged(tmp, tb, in, flags, out, dn, (int)n, h->stream);
    RQ_CUDA(h, cudaMemcpyAsync(&nout, dn, sizeof(int64_t), cudaMemcpyDeviceToHost, h->stream));
    return sync(h, "compact");
}

int sort_i64(risqgpu* h, int64_t* keys, int64_t n) {
    if (n <= 1) return RISQGPU_OK;
    int64_t* alt = nullptr;
    char* tmp = nullptr;
    ScopedFree<2> release(alt, tmp);
    RQ_TRY(dalloc(h, alt, n));
    size_t tb = 0;
    cub::DoubleBuffer<int64_t> dk(keys, alt);
    cub::DeviceRadixSort::SortKeys(nullptr, tb, dk, (int)n, 0, 64, h->stream);
    RQ_TRY(dalloc(h, tmp, tb));
    cub::DeviceRadixSort::SortKeys(tmp, tb, dk, (int)n, 0, 64, h->stream);
    if (dk.Current() != keys) RQ_CUDA(h, cudaMemcpyAsync(keys, dk.Current(), sizeof(int64_t) * n, cudaMemcpyDeviceToDevice, h->stream));
    return sync(h, "sort_i64");
}

// Unique by configuration keeping the smallest index: `idx` (n entries, values
// index cfg columns) in increasing order on entry; on return the kept indices in
// increasing order and their count.
template <int W>
int unique_first(risqgpu* h, const uint64_t* cfg, int64_t M, int64_t* idx, int64_t n, int64_t& nk) {
    RQ_TRY(sort_by_cfg<W>(h, cfg, M, idx, n));
    int32_t* head = nullptr;
    int64_t* out = nullptr;
    ScopedFree<2> release(head, out);
    RQ_TRY(dalloc(h, head, n));
    RQ_TRY(dalloc(h, out, n));
    k_heads<W><<<grid_of(h, n), 256, 0, h->stream>>>(cfg, M, idx, n, head);
    RQ_TRY(check_launch(h, "heads"));
    RQ_TRY(compact_i64(h, idx, head, n, out, nk));
    RQ_TRY(sort_i64(h, out, nk));
    RQ_CUDA(h, cudaMemcpyAsync(idx, out, sizeof(int64_t) * nk, cudaMemcpyDeviceToDevice, h->stream));
    return sync(h, "unique");
}

__global__ void k_gather_out(const int64_t* __restrict__ idx, int64_t K, const uint64_t* __restrict__ cfg, int64_t L,
                             const double* __restrict__ dg, int W, uint64_t* __restrict__ aos,
                             double* __restrict__ dout) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < K; k += (int64_t)gridDim.x * blockDim.x) {
        const int64_t e = idx[k];
        for (int q = 0; q < 2; q++) {
            aos[k * 4 + q] = q < W ? cfg[q * L + e] : 0ull;
            aos[k * 4 + 2 + q] = q < W ? cfg[(W + q) * L + e] : 0ull;
        }
        dout[k] = dg[e];
    }
}

template <int W>
int find_new_impl(risqgpu* h, const double* coeffs, double eps, bool singles, const SelectTables& tab,
                  std::vector<uint64_t>& new_dets, std::vector<double>& new_diag, SelectStats* st, bool groups) {
    const int64_t N = (int64_t)h->N;
    new_dets.clear();
    new_diag.clear();
    // caller-order determinants, coefficients and diagonals on the device
    uint64_t* aos = nullptr;
    double *cf = nullptr, *dgc = nullptr;
    ScopedFree<3> release(aos, cf, dgc);
    RQ_TRY(dalloc(h, aos, 4 * N));
    RQ_TRY(dalloc(h, cf, N));
    RQ_TRY(dalloc(h, dgc, N));
    RQ_CUDA(h, cudaMemcpyAsync(aos, h->h_dets.data(), sizeof(uint64_t) * 4 * N, cudaMemcpyHostToDevice, h->stream));
    RQ_CUDA(h, cudaMemcpyAsync(cf, coeffs, sizeof(double) * N, cudaMemcpyHostToDevice, h->stream));
    RQ_TRY(permute_out(h, h->d_diag, dgc));
    // tables: on the device already, or brought there for this call
    int32_t *oo = nullptr, *so = nullptr, *go = nullptr;
    uint8_t *tr = nullptr, *ts = nullptr;
    double* th = nullptr;
    uint64_t* alpha = nullptr;
    ScopedFree<7> release_tables(oo, so, go, tr, ts, th, alpha);
    RQ_TRY(dalloc(h, oo, tab.opp_off.size()));
    RQ_TRY(dalloc(h, so, tab.same_off.size()));
    RQ_TRY(dalloc(h, go, tab.sing_off.size()));
    RQ_CUDA(h, cudaMemcpyAsync(oo, tab.opp_off.data(), 4 * tab.opp_off.size(), cudaMemcpyHostToDevice, h->stream));
    RQ_CUDA(h, cudaMemcpyAsync(so, tab.same_off.data(), 4 * tab.same_off.size(), cudaMemcpyHostToDevice, h->stream));
    RQ_CUDA(h, cudaMemcpyAsync(go, tab.sing_off.data(), 4 * tab.sing_off.size(), cudaMemcpyHostToDevice, h->stream));
    if (!tab.d_habs) {
        RQ_TRY(dalloc(h, tr, tab.r.size()));
        RQ_TRY(dalloc(h, ts, tab.s.size()));
        RQ_TRY(dalloc(h, th, tab.habs.size()));
        RQ_CUDA(h, cudaMemcpyAsync(tr, tab.r.data(), tab.r.size(), cudaMemcpyHostToDevice, h->stream));
        RQ_CUDA(h, cudaMemcpyAsync(ts, tab.s.data(), tab.s.size(), cudaMemcpyHostToDevice, h->stream));
        RQ_CUDA(h, cudaMemcpyAsync(th, tab.habs.data(), 8 * tab.habs.size(), cudaMemcpyHostToDevice, h->stream));
    }
    Tables T{oo, so, go, tab.d_habs ? tab.d_r : tr, tab.d_habs ? tab.d_s : ts, tab.d_habs ? tab.d_habs : th, h->norb,
             tab.max_opp, tab.max_same, tab.max_sing};
    Bits<W> val;
    for (int q = 0; q < W; q++) val.w[q] = tab.valence[q];
    Ints I{h->d_h1, h->d_h2, h->nuc};
    if (groups) {
        RQ_TRY(dalloc(h, alpha, (size_t)h->G_a));
        k_unique_alpha<<<grid_of(h, h->G_a), 256, 0, h->stream>>>(h->d_up, h->d_ga_start, h->G_a, alpha);
        RQ_TRY(check_launch(h, "unique alpha strings"));
    }
    SortedSet<W> set{h->d_up, h->d_dn, N, alpha, h->G_a, DetTable{h->d_ht, h->ht_bits}};
    // alpha groups of single excitations, per warp, when eight warps' fit 64 KiB
    int cache = groups ? h->n_up * h->norb : 0;
    if ((size_t)cache * 8 * sizeof(int32_t) > ((size_t)64 << 10)) cache = 0;
    const size_t smem = (size_t)cache * 8 * sizeof(int32_t);
    RQ_TRY((allow_smem(h, k_expand<W, false>, smem)));
    RQ_TRY((allow_smem(h, k_expand<W, true>, smem)));
    int* counter = nullptr;
    int64_t *cnt = nullptr, *off = nullptr;
    ScopedFree<3> release_counts(counter, cnt, off);
    RQ_TRY(dalloc(h, counter, 1));
    RQ_TRY(dalloc(h, cnt, N + 1));
    RQ_TRY(dalloc(h, off, N + 1));
    int occ = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_expand<W, true>, 256, smem);
    const int blocks = num_sms(h) * std::max(occ, 1);
    RQ_CUDA(h, cudaMemsetAsync(counter, 0, sizeof(int), h->stream));
    RQ_CUDA(h, cudaMemsetAsync(cnt + N, 0, sizeof(int64_t), h->stream));
    k_expand<W, false><<<blocks, 256, smem, h->stream>>>(aos, cf, N, eps, singles ? 1 : 0, T, val, I, set, counter, cnt,
                                                      nullptr, nullptr, nullptr, nullptr, 0, cache);
    RQ_TRY(check_launch(h, "expand count"));
    {
        size_t tb = 0;
        cub::DeviceScan::ExclusiveSum(nullptr, tb, cnt, off, (int)(N + 1), h->stream);
        char* tmp = nullptr;
        ScopedFree<1> release_tmp(tmp);
        RQ_TRY(dalloc(h, tmp, tb));
        cub::DeviceScan::ExclusiveSum(tmp, tb, cnt, off, (int)(N + 1), h->stream);
        RQ_TRY(sync(h, "expand scan"));
    }
    int64_t M = 0;
    RQ_CUDA(h, cudaMemcpy(&M, off + N, sizeof(int64_t), cudaMemcpyDeviceToHost));
    if (st) st->candidates = (uint64_t)M;
    if (M > 0) {
        uint64_t* cfg = nullptr;
        int32_t* parent = nullptr;
        uint32_t* code = nullptr;
        int64_t* idx = nullptr;
        uint64_t *pcfg = nullptr, *outd = nullptr;
        double *pdg = nullptr, *outg = nullptr;
        int32_t* keep = nullptr;
        int64_t *lidx = nullptr, *lkeep = nullptr;
        ScopedFree<11> release_cand(cfg, parent, code, idx, pcfg, pdg, keep, lidx, lkeep, outd, outg);
        RQ_TRY(dalloc(h, cfg, (size_t)2 * W * M));
        RQ_TRY(dalloc(h, parent, M));
        RQ_TRY(dalloc(h, code, M));
        RQ_CUDA(h, cudaMemsetAsync(counter, 0, sizeof(int), h->stream));
        k_expand<W, true><<<blocks, 256, smem, h->stream>>>(aos, cf, N, eps, singles ? 1 : 0, T, val, I, set, counter,
                                                         nullptr, off, cfg, parent, code, M, cache);
        RQ_TRY(check_launch(h, "expand fill"));
        // first occurrence of each configuration
        RQ_TRY(dalloc(h, idx, M));
        k_iota64<<<grid_of(h, M), 256, 0, h->stream>>>(idx, M);
        int64_t K = 0;
        RQ_TRY(unique_first<W>(h, cfg, M, idx, M, K));
        // diagonals and [flip(d), d] pairs
        const int64_t L = 2 * K;
        RQ_TRY(dalloc(h, pcfg, (size_t)2 * W * L));
        RQ_TRY(dalloc(h, pdg, L));
        k_finish<W><<<grid_of(h, K), 256, 0, h->stream>>>(idx, K, cfg, M, parent, code, aos, dgc, I, pcfg, pdg);
        RQ_TRY(check_launch(h, "finish"));
        dfree(cfg); dfree(parent); dfree(code); dfree(idx);
        // drop flips already in the space, then first occurrence again
        RQ_TRY(dalloc(h, keep, L));
        RQ_TRY(dalloc(h, lidx, L));
        RQ_TRY(dalloc(h, lkeep, L));
        k_not_in_set<W><<<grid_of(h, L), 256, 0, h->stream>>>(pcfg, L, set, keep);
        k_iota64<<<grid_of(h, L), 256, 0, h->stream>>>(lidx, L);
        int64_t L2 = 0;
        RQ_TRY(compact_i64(h, lidx, keep, L, lkeep, L2));
        int64_t F = 0;
        RQ_TRY(unique_first<W>(h, pcfg, L, lkeep, L2, F));
        RQ_TRY(dalloc(h, outd, 4 * std::max<int64_t>(F, 1)));
        RQ_TRY(dalloc(h, outg, std::max<int64_t>(F, 1)));
        k_gather_out<<<grid_of(h, std::max<int64_t>(F, 1)), 256, 0, h->stream>>>(lkeep, F, pcfg, L, pdg, W, outd, outg);
        RQ_TRY(check_launch(h, "gather out"));
        new_dets.resize(4 * F);
        new_diag.resize(F);
        RQ_CUDA(h, cudaMemcpyAsync(new_dets.data(), outd, sizeof(uint64_t) * 4 * F, cudaMemcpyDeviceToHost, h->stream));
        RQ_CUDA(h, cudaMemcpyAsync(new_diag.data(), outg, sizeof(double) * F, cudaMemcpyDeviceToHost, h->stream));
        RQ_TRY(sync(h, "select out"));
        if (st) { st->unique = (uint64_t)K; st->added = (uint64_t)F; }
    } else if (st) {
        st->unique = st->added = 0;
    }
    return RISQGPU_OK;
}

}  // namespace

namespace {

// |H| of the opposite-spin doubles (p, q) -> (r, s), one block per (p, q), in the
// reference's loop order: r over the valence orbitals but p, s over those but q.
__global__ void k_opp_lists(Ints I, int n, int nv, const uint8_t* __restrict__ vo, const int32_t* __restrict__ off,
                            double* __restrict__ key, uint16_t* __restrict__ rs) {
    __shared__ uint8_t vr[128], vs[128];  // the valence orbitals without p, without q
    const int p = blockIdx.x / n, q = blockIdx.x % n;
    const int m = nv - 1, lo = off[blockIdx.x], len = off[blockIdx.x + 1] - lo;
    if (len == 0) return;
    for (int k = threadIdx.x; k < nv; k += blockDim.x) {
        const int o = vo[k];
        int kp = 0, kq = 0;
        while (vo[kp] != p) kp++;
        while (vo[kq] != q) kq++;
        if (o != p) vr[k - (k > kp)] = (uint8_t)o;
        if (o != q) vs[k - (k > kq)] = (uint8_t)o;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < len; t += blockDim.x) {
        const int r = vr[t / m], s = vs[t % m];
        key[lo + t] = fabs(direct(I, p, q, r, s));
        rs[lo + t] = (uint16_t)((r << 8) | s);
    }
}

// |H| of the same-spin doubles (p < q) -> (r < s), one warp per (p, q): r, then s, over the
// valence orbitals but p and q, pairs with r >= s left out.
__global__ void k_same_lists(Ints I, int n, int nv, const uint8_t* __restrict__ vo, const int32_t* __restrict__ off,
                             double* __restrict__ key, uint16_t* __restrict__ rs) {
    const int p = blockIdx.x / n, q = blockIdx.x % n, lane = threadIdx.x;
    int at = off[blockIdx.x];
    if (off[blockIdx.x + 1] == at) return;
    for (int t0 = 0; t0 < nv * nv; t0 += 32) {
        const int t = t0 + lane;
        int r = 0, s = 0;
        bool ok = t < nv * nv;
        if (ok) {
            r = vo[t / nv];
            s = vo[t % nv];
            ok = r < s && r != p && r != q && s != p && s != q;
        }
        const unsigned m = __ballot_sync(FULL, ok);
        if (ok) {
            const int k = at + __popc(m & ((1u << lane) - 1u));
            key[k] = fabs(dpe(I, p, q, r, s));
            rs[k] = (uint16_t)((r << 8) | s);
        }
        at += __popc(m);
    }
}

__global__ void k_split_rs(const uint16_t* __restrict__ rs, int64_t n, uint8_t* __restrict__ r, uint8_t* __restrict__ s) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        r[i] = (uint8_t)(rs[i] >> 8);
        s[i] = (uint8_t)(rs[i] & 255);
    }
}

// Largest |H| of sorted lists: of their first entries.
__global__ void k_list_max(const double* __restrict__ key, const int32_t* __restrict__ off, int segs,
                           unsigned long long* __restrict__ out) {
    unsigned long long m = 0ull;  // bits of non-negative doubles order like the doubles
    for (int k = threadIdx.x; k < segs; k += blockDim.x)
        if (off[k + 1] > off[k]) m = max(m, (unsigned long long)__double_as_longlong(key[off[k]]));
    atomicMax(out, m);
}

}  // namespace

int sort_double_lists(risqgpu* h, SelectTables& t) {
    const int n = h->norb, nv = (int)t.valence_orbs.size(), segs = n * n;
    const int32_t total = t.same_off.back();
    RQ_TRY(dalloc(h, t.d_r, t.entries));
    RQ_TRY(dalloc(h, t.d_s, t.entries));
    RQ_TRY(dalloc(h, t.d_habs, t.entries));
    if (total == 0) return RISQGPU_OK;
    // list starts of both kinds in one array: the opposite-spin lists, then the same-spin ones
    std::vector<int32_t> off(t.opp_off.begin(), t.opp_off.end() - 1);
    off.insert(off.end(), t.same_off.begin(), t.same_off.end());
    std::vector<uint8_t> vo(t.valence_orbs.begin(), t.valence_orbs.end());
    int32_t* doff = nullptr;
    uint8_t* dvo = nullptr;
    double* key = nullptr;
    uint16_t *rs = nullptr, *rs2 = nullptr;
    char* tmp = nullptr;
    unsigned long long* mx = nullptr;
    ScopedFree<7> release(doff, dvo, key, rs, rs2, tmp, mx);
    RQ_TRY(dalloc(h, doff, off.size()));
    RQ_TRY(dalloc(h, dvo, vo.size()));
    RQ_TRY(dalloc(h, key, (size_t)total));
    RQ_TRY(dalloc(h, rs, (size_t)total));
    RQ_TRY(dalloc(h, rs2, (size_t)total));
    RQ_TRY(dalloc(h, mx, 2));
    RQ_CUDA(h, cudaMemcpyAsync(doff, off.data(), 4 * off.size(), cudaMemcpyHostToDevice, h->stream));
    RQ_CUDA(h, cudaMemcpyAsync(dvo, vo.data(), vo.size(), cudaMemcpyHostToDevice, h->stream));
    RQ_CUDA(h, cudaMemsetAsync(mx, 0, 16, h->stream));
    Ints I{h->d_h1, h->d_h2, h->nuc};
    k_opp_lists<<<segs, 128, 0, h->stream>>>(I, n, nv, dvo, doff, key, rs);
    k_same_lists<<<segs, 32, 0, h->stream>>>(I, n, nv, dvo, doff + segs, key, rs);
    RQ_TRY(check_launch(h, "double lists"));
    // falling |H|, equal ones in loop order
    size_t tb = 0;
    cub::DeviceSegmentedSort::StableSortPairsDescending(nullptr, tb, key, t.d_habs, rs, rs2, total, 2 * segs, doff, doff + 1,
                                                        h->stream);
    RQ_TRY(dalloc(h, tmp, tb));
    cub::DeviceSegmentedSort::StableSortPairsDescending(tmp, tb, key, t.d_habs, rs, rs2, total, 2 * segs, doff, doff + 1,
                                                        h->stream);
    k_split_rs<<<grid_of(h, total), 256, 0, h->stream>>>(rs2, total, t.d_r, t.d_s);
    k_list_max<<<1, 1024, 0, h->stream>>>(t.d_habs, doff, segs, mx);
    k_list_max<<<1, 1024, 0, h->stream>>>(t.d_habs, doff + segs, segs, mx + 1);
    RQ_TRY(check_launch(h, "sorted double lists"));
    double m[2] = {0.0, 0.0};
    RQ_CUDA(h, cudaMemcpyAsync(m, mx, 16, cudaMemcpyDeviceToHost, h->stream));
    RQ_TRY(sync(h, "double lists"));
    t.max_opp = m[0];
    t.max_same = m[1];
    return RISQGPU_OK;
}

int find_new_dets_impl(risqgpu* h, const double* coeffs, double eps, bool singles, const SelectTables& tab,
                       std::vector<uint64_t>& new_dets, std::vector<double>& new_diag, SelectStats* st) {
    if (h->N == 0 || !h->d_diag) { h->err = "no determinants set"; return RISQGPU_ERR_INVALID; }
    if (h->W != 1) return find_new_impl<2>(h, coeffs, eps, singles, tab, new_dets, new_diag, st, false);
    // a refused set has no groups, and its determinants may hold more electrons than n_up
    int rc = RISQGPU_ERR_OOM;
    if (h->grouped) rc = find_new_impl<1>(h, coeffs, eps, singles, tab, new_dets, new_diag, st, true);
    // without room for the group strings: the general search
    if (rc == RISQGPU_ERR_OOM) {
        h->err.clear();
        rc = find_new_impl<1>(h, coeffs, eps, singles, tab, new_dets, new_diag, st, false);
    }
    return rc;
}

}  // namespace risq
