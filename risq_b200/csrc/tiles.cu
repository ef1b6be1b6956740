// Tiled upper-triangle storage and its sigma.
//
// The reference's SparseMatUpperTri (src/var/sparse.rs:24-36) holds every pair
// once and its matrix_vector_prod (src/var/sparse.rs:64-78) adds each element to
// two outputs: y_p += H_pq x_q and y_q += H_pq x_p.  On the GPU the second of
// these is a scattered atomic per pair, and a gather plus a scattered atomic per
// pair bound the plain kernel by L1/L2 request throughput, not by HBM.
//
// Here rows are cut into panels of R = 2^rb consecutive rows and columns into windows of
// C = 2^cb.  A (panel, window) tile that holds enough pairs is "dense": sigma stages x of
// its window and zeroes a window of accumulators in shared memory, and one lane takes one
// row of the tile: its x_p and its row sum stay in registers, so that a pair costs one
// shared load (x_q), one shared atomic (the column sum) and 2 + s_v bytes of HBM (its
// column in the window and its value).  Rows (long ones
// in slots of 64 elements) are held in groups of 32 of falling length, two elements per
// lane and step, step after step, short ones padded with zeros to their group's length, so
// that the loads are coalesced and nearly all lanes busy.  Pairs of sparse tiles stay as leftovers, a list per panel with row and
// column of each, summed with global gathers and atomics.
//
// The build counts the candidates of every (block of 2^kb rows, window) bin in its search
// pass, and its fill pass writes each pair into its bin (build_h.cu); k_tile_arrange then
// turns every bin into groups of rows.
//
// Column windows sum in 32-bit fixed point (k_sigma_fx): each product is rounded, by a
// fixed rule, at a scale chosen per tile from the tile's largest column sum of |H| (the exact
// largest one, rounded up) and the
// largest |x| of the panel, and integer atomics are associative, so a window's sum does
// not depend on the order in which the pairs land.  The FP64 sigma (and the FP32 sigma
// when reproducible sums are asked for) sums the rows in integers too and adds all window
// and row sums in 64-bit fixed point (scale 2^s per call, from max |x| and a bound on the
// row sums of |H| over both triangles, found during the build), so two runs give
// bitwise-equal vectors.
#include <cub/cub.cuh>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "internal.cuh"
#include "tiles.cuh"

namespace risq {

namespace {

constexpr int TT = 256;   // threads per CTA of the planning kernels and of tiles_each
constexpr int AT = 512;   // threads per CTA of k_tile_arrange
constexpr int CT = 1024;  // threads per CTA of k_tile_count and k_tile_scatter
constexpr int MAX_BINS = 16384;  // windows one panel may span in those
constexpr int ST = 256;   // threads per CTA of k_sigma_fx
constexpr unsigned FULL = 0xffffffffu;
// Rows of a bin longer than this are cut into slots of this many elements, so that no group
// of 32 slots keeps one warp busy for long.
constexpr int SEG = 64;

// A tile is staged in shared memory when it holds at least max(DENSE_MIN, w >> DENSE_SHIFT)
// candidates (w = width of its window): staging w values of x, zeroing w accumulators and
// flushing them costs about as much as w >> DENSE_SHIFT scattered pairs.
constexpr int DENSE_MIN = 64;
constexpr int DENSE_SHIFT = 3;

__device__ __forceinline__ bool dense_tile(int64_t count, int w) {
    return count >= DENSE_MIN && count >= (w >> DENSE_SHIFT);
}

__device__ __forceinline__ int window_width(int64_t N, int64_t J, int cb) {
    const int64_t c0 = J << cb;
    return (int)min((int64_t)1 << cb, N - c0);
}

// ---------------------------------------------------------------- conversion

// Candidates of panel P's tile in window J, over its row blocks.
__device__ __forceinline__ int64_t tile_count(const uint32_t* __restrict__ hist, const int64_t* __restrict__ bin_off,
                                              int64_t P, int64_t J, int rb, int cb, int kb, int64_t n_blocks) {
    int64_t c = 0;
    const int64_t b0 = P << (rb - kb), b1 = min(n_blocks, (P + 1) << (rb - kb));
    for (int64_t b = b0; b < b1; b++) {
        const int64_t J0 = (b << kb) >> cb;
        if (J >= J0) c += hist[bin_off[b] + J - J0];
    }
    return c;
}

// Per panel: candidates in dense tiles, candidates left over, dense tiles, and the
// non-empty row blocks of dense tiles with about the pairs of elements and groups they need.
__global__ void __launch_bounds__(TT) k_panel_count(int64_t N, int64_t n_panels, int64_t n_blocks, int rb, int cb, int kb,
                                                    const uint32_t* __restrict__ hist,
                                                    const int64_t* __restrict__ bin_off,
                                                    PanelCount* __restrict__ out) {
    using BR = cub::BlockReduce<long long, TT>;
    __shared__ typename BR::TempStorage red;
    for (int64_t P = blockIdx.x; P < n_panels; P += gridDim.x) {
        const int64_t Jlo = (P << rb) >> cb, Jhi = ((N - 1) >> cb) + 1;
        const int64_t b0 = P << (rb - kb), b1 = min(n_blocks, (P + 1) << (rb - kb));
        long long v[6] = {0, 0, 0, 0, 0, 0};
        for (int64_t J = Jlo + threadIdx.x; J < Jhi; J += TT) {
            const int64_t c = tile_count(hist, bin_off, P, J, rb, cb, kb, n_blocks);
            if (!dense_tile(c, window_width(N, J, cb))) {
                v[1] += c;
                continue;
            }
            v[0] += c;
            v[2]++;
            for (int64_t b = b0; b < b1; b++) {
                const int64_t J0 = (b << kb) >> cb;
                const int64_t e = J >= J0 ? hist[bin_off[b] + J - J0] : 0;
                if (e == 0) continue;
                const int64_t rows = min(e, (int64_t)1 << kb);
                v[3]++;
                v[4] += (e + rows + 1) >> 1;   // pairs of elements, every row rounded up
                v[5] += (rows + e / SEG + 31) >> 5;
            }
        }
        long long t[6];
        for (int k = 0; k < 6; k++) {
            t[k] = BR(red).Sum(v[k]);
            __syncthreads();
        }
        if (threadIdx.x == 0) out[P] = PanelCount{t[0], t[1], t[2], t[3], t[4], t[5]};
    }
}

// Tiles and row blocks of the panels [p_lo, p_hi) in window order, and the fill cursor of
// every bin: where its elements start in the temporary arrays (counted from el0 of the
// panel), or LEFT_BIN for the bins of sparse tiles.
__global__ void __launch_bounds__(TT) k_panel_plan(int64_t N, int64_t p_lo, int64_t p_hi, int64_t n_blocks, int rb, int cb,
                                                   int kb, const uint32_t* __restrict__ hist,
                                                   const int64_t* __restrict__ bin_off,
                                                   const PanelBase* __restrict__ base, int32_t* __restrict__ tile_win,
                                                   int32_t* __restrict__ tile_blk, TileBlock* __restrict__ blocks,
                                                   unsigned long long* __restrict__ cur) {
    using BS = cub::BlockScan<long long, TT>;
    __shared__ typename BS::TempStorage scan;
    for (int64_t P = p_lo + blockIdx.x; P < p_hi; P += gridDim.x) {
        const int64_t Jlo = (P << rb) >> cb, Jhi = ((N - 1) >> cb) + 1;
        const int64_t b0 = P << (rb - kb), b1 = min(n_blocks, (P + 1) << (rb - kb));
        const PanelBase pb = base[P];
        const int64_t per = (Jhi - Jlo + TT - 1) / TT;
        const int64_t lo = min(Jhi, Jlo + threadIdx.x * per), hi = min(Jhi, lo + per);
        long long el = 0, nt = 0, nb = 0;
        for (int64_t J = lo; J < hi; J++) {
            const int64_t c = tile_count(hist, bin_off, P, J, rb, cb, kb, n_blocks);
            if (!dense_tile(c, window_width(N, J, cb))) continue;
            el += c;
            nt++;
            for (int64_t b = b0; b < b1; b++) {
                const int64_t J0 = (b << kb) >> cb;
                nb += J >= J0 && hist[bin_off[b] + J - J0] > 0;
            }
        }
        long long ex_el, ex_t, ex_b;
        BS(scan).ExclusiveSum(el, ex_el);
        __syncthreads();
        BS(scan).ExclusiveSum(nt, ex_t);
        __syncthreads();
        BS(scan).ExclusiveSum(nb, ex_b);
        __syncthreads();
        long long e = pb.el + ex_el, t = pb.tile + ex_t, k = pb.block + ex_b;
        for (int64_t J = lo; J < hi; J++) {
            const int64_t c = tile_count(hist, bin_off, P, J, rb, cb, kb, n_blocks);
            const bool dense = dense_tile(c, window_width(N, J, cb));
            if (dense) {
                tile_win[t] = (int32_t)J;
                tile_blk[t] = (int32_t)k;
            }
            for (int64_t b = b0; b < b1; b++) {
                const int64_t J0 = (b << kb) >> cb;
                if (J < J0) continue;
                const int64_t bin = bin_off[b] + J - J0;
                const uint32_t n = hist[bin];
                cur[bin] = dense ? (unsigned long long)e : LEFT_BIN;
                if (dense && n > 0) {
                    blocks[k].bin = bin;
                    blocks[k].el = e;
                    blocks[k].row = (int32_t)(b << kb);
                    e += n;
                    k++;
                }
            }
            if (dense) t++;
        }
    }
}

// How a bin's rows become slots: every full run of SEG elements is a slot, those first
// (row by row), then the rows' remainders by falling length.  Group g holds the slots
// 32 g .. 32 g + 31, each padded to the first one's length.
struct SlotPlan {
    int full;     // full slots
    int slots;    // all of them
    int groups;
    int vecs;     // pairs of elements, padding included
};

// Called by the whole CTA with the row lengths in cnt: fpre[r] <- first full slot of row r,
// rank[r] <- slot of its remainder; gbase[g - full / 32] <- first pair of elements of
// group g, for the groups that start with a remainder or the last full ones.
__device__ __forceinline__ SlotPlan plan_slots(const int* cnt, int B, int* fpre, int* rank, int* gbase) {
    using BS = cub::BlockScan<int, AT>;
    __shared__ typename BS::TempStorage scan;
    __shared__ int bin[SEG];      // rows by remainder, then where the next one goes
    __shared__ int first[SEG];    // first slot of each remainder length
    __shared__ SlotPlan plan;
    const int tid = threadIdx.x;
    if (tid < SEG) bin[tid] = 0;
    __syncthreads();
    int full = 0;
    for (int r0 = 0; r0 < B; r0 += AT) {
        const int r = r0 + tid, c = r < B ? cnt[r] : 0;
        int ex, sum;
        BS(scan).ExclusiveSum(c / SEG, ex, sum);
        if (r < B) {
            fpre[r] = full + ex;
            if (c % SEG) atomicAdd(bin + c % SEG, 1);
        }
        full += sum;
        __syncthreads();
    }
    if (tid == 0) {
        int s = full;
        for (int l = SEG - 1; l >= 1; l--) {
            first[l] = s;
            s += bin[l];
            bin[l] = first[l];
        }
        plan.full = full;
        plan.slots = s;
        plan.groups = (s + 31) >> 5;
        // length of each group's first slot: the longest remainder whose slots end after it
        int at = (full >> 5) * 32 * (SEG / 2), l = SEG - 1;
        for (int g = full >> 5; g < plan.groups; g++) {
            while (32 * g >= full && l > 1 && first[l - 1] <= 32 * g) l--;
            gbase[g - (full >> 5)] = at;
            at += 32 * (((32 * g < full ? SEG : l) + 1) >> 1);
        }
        plan.vecs = at;
    }
    __syncthreads();
    for (int r = tid; r < B; r += AT) {
        const int l = cnt[r] % SEG;
        rank[r] = l ? atomicAdd(bin + l, 1) : 0;
    }
    __syncthreads();
    return plan;
}

// Row lengths of every bin (its elements end at its cursor, or there are `len` of them),
// and room for its groups: counters[0] takes pairs of elements,
// [1] groups, [2] hands out the bins.
__global__ void __launch_bounds__(AT) k_tile_size(int64_t k_lo, int64_t k_hi, int rb, int cb, int kb, int64_t chunk_el0,
                                                  TileBlock* __restrict__ blocks,
                                                  const unsigned long long* __restrict__ cur,
                                                  const uint32_t* __restrict__ code, uint16_t* __restrict__ row_cnt,
                                                  unsigned long long* __restrict__ counters) {
    extern __shared__ __align__(16) unsigned char sm[];
    const int B = 1 << kb;
    int* cnt = reinterpret_cast<int*>(sm);
    int* fpre = cnt + B;
    int* rank = fpre + B;
    int* gbase = rank + B;  // B / 32 + 2
    __shared__ long long s_k;
    const int tid = threadIdx.x;
    for (;;) {
        if (tid == 0) s_k = k_lo + (long long)atomicAdd(counters + 2, 1ull);
        for (int i = tid; i < B; i += AT) cnt[i] = 0;
        __syncthreads();
        const int64_t kk = s_k;
        if (kk >= k_hi) break;
        const int64_t e0 = blocks[kk].el - chunk_el0;
        const int E = cur ? (int)((int64_t)cur[blocks[kk].bin] - blocks[kk].el) : blocks[kk].len;
        const int row0 = blocks[kk].row & ((1 << rb) - 1);
        for (int i = tid; i < E; i += AT) atomicAdd(cnt + (((code[e0 + i] >> cb) - row0) & (B - 1)), 1);
        __syncthreads();
        for (int i = tid; i < B; i += AT) row_cnt[(kk - k_lo) * B + i] = (uint16_t)cnt[i];
        const SlotPlan p = plan_slots(cnt, B, fpre, rank, gbase);
        if (tid == 0) {
            blocks[kk].vec = (int64_t)atomicAdd(counters + 0, (unsigned long long)p.vecs);
            blocks[kk].group = (int64_t)atomicAdd(counters + 1, (unsigned long long)p.groups);
            blocks[kk].n_groups = p.groups;
            blocks[kk].len = E;
        }
        __syncthreads();
    }
}

// One bin (row block x window) into groups of 32 slots.  The bin's elements (code = row in
// panel << cb | column in window, value) lie in the order in which the fill's warps
// reached it.  A group holds, step by step, two elements of each of its 32 slots; what a
// slot lacks to its group's length is padded with zeros (columns spread over the banks).
// Bins that fit are put together in shared memory and written out coalesced; larger ones
// are scattered.  Also the bin's largest row sum of |H|: FP32 values in integers, every
// element rounded up, so it bounds the exact sum and does not depend on the order (the
// column sums of a tile run over its bins: k_tile_finish, which takes the bin's largest |H|
// from col_bound); FP64 values (whose bins are whole tiles) in FP32 with a margin, and the
// larger of the row and column sums for both.
template <typename V, bool VLO>
__global__ void __launch_bounds__(AT) k_tile_arrange(int64_t k_lo, int64_t k_hi, int rb, int cb, int kb, int64_t chunk_el0,
                                                     TileBlock* __restrict__ blocks, const uint32_t* __restrict__ code,
                                                     const V* __restrict__ vin, const float* __restrict__ lin,
                                                     const uint16_t* __restrict__ row_cnt, int stage_cap,
                                                     unsigned long long* __restrict__ counters,
                                                     uint32_t* __restrict__ slots, int64_t* __restrict__ grp_off,
                                                     uint16_t* __restrict__ ocol, V* __restrict__ oval,
                                                     float* __restrict__ olo) {
    constexpr bool DBL = std::is_same<V, double>::value;
    extern __shared__ __align__(16) unsigned char sm[];
    const int B = 1 << kb, C = 1 << cb;
    uint32_t* cabs = reinterpret_cast<uint32_t*>(sm);       // FP64 values, C: column sums
    uint32_t* rabs = cabs + (DBL ? C : 0);                  // B: row sums
    int* cnt = reinterpret_cast<int*>(rabs + B);            // B: row lengths
    int* next = cnt + B;                                    // B: next element of each row
    int* fpre = next + B;                                   // B
    int* rank = fpre + B;                                   // B
    int* gbase = rank + B;                                  // B / 32 + 4
    V* stv = reinterpret_cast<V*>(gbase + B / 32 + 4);
    float* stl = reinterpret_cast<float*>(stv + stage_cap);
    uint16_t* stc = reinterpret_cast<uint16_t*>(stl + (VLO ? stage_cap : 0));
    __shared__ float s_max[AT / 32];
    __shared__ uint32_t s_rm, s_cm;
    __shared__ long long s_k;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t cmask = (uint32_t)C - 1u;
    for (;;) {
        if (tid == 0) {
            s_k = k_lo + (long long)atomicAdd(counters + 2, 1ull);
            s_rm = s_cm = 0;
        }
        __syncthreads();
        const int64_t kk = s_k;
        if (kk >= k_hi) break;
        const TileBlock b = blocks[kk];
        const int64_t e0 = b.el - chunk_el0;
        const int E = b.len, row0 = b.row & ((1 << rb) - 1);
        if constexpr (DBL)
            for (int i = tid; i < C; i += AT) cabs[i] = 0;
        for (int i = tid; i < B; i += AT) {
            rabs[i] = 0;
            next[i] = 0;
            cnt[i] = row_cnt[(kk - k_lo) * B + i];
        }
        float vmax = 0.f;
        if constexpr (!DBL)
            for (int i = tid; i < E; i += AT) vmax = fmaxf(vmax, fabsf(vin[e0 + i]));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) vmax = fmaxf(vmax, __shfl_xor_sync(FULL, vmax, o));
        if (lane == 0) s_max[warp] = vmax;
        __syncthreads();
        vmax = 0.f;
        for (int k = 0; k < AT / 32; k++) vmax = fmaxf(vmax, s_max[k]);
        const SlotPlan p = plan_slots(cnt, B, fpre, rank, gbase);
        const int gf = p.full >> 5;  // groups of full slots only
        auto base_of = [&](int g) { return g < gf ? g * 32 * (SEG / 2) : gbase[g - gf]; };
        const bool staged = 2 * p.vecs <= stage_cap;
        V* const dv = staged ? stv : oval + 2 * b.vec;
        float* const dl = staged ? stl : (VLO ? olo + 2 * b.vec : nullptr);
        uint16_t* const dc = staged ? stc : ocol + 2 * b.vec;
        for (int i = tid; i < 2 * p.vecs; i += AT) {
            dv[i] = 0;
            if constexpr (VLO) dl[i] = 0.f;
            dc[i] = (uint16_t)((i >> 1) & 31);
        }
        for (int g = tid; g < p.groups; g += AT) grp_off[b.group + g] = b.vec + base_of(g);
        for (int s = p.slots + tid; s < 32 * p.groups; s += AT) slots[32 * b.group + s] = 0u;  // lanes without a row
        for (int r = tid; r < B; r += AT) {
            const int c = cnt[r];
            for (int k = 0; k < c / SEG; k++)
                slots[32 * b.group + fpre[r] + k] = (uint32_t)(row0 + r) | ((uint32_t)SEG << 16);
            if (c % SEG) slots[32 * b.group + rank[r]] = (uint32_t)(row0 + r) | ((uint32_t)(c % SEG) << 16);
        }
        __syncthreads();
        // |H| in units of 2^-u, rounded up: at most C elements of at most vmax + 2 units
        int ex = 0;
        if (vmax > 0.f) frexpf(vmax, &ex);
        const int u = 31 - cb - 1 - ex;
        const double unit = ldexp(1.0, u);
        for (int i = tid; i < E; i += AT) {
            const uint32_t cd = code[e0 + i];
            const V v = vin[e0 + i];
            const int r = ((cd >> cb) - row0) & (B - 1), c = cd & cmask;
            if constexpr (DBL) {
                const float a = (float)fabs(v) * (1.f + 0x1p-20f);
                atomicAdd(reinterpret_cast<float*>(rabs) + r, a);
                atomicAdd(reinterpret_cast<float*>(cabs) + c, a);
            } else {
                atomicAdd(rabs + r, (uint32_t)__double2ll_ru(fabs((double)v) * unit) + (VLO ? 1u : 0u));
            }
            const int k = atomicAdd(next + r, 1), seg = k / SEG, kk2 = k % SEG;
            const int s = seg < cnt[r] / SEG ? fpre[r] + seg : rank[r];
            const int at = 2 * (base_of(s >> 5) + (kk2 >> 1) * 32 + (s & 31)) + (kk2 & 1);
            dv[at] = v;
            if constexpr (VLO) dl[at] = lin[e0 + i];
            dc[at] = (uint16_t)c;
        }
        __syncthreads();
        if (staged) {
            for (int i = tid; i < 2 * p.vecs; i += AT) {
                oval[2 * b.vec + i] = stv[i];
                if constexpr (VLO) olo[2 * b.vec + i] = stl[i];
                ocol[2 * b.vec + i] = stc[i];
            }
        }
        uint32_t rm = 0, cm = 0;
        for (int i = tid; i < B; i += AT) rm = max(rm, rabs[i]);
        if constexpr (DBL)
            for (int i = tid; i < C; i += AT) cm = max(cm, cabs[i]);
        rm = __reduce_max_sync(FULL, rm);
        cm = __reduce_max_sync(FULL, cm);
        if (lane == 0) {
            atomicMax(&s_rm, rm);
            atomicMax(&s_cm, cm);
        }
        __syncthreads();
        if (tid == 0) {
            if constexpr (DBL) {  // bits of non-negative floats order like the floats
                const float m = __uint_as_float(max(s_rm, s_cm)) * (1.f + 0x1p-16f);
                blocks[kk].row_bound = blocks[kk].col_bound = m;
            } else {
                blocks[kk].row_bound = __double2float_ru(ldexp((double)s_rm, -u));
                blocks[kk].col_bound = vmax;
            }
        }
        __syncthreads();
    }
}

// Per tile of a chunk (its first bin element: el0), one CTA each: pairs, the largest row sum
// of |H| of its row blocks, and its largest column sum, over all of them (integers as in
// k_tile_arrange: the largest of the blocks' own column sums, added, belongs to different
// columns and was 2.7 to 8 times the tile's, two to three bits of every product).  And into
// sums (units of 2^-20, rounded up) the row bounds per panel and the column bounds per
// window.  Bound by the read of code and value, 8 bytes a pair.
template <bool VLO>
__global__ void __launch_bounds__(TT) k_tile_finish(int64_t t_lo, int64_t t_hi, int64_t b_hi, int rb, int cb,
                                                    int64_t n_panels, int32_t chunk, int64_t el0,
                                                    TileBlock* __restrict__ blocks, const int32_t* __restrict__ tile_blk,
                                                    const int32_t* __restrict__ tile_win, const uint32_t* __restrict__ code,
                                                    const float* __restrict__ val, float2* __restrict__ tile_bound,
                                                    unsigned long long* __restrict__ sums,
                                                    unsigned long long* __restrict__ n_dense) {
    extern __shared__ __align__(16) unsigned char sm[];
    uint32_t* cabs = reinterpret_cast<uint32_t*>(sm);  // C column sums
    __shared__ uint32_t s_cm;
    const int C = 1 << cb;
    const uint32_t cmask = (uint32_t)C - 1u;
    for (int64_t t = t_lo + blockIdx.x; t < t_hi; t += gridDim.x) {
        const int64_t ka = tile_blk[t], kz = t + 1 < t_hi ? tile_blk[t + 1] : b_hi;
        for (int i = threadIdx.x; i < C; i += TT) cabs[i] = 0;
        if (threadIdx.x == 0) s_cm = 0;
        int len = 0;
        float rbnd = 0.f, vmax = 0.f;
        for (int64_t k = ka; k < kz; k++) {
            len += blocks[k].len;
            rbnd = fmaxf(rbnd, blocks[k].row_bound);
            vmax = fmaxf(vmax, blocks[k].col_bound);
        }
        __syncthreads();
        // units of 2^-u: at most 2^rb elements of at most vmax + 2 units in a column
        int ex = 0;
        if (vmax > 0.f) frexpf(vmax, &ex);
        const int u = 31 - rb - 1 - ex;
        const double unit = ldexp(1.0, u);
        for (int64_t k = ka; k < kz; k++) {
            const int64_t e0 = blocks[k].el - el0;
            const int E = blocks[k].len;
            for (int i = threadIdx.x; i < E; i += TT)
                atomicAdd(cabs + (code[e0 + i] & cmask),
                          (uint32_t)__double2ll_ru(fabs((double)val[e0 + i]) * unit) + (VLO ? 1u : 0u));
        }
        __syncthreads();
        uint32_t cm = 0;
        for (int i = threadIdx.x; i < C; i += TT) cm = max(cm, cabs[i]);
        cm = __reduce_max_sync(FULL, cm);
        if ((threadIdx.x & 31) == 0) atomicMax(&s_cm, cm);
        __syncthreads();
        if (threadIdx.x == 0) {
            const float cbnd = __double2float_ru(ldexp((double)s_cm, -u));
            tile_bound[t] = make_float2(rbnd, cbnd);
            atomicAdd(n_dense, (unsigned long long)len);
            const int64_t P = blocks[ka].row >> rb;
            atomicAdd(sums + P, (unsigned long long)__double2ll_ru((double)rbnd * 1048576.0));
            atomicAdd(sums + n_panels + tile_win[t], (unsigned long long)__double2ll_ru((double)cbnd * 1048576.0));
            for (int64_t k = ka; k < kz; k++) blocks[k].chunk = chunk;
        }
        __syncthreads();
    }
}

// |H| of the leftover pairs into the panels' and windows' sums.
template <bool VLO>
__global__ void k_left_sums(int64_t p_lo, int64_t p_hi, int cb, int64_t n_panels, const int64_t* __restrict__ left_off,
                            const int32_t* __restrict__ left_len, const uint32_t* __restrict__ col,
                            const float* __restrict__ val, unsigned long long* __restrict__ sums,
                            unsigned long long* __restrict__ n_left) {
    for (int64_t P = p_lo + blockIdx.x; P < p_hi; P += gridDim.x) {
        const int64_t s = left_off[P];
        const int n = left_len[P];
        unsigned long long mine = 0ull;
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const unsigned long long a =
                (unsigned long long)__double2ll_ru(fabs((double)val[s + i]) * 1048576.0) + (VLO ? 1ull : 0ull);
            mine += a;
            atomicAdd(sums + n_panels + (col[s + i] >> cb), a);
        }
        if (mine) atomicAdd(sums + P, mine);
        if (threadIdx.x == 0) atomicAdd(n_left, (unsigned long long)n);
    }
}

__global__ void k_block_len(int64_t nb, const TileBlock* __restrict__ blocks, int32_t* __restrict__ len) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < nb; k += (int64_t)gridDim.x * blockDim.x)
        len[k] = blocks[k].len;
}

// Leftover pairs of the panels [p_lo, p_hi): where the fill stopped.
__global__ void k_left_len(int64_t p_lo, int64_t p_hi, const unsigned long long* __restrict__ cur,
                           const int64_t* __restrict__ off, int32_t* __restrict__ len) {
    for (int64_t P = p_lo + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; P < p_hi; P += (int64_t)gridDim.x * blockDim.x)
        len[P] = (int32_t)((int64_t)cur[P] - off[P]);
}

// ---------------------------------------------------------------- conversion, FP64 values
//
// The FP64 upper triangle is regrouped from CSR rows: its tiles (tile_shape64), its split
// into dense tiles and leftovers and the order of a row's leftovers decide how its sigma
// rounds, and solves with a thick restart turn a difference of 1e-13 into another course of
// iterations, so these stay what they were.

// Per panel of the chunk [p_lo, p_hi): pairs in dense tiles, dense tiles, and per row the
// number of leftover pairs.  CSR input: row p's columns at cols[row_start[p] - base ...],
// row_len[p] of them.
__global__ void __launch_bounds__(CT) k_tile_count(int64_t N, int64_t p_lo, int64_t p_hi, int rb, int cb,
                                                   const int64_t* __restrict__ row_start, int64_t base,
                                                   const int32_t* __restrict__ row_len,
                                                   const int32_t* __restrict__ cols, PanelCount* __restrict__ out,
                                                   int32_t* __restrict__ left_len) {
    extern __shared__ int32_t hist[];
    using BR = cub::BlockReduce<long long, CT>;
    __shared__ typename BR::TempStorage red;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int64_t P = p_lo + blockIdx.x; P < p_hi; P += gridDim.x) {
        const int64_t r0 = P << rb, r1 = min(N, r0 + ((int64_t)1 << rb));
        const int64_t J0 = r0 >> cb;
        const int nb = (int)(((N - 1) >> cb) - J0 + 1);
        for (int b = threadIdx.x; b < nb; b += CT) hist[b] = 0;
        __syncthreads();
        for (int64_t r = r0 + warp; r < r1; r += CT / 32) {
            const int64_t s = row_start[r] - base;
            const int len = row_len[r];
            for (int k = lane; k < len; k += 32) atomicAdd(&hist[(cols[s + k] >> cb) - J0], 1);
        }
        __syncthreads();
        long long my_tiles = 0, my_dense = 0, my_left = 0;
        for (int b = threadIdx.x; b < nb; b += CT) {
            const int c = hist[b];
            if (c > 0 && dense_tile(c, window_width(N, J0 + b, cb))) {
                my_tiles++;
                my_dense += c;
            } else {
                my_left += c;
            }
        }
        for (int64_t r = r0 + warp; r < r1; r += CT / 32) {
            const int64_t s = row_start[r] - base;
            const int len = row_len[r];
            int nl = 0;
            for (int k = lane; k < len; k += 32) {
                const int64_t b = (cols[s + k] >> cb) - J0;
                nl += dense_tile(hist[b], window_width(N, J0 + b, cb)) ? 0 : 1;
            }
            nl = __reduce_add_sync(FULL, nl);
            if (lane == 0) left_len[r] = nl;
        }
        const long long t_tiles = BR(red).Sum(my_tiles);
        __syncthreads();
        const long long t_dense = BR(red).Sum(my_dense);
        __syncthreads();
        const long long t_left = BR(red).Sum(my_left);
        if (threadIdx.x == 0) out[P - p_lo] = PanelCount{t_dense, t_left, t_tiles, 0, 0, 0};
        __syncthreads();
    }
}

// Scatter the chunk's pairs: those of dense tiles, tile by tile, into code / val / lo, the
// leftovers in row order into lcol / lval / llo.  off: first element, tile and leftover of
// every panel.  A tile's place goes into its block, or into t_off / t_len.  Also adds |H_pq| to the row sums of both p and q (units of 2^-32:
// integer sums are exact, so the sums and the fixed-point scale derived from them do not
// depend on the order of the additions, nor on how the rows are split between ranks).
template <typename V, bool VLO>
__global__ void __launch_bounds__(CT) k_tile_scatter(
    int64_t N, int64_t p_lo, int64_t p_hi, int rb, int cb, const int64_t* __restrict__ row_start, int64_t base,
    const int32_t* __restrict__ row_len, const int32_t* __restrict__ cols, const V* __restrict__ vin,
    const float* __restrict__ lin, const PanelBase* __restrict__ off, int64_t left0, const int32_t* __restrict__ left_len,
    int32_t* __restrict__ tile_win, TileBlock* __restrict__ blocks, int64_t* __restrict__ t_off, int32_t* __restrict__ t_len,
    int64_t* __restrict__ row_left, uint32_t* code, V* val, float* lo, uint32_t* lcol, V* lval, float* llo,
    unsigned long long* __restrict__ row_abs) {
    extern __shared__ int32_t sm_i[];
    int32_t* cursor = sm_i;              // per window: next dense slot (panel-relative), or -1
    int32_t* lcur = sm_i + MAX_BINS;     // per row of the panel: leftover start (panel-relative)
    using BS = cub::BlockScan<long long, CT>;
    __shared__ typename BS::TempStorage scan;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const uint32_t cmask = (1u << cb) - 1u;
    for (int64_t P = p_lo + blockIdx.x; P < p_hi; P += gridDim.x) {
        const int64_t r0 = P << rb, r1 = min(N, r0 + ((int64_t)1 << rb));
        const int nr = (int)(r1 - r0);
        const int64_t J0 = r0 >> cb;
        const int nb = (int)(((N - 1) >> cb) - J0 + 1);
        const PanelBase pb = off[P - p_lo];
        for (int b = threadIdx.x; b < nb; b += CT) cursor[b] = 0;
        __syncthreads();
        for (int64_t r = r0 + warp; r < r1; r += CT / 32) {
            const int64_t s = row_start[r] - base;
            const int len = row_len[r];
            for (int k = lane; k < len; k += 32) atomicAdd(&cursor[(cols[s + k] >> cb) - J0], 1);
        }
        __syncthreads();
        // dense windows in window order: element and tile prefix sums over contiguous
        // chunks of windows per thread
        const int per = (nb + CT - 1) / CT;
        const int b_lo = min(nb, (int)threadIdx.x * per), b_hi = min(nb, b_lo + per);
        long long my_el = 0, my_t = 0;
        for (int b = b_lo; b < b_hi; b++) {
            const int c = cursor[b];
            if (c > 0 && dense_tile(c, window_width(N, J0 + b, cb))) {
                my_el += c;
                my_t++;
            }
        }
        long long ex_el, ex_t;
        BS(scan).ExclusiveSum(my_el, ex_el);
        __syncthreads();
        BS(scan).ExclusiveSum(my_t, ex_t);
        __syncthreads();
        for (int b = b_lo; b < b_hi; b++) {
            const int c = cursor[b];
            if (c > 0 && dense_tile(c, window_width(N, J0 + b, cb))) {
                const long long t = pb.tile + ex_t;
                tile_win[t] = (int32_t)(J0 + b);
                if (blocks) {
                    blocks[t].el = pb.el + ex_el;
                    blocks[t].len = c;
                    blocks[t].row = (int32_t)r0;
                } else {
                    t_off[t] = pb.el + ex_el;
                    t_len[t] = c;
                }
                cursor[b] = (int32_t)ex_el;
                ex_el += c;
                ex_t++;
            } else {
                cursor[b] = -1;
            }
        }
        // leftover regions of the rows, in row order
        {
            const int rper = (nr + CT - 1) / CT;
            const int q_lo = min(nr, (int)threadIdx.x * rper), q_hi = min(nr, q_lo + rper);
            long long my_l = 0;
            for (int i = q_lo; i < q_hi; i++) my_l += left_len[r0 + i];
            long long ex_l;
            BS(scan).ExclusiveSum(my_l, ex_l);
            for (int i = q_lo; i < q_hi; i++) {
                lcur[i] = (int32_t)ex_l;
                row_left[r0 + i] = left0 + pb.block + ex_l;
                ex_l += left_len[r0 + i];
            }
        }
        __syncthreads();
        for (int64_t r = r0 + warp; r < r1; r += CT / 32) {
            const int64_t s = row_start[r] - base;
            const int len = row_len[r];
            const uint32_t lr = (uint32_t)(r - r0);
            int lnext = lcur[lr];
            unsigned long long rsum = 0ull;
            for (int k0 = 0; k0 < len; k0 += 32) {
                const int k = k0 + lane;
                const bool act = k < len;
                int q = 0;
                int32_t cur = -1;
                if (act) {
                    q = cols[s + k];
                    cur = cursor[(q >> cb) - J0];
                }
                const bool left = act && cur < 0;
                const unsigned ml = __ballot_sync(FULL, left);
                // this row's pairs that fall in one dense tile take consecutive slots
                const bool dense = act && !left;
                const int bin = (int)((q >> cb) - J0);
                const unsigned grp = __match_any_sync(FULL, dense ? bin : (int)(0x80000000u | (unsigned)lane));
                const int leader = __ffs(grp) - 1;
                int slot = 0;
                if (dense && lane == leader) slot = atomicAdd(&cursor[bin], __popc(grp));
                slot = __shfl_sync(FULL, slot, leader);
                if (act) {
                    const V v = vin[s + k];
                    if (left) {
                        const int64_t pos = pb.block + lnext + __popc(ml & lt);
                        lcol[pos] = (uint32_t)q;
                        lval[pos] = v;
                        if constexpr (VLO) llo[pos] = lin[s + k];
                    } else {
                        const int64_t pos = pb.el + slot + __popc(grp & lt);
                        code[pos] = (lr << cb) | ((uint32_t)q & cmask);
                        val[pos] = v;
                        if constexpr (VLO) lo[pos] = lin[s + k];
                    }
                    const unsigned long long ai = (unsigned long long)llrint(fabs((double)v) * 4294967296.0);
                    rsum += ai;
                    atomicAdd(row_abs + q, ai);
                }
                lnext += __popc(ml);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) rsum += __shfl_xor_sync(FULL, rsum, o);
            if (lane == 0 && rsum) atomicAdd(row_abs + r, rsum);
        }
        __syncthreads();
    }
}

__global__ void k_max_u64(const unsigned long long* __restrict__ a, int64_t n, unsigned long long* __restrict__ out) {
    unsigned long long m = 0ull;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        m = max(m, a[i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(FULL, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

// Bound and chunk of every tile once it is arranged.
__global__ void k_tile_finish64(int64_t nt, int32_t chunk, TileBlock* __restrict__ blocks, float2* __restrict__ bound,
                                unsigned long long* __restrict__ n_dense) {
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < nt; t += (int64_t)gridDim.x * blockDim.x) {
        blocks[t].chunk = chunk;
        bound[t] = make_float2(blocks[t].row_bound, blocks[t].col_bound);
        atomicAdd(n_dense, (unsigned long long)blocks[t].len);
    }
}

// ---------------------------------------------------------------- sigma

// Block b of 2^wb entries: max |x| into wmax[b], the accumulator zeroed.  The last block
// to finish gathers the largest of all and sets the scale of the whole sigma:
// scalars[0] max |x|, [1] 2^s, [2] 2^-s, [3] the work-unit counter; [4] counts the blocks.
template <typename X, typename Y>
__global__ void __launch_bounds__(256) k_sigma_prep(const X* __restrict__ x, int64_t N, int wb, Y* __restrict__ acc,
                                                    long long* __restrict__ acc_row, double* __restrict__ wmax, double row_abs_max, int smax, int top,
                                                    double* __restrict__ scalars, const int* __restrict__ stop) {
    if (stop && *stop) return;
    __shared__ double s_m[8];
    __shared__ bool s_last;
    auto block_max = [&](double v) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(FULL, v, o));
        if ((threadIdx.x & 31) == 0) s_m[threadIdx.x >> 5] = v;
        __syncthreads();
        double r = 0.0;
        for (int k = 0; k < 8; k++) r = fmax(r, s_m[k]);
        __syncthreads();
        return r;
    };
    const int64_t i0 = (int64_t)blockIdx.x << wb, i1 = min(N, i0 + ((int64_t)1 << wb));
    double m = 0.0;
    for (int64_t i = i0 + threadIdx.x; i < i1; i += 256) {
        m = fmax(m, fabs((double)x[i]));
        acc[i] = 0;
        if (acc_row) acc_row[i] = 0;
    }
    m = block_max(m);
    unsigned long long* const done = reinterpret_cast<unsigned long long*>(scalars) + 4;
    if (threadIdx.x == 0) {
        wmax[blockIdx.x] = m;
        __threadfence();
        s_last = atomicAdd(done, 1ull) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    m = 0.0;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += 256) m = fmax(m, __ldcg(wmax + b));
    m = block_max(m);
    if (threadIdx.x == 0) {
        const double bound = row_abs_max * m;
        int s = 0;
        if (bound > 0.0 && isfinite(bound)) s = top - ilogb(bound);
        s = max(-smax, min(smax, s));
        scalars[0] = m;
        scalars[1] = ldexp(1.0, s);
        scalars[2] = ldexp(1.0, -s);
        reinterpret_cast<unsigned long long*>(scalars)[3] = 0ull;
        *done = 0ull;
    }
}

// Four FP32 sums added to four consecutive global floats (16-byte aligned) by one
// vector reduction.
__device__ __forceinline__ void red_add_v4(float* a, const float4 v) {
    asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(a), "f"(v.x), "f"(v.y),
                 "f"(v.z), "f"(v.w)
                 : "memory");
}

// Stages x[0, n) into shared memory (16-byte vector loads when x is aligned).
template <typename X>
__device__ __forceinline__ void stage_window(X* __restrict__ dst, const X* __restrict__ x, int n) {
    constexpr int PER = 16 / sizeof(X);
    int i0 = 0;
    if ((reinterpret_cast<uintptr_t>(x) & 15u) == 0) {
        const int nv = n / PER;
        for (int i = threadIdx.x; i < nv; i += ST) reinterpret_cast<uint4*>(dst)[i] = __ldg(reinterpret_cast<const uint4*>(x) + i);
        i0 = nv * PER;
    }
    for (int i = i0 + threadIdx.x; i < n; i += ST) dst[i] = x[i];
}

// Two consecutive stored values as the vector type.
template <typename V, typename X, bool VLO>
__device__ __forceinline__ void load2(const V* __restrict__ vals, const float* __restrict__ vlo, X (&v)[2]) {
    if constexpr (std::is_same<V, double>::value) {
        const double2 a = __ldcs(reinterpret_cast<const double2*>(vals));
        v[0] = (X)a.x;
        v[1] = (X)a.y;
    } else {
        const float2 a = __ldcs(reinterpret_cast<const float2*>(vals));
        v[0] = (X)a.x;
        v[1] = (X)a.y;
        if constexpr (VLO) {
            const float2 l = __ldcs(reinterpret_cast<const float2*>(vlo));
            v[0] += (X)l.x;
            v[1] += (X)l.y;
        }
    }
}

// The tiles of a handle, for the kernels.
template <typename V>
struct TileView {
    int rb, cb, wb;  // log2 of the rows of a panel, the columns of a window, the entries per max |x|
    const int64_t* __restrict__ panel_tile;
    const int32_t* __restrict__ tile_win;
    const int32_t* __restrict__ tile_blk;   // n_tiles + 1
    const float2* __restrict__ tile_bound;  // largest row sum, bound on the column sums
    const TileBlock* __restrict__ blocks;
    const TileChunk* __restrict__ chunks;   // the arrays of each chunk of panels
    const int64_t* __restrict__ left_off;   // per panel
    const int32_t* __restrict__ left_len;
    const uint32_t* __restrict__ lcol;
    const uint16_t* __restrict__ lrow;
    const V* __restrict__ lval;
    const float* __restrict__ llo;
    const int64_t* __restrict__ row_left;   // FP64 values: leftovers per row
    const int32_t* __restrict__ row_nleft;
};

// Power of two, as an exponent, that takes sums of at most b below 2^(top + 1).
__device__ __forceinline__ int fixed_shift(double b, int most, int top) {
    int sh = 0;
    if (b > 0.0 && isfinite(b)) sh = top - ilogb(b);
    return max(-most, min(most, sh));
}

// The largest such for 32-bit sums: the margin of 2^-13 (2^18 units) covers what the up to
// 2^11 products of a sum are rounded by.
__device__ __forceinline__ int fixed_shift32(double b, int most) { return fixed_shift(b * (1.0 + 0x1p-13), most, 30); }

// Fixed-point tile sigma.  Shared-memory integer atomics are single instructions,
// where FP32 shared atomics are compare-and-swap loops and 64-bit ones slower still
// (measured on B200: 7.9, 2.6 and 1.5 per clock per SM), so each tile's column sums are
// formed in 32-bit integers: every product is scaled by 2^s_t, s_t chosen from the tile's
// largest column sum of |H| times the panel's max |x| so that no sum reaches 2^31,
// and rounded to an integer (FP32 vectors) or, at 2^lb times that scale, to a 64-bit
// integer whose high part and low lb = 32 - rb bits are added apart (FP64 vectors: 51 or
// more bits below the largest sum; the 2^rb rows of a panel cannot overflow the low parts).
// Row sums stay in the register of the lane that holds the row: 32-bit integers, scaled
// like the columns by the tile's largest row sum and the window's max |x|, for FP32
// vectors, 64-bit integers at the scale 2^S of the whole sigma for FP64 ones.  EXACT: all
// sums are shifted to the scale 2^S and added with 64-bit global atomics, so sigma is
// bitwise reproducible and ranks' partial sums add exactly; otherwise (FP32 vectors) the
// rows' are (in FP32, a row's sums from every tile of its panel were what rounded most on a
// vector without signs: 6.6e-8 of |y|, against 4.1e-8), and a window's are added in FP32,
// four columns at a time.
//
// FP64 values: rows and columns of a tile share one scale, 2^20 times finer than the one
// that takes the tile's bound times max |x| to 2^30, and a sum that the scale 2^S cannot
// hold exactly is rounded to it once per tile (row sums then gather in shared memory).
//
// A work unit is a run of one tile's row blocks, or leftovers of a panel.  Its warps take
// groups of 32 rows from a counter and meet only when the window is flushed; the next
// group's header is loaded while this one's elements are summed.
template <typename X, typename V, bool VLO, bool EXACT>
__global__ void __launch_bounds__(ST, sizeof(X) == 4 ? 6 : 3)
    k_sigma_fx(int64_t N, int64_t n_units, const SigmaUnit* __restrict__ units, TileView<V> T, const X* __restrict__ x,
               const double* __restrict__ wmax, void* __restrict__ acc_out, unsigned long long* __restrict__ acc_row,
               double* __restrict__ scalars, const int* __restrict__ stop) {
    if (stop && *stop) return;
    constexpr bool DBL = std::is_same<X, double>::value;
    constexpr bool V64 = std::is_same<V, double>::value;
    using RS = typename std::conditional<DBL, long long, typename std::conditional<EXACT, int, float>::type>::type;
    constexpr int PARTS = DBL || EXACT ? 1 : 4;  // of an FP32 row sum: a quarter of the elements each
    constexpr int U = DBL ? 2 : 4;  // steps in flight
    extern __shared__ __align__(16) unsigned char sm[];
    const int C = 1 << T.cb, lb = 32 - T.rb;
    X* xJ = reinterpret_cast<X*>(sm);
    int* yJa = reinterpret_cast<int*>(xJ + C);
    unsigned* yJb = reinterpret_cast<unsigned*>(yJa + C);  // FP64 vectors
    unsigned long long* yR = reinterpret_cast<unsigned long long*>(yJb + C);  // FP64 values: 2^rb row sums
    __shared__ long long s_unit;
    __shared__ int s_next;
    const int lane = threadIdx.x & 31;
    const double gscale = scalars[1];  // 2^S
    const int S = ilogb(gscale);
    unsigned long long* counter = reinterpret_cast<unsigned long long*>(scalars) + 3;
    unsigned long long* acc_ll = reinterpret_cast<unsigned long long*>(acc_out);
    X* acc_x = reinterpret_cast<X*>(acc_out);
    auto max_of = [&](int64_t i0, int64_t i1) {  // max |x| over the entries [i0, i1) (a panel's or window's)
        double m = 0.0;
        for (int64_t b = i0 >> T.wb; b << T.wb < i1; b++) m = fmax(m, wmax[b]);
        return m;
    };
    for (;;) {
        if (threadIdx.x == 0) {
            s_unit = (long long)atomicAdd(counter, 1ull);
            s_next = 0;
        }
        __syncthreads();
        if (s_unit >= n_units) break;
        const SigmaUnit u = units[s_unit];
        const int64_t r0 = (int64_t)u.panel << T.rb;
        if (V64 && u.tile < 0) {
            // leftover pairs: one warp per row, private row sum, column sums of the rounded products
            for (int64_t p = r0 + u.lo + (threadIdx.x >> 5); p < r0 + u.hi; p += ST / 32) {
                const int64_t s = T.row_left[p];
                const int len = T.row_nleft[p];
                if (len == 0) continue;
                const X xp = __ldg(x + p);
                X rs = 0;
                for (int k = lane; k < len; k += 32) {
                    const uint32_t q = __ldcs(T.lcol + s + k);
                    const X v = (X)__ldcs(T.lval + s + k);
                    rs += v * __ldg(x + q);
                    atomicAdd(acc_ll + q, (unsigned long long)llrint((double)(v * xp) * gscale));
                }
                // fixed lane order: the warp sum does not depend on timing
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) rs += __shfl_xor_sync(FULL, rs, o);
                if (lane == 0) atomicAdd(acc_ll + p, (unsigned long long)llrint((double)rs * gscale));
            }
            __syncthreads();
            continue;
        }
        if (u.tile < 0) {
            // leftover pairs: row and column sums of the rounded products
            const int64_t s = T.left_off[u.panel] + u.lo;
            for (int i = threadIdx.x; i < u.hi - u.lo; i += ST) {
                const uint32_t q = __ldcs(T.lcol + s + i);
                const int64_t p = r0 + __ldcs(T.lrow + s + i);
                X v = (X)__ldcs(T.lval + s + i);
                if constexpr (VLO) v += (X)__ldcs(T.llo + s + i);
                const X pr = v * __ldg(x + q), pc = v * __ldg(x + p);
                if constexpr (EXACT) {
                    atomicAdd(acc_ll + p, (unsigned long long)llrint((double)pr * gscale));
                    atomicAdd(acc_ll + q, (unsigned long long)llrint((double)pc * gscale));
                } else {
                    atomicAdd(acc_row + p, (unsigned long long)llrint((double)pr * gscale));
                    atomicAdd(acc_x + q, pc);
                }
            }
            __syncthreads();
            continue;
        }
        const int64_t c0 = (int64_t)T.tile_win[u.tile] << T.cb;
        const int w = (int)min((int64_t)C, N - c0);
        const float2 bound = T.tile_bound[u.tile];
        // EXACT: no finer than the scale of the whole sigma, so that every sum is converted to
        // it without rounding and neither the cut into slots and units nor the order matters
        int sh, rsh = S;  // of the column sums (FP64 vectors: lb bits finer) and of the row sums
        if constexpr (V64) {
            sh = fixed_shift((double)bound.y * scalars[0], 200, 29) + 20 - lb;
            rsh = sh + lb;
        } else {
            sh = fixed_shift32((double)bound.y * max_of(r0, min(N, r0 + ((int64_t)1 << T.rb))), DBL ? 800 : 120);
            if constexpr (EXACT) sh = min(sh, DBL ? S - lb : S);
            if constexpr (EXACT && !DBL) rsh = min(S, fixed_shift32((double)bound.x * max_of(c0, c0 + w), 120));
        }
        const X csc = (X)ldexp(1.0, DBL ? sh + lb : sh);
        const X rsc = (X)ldexp(1.0, rsh);
        const bool gather = V64 && rsh > S;  // row sums round to 2^S: together, once
        if (gather)
            for (int i = threadIdx.x; i < (1 << T.rb); i += ST) yR[i] = 0ull;
        stage_window<X>(xJ, x + c0, w);
        // padding has columns 0..31: in a narrower window they have to hold a finite x too
        for (int i = w + threadIdx.x; i < 32; i += ST) xJ[i] = 0;
        for (int i = threadIdx.x; i < w; i += ST) {
            yJa[i] = 0;
            if constexpr (DBL) yJb[i] = 0u;
        }
        // this lane's row block of the unit
        const TileChunk ch = T.chunks[u.chunk];
        const int nb = u.hi - u.lo;
        const int my_n = lane < nb ? T.blocks[u.lo + lane].n_groups : 0;
        const int64_t my_g = lane < nb ? T.blocks[u.lo + lane].group : 0;
        const int n_items = nb * __reduce_max_sync(FULL, my_n);
        __syncthreads();
        // The next group: its row slots (this lane's, 0 when there is none) and first pair of
        // elements.  The blocks' first groups go first, then their second ones: groups are of
        // falling length in a block, so the long ones are not left for the end.
        auto take = [&](uint32_t& hd, int64_t& off) -> bool {
            for (;;) {
                int k = 0;
                if (lane == 0) k = atomicAdd(&s_next, 1);
                k = __shfl_sync(FULL, k, 0);
                if (k >= n_items) {
                    hd = 0;
                    return false;
                }
                const int gi = k / nb, b = k - gi * nb;
                if (gi >= __shfl_sync(FULL, my_n, b)) continue;
                const int64_t g = __shfl_sync(FULL, my_g, b) + gi;
                hd = __ldg(ch.slots + 32 * g + lane);
                off = __ldg(ch.grp_off + g);
                return true;
            }
        };
        uint32_t hd = 0, hd_next = 0;
        int64_t off = 0, off_next = 0;
        bool have = take(hd, off);
        while (have) {
            const bool more = take(hd_next, off_next);
            const int len = (int)(hd >> 16);
            const int64_t row = r0 + (hd & 0xffffu);
            const X xr = len > 0 ? __ldg(x + row) * csc : (X)0;
            RS rs[PARTS] = {};
            auto add = [&](RS& rs, int cc, X vv) {
                if constexpr (DBL) {
                    rs += __double2ll_rn(vv * xJ[cc] * rsc);
                    const long long q = __double2ll_rn(vv * xr);
                    atomicAdd(yJa + cc, (int)(q >> lb));
                    atomicAdd(yJb + cc, (unsigned)q & ((1u << lb) - 1u));
                } else {
                    if constexpr (EXACT) rs += __float2int_rn(vv * xJ[cc] * rsc);
                    else rs += vv * xJ[cc];
                    atomicAdd(yJa + cc, __float2int_rn(vv * xr));
                }
            };
            const ushort2* pc = reinterpret_cast<const ushort2*>(ch.col) + off + lane;
            const V* pv = reinterpret_cast<const V*>(ch.val) + 2 * (off + lane);
            const float* pl = VLO ? ch.lo + 2 * (off + lane) : nullptr;
            const int steps = (__shfl_sync(FULL, len, 0) + 1) >> 1;
            int j = 0;
            for (; j + U <= steps; j += U) {
                ushort2 c[U];
                X v[U][2];
#pragma unroll
                for (int k = 0; k < U; k++) {
                    c[k] = __ldcs(pc + 32 * k);
                    load2<V, X, VLO>(pv + 64 * k, pl + 64 * k, v[k]);
                }
                pc += 32 * U;
                pv += 64 * U;
                if constexpr (VLO) pl += 64 * U;
#pragma unroll
                for (int k = 0; k < U; k++) {
                    add(rs[2 * k % PARTS], c[k].x, v[k][0]);
                    add(rs[(2 * k + 1) % PARTS], c[k].y, v[k][1]);
                }
            }
            for (; j < steps; j++) {
                const ushort2 c = __ldcs(pc);
                X v[2];
                load2<V, X, VLO>(pv, pl, v);
                pc += 32;
                pv += 64;
                if constexpr (VLO) pl += 64;
                add(rs[0], c.x, v[0]);
                add(rs[1 % PARTS], c.y, v[1]);
            }
            if (len > 0) {
                if (gather) atomicAdd(yR + (row - r0), (unsigned long long)rs[0]);
                else if constexpr (EXACT) atomicAdd(acc_row + row, (unsigned long long)((long long)rs[0] << (S - rsh)));
                else {
                    double sum = 0.0;
#pragma unroll
                    for (int k = 0; k < PARTS; k++) sum += (double)rs[k];
                    atomicAdd(acc_row + row, (unsigned long long)llrint(sum * gscale));
                }
            }
            hd = hd_next;
            off = off_next;
            have = more;
        }
        __syncthreads();
        // column window sums to the global accumulator
        if constexpr (EXACT) {
            const int up = DBL ? S - sh - lb : S - sh;
            for (int i = threadIdx.x; i < w; i += ST) {
                long long q;
                if constexpr (DBL) q = ((long long)yJa[i] << lb) + (long long)yJb[i];
                else q = yJa[i];
                if (V64 && up < 0) q = llrint((double)q * ldexp(1.0, up));
                else q <<= up;
                if (q != 0) atomicAdd(acc_ll + c0 + i, (unsigned long long)q);
            }
            if (gather)
                for (int i = threadIdx.x; i < (1 << T.rb); i += ST) {
                    const long long q = llrint((double)(long long)yR[i] * ldexp(1.0, S - rsh));
                    if (q != 0) atomicAdd(acc_ll + r0 + i, (unsigned long long)q);
                }
        } else {
            const float inv = ldexpf(1.f, -sh);
            float* dst = reinterpret_cast<float*>(acc_x) + c0;
            // c0 is a multiple of 4 and the accumulator is 256-byte aligned
            for (int i = threadIdx.x; i < (w >> 2); i += ST) {
                const int4 a = reinterpret_cast<const int4*>(yJa)[i];
                if (a.x | a.y | a.z | a.w)
                    red_add_v4(dst + 4 * i, make_float4((float)a.x * inv, (float)a.y * inv, (float)a.z * inv,
                                                        (float)a.w * inv));
            }
            for (int i = 4 * (w >> 2) + threadIdx.x; i < w; i += ST)
                if (yJa[i] != 0) atomicAdd(dst + i, (float)yJa[i] * inv);
        }
        __syncthreads();
    }
}

// y = diag x + acc 2^-s, or with FP32 column sums diag x + acc + acc_row 2^-s
template <typename X, typename T>
__global__ void k_fixed_finish(int64_t N, const double* __restrict__ diag, const X* __restrict__ x,
                               const T* __restrict__ acc, const long long* __restrict__ acc_row,
                               const double* __restrict__ scalars, X* __restrict__ y) {
    constexpr bool FX = std::is_same<T, long long>::value;
    const double inv = scalars[2];
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < N; p += (int64_t)gridDim.x * blockDim.x)
        y[p] = (X)(diag[p] * (double)x[p] + (FX ? (double)acc[p] * inv : (double)acc[p] + (double)acc_row[p] * inv));
}

#include "tiles_list.cuh"

// Calls f(p, q, v) for every stored pair (p < q, internal indices, FP64 value): one CTA
// per panel, a warp per group of rows of its tiles, then its leftovers.
template <typename V, bool VLO, typename F>
__global__ void __launch_bounds__(TT) k_tiles_each(int64_t N, int64_t p_lo, int64_t p_hi, TileView<V> T, F f) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int64_t P = p_lo + blockIdx.x; P < p_hi; P += gridDim.x) {
        const int64_t r0 = P << T.rb;
        for (int64_t t = T.panel_tile[P]; t < T.panel_tile[P + 1]; t++) {
            const int64_t c0 = (int64_t)T.tile_win[t] << T.cb;
            for (int k = T.tile_blk[t]; k < T.tile_blk[t + 1]; k++) {
                const TileBlock b = T.blocks[k];
                const TileChunk ch = T.chunks[b.chunk];
                const V* val = reinterpret_cast<const V*>(ch.val);
                for (int g = warp; g < b.n_groups; g += TT / 32) {
                    const uint32_t hd = ch.slots[32 * (b.group + g) + lane];
                    const int row = (int)(hd & 0xffffu), len = (int)(hd >> 16);
                    const int64_t at = ch.grp_off[b.group + g] + lane;
                    for (int i = 0; i < len; i++) {
                        const int64_t e = 2 * (at + 32 * (i >> 1)) + (i & 1);
                        double v = (double)val[e];
                        if constexpr (VLO) v += (double)ch.lo[e];
                        f(r0 + row, c0 + ch.col[e], v);
                    }
                }
            }
        }
        if constexpr (std::is_same<V, double>::value) {
            for (int64_t p = r0 + warp; p < min(N, r0 + ((int64_t)1 << T.rb)); p += TT / 32)
                for (int k = lane; k < T.row_nleft[p]; k += 32)
                    f(p, (int64_t)T.lcol[T.row_left[p] + k], T.lval[T.row_left[p] + k]);
            continue;
        }
        const int64_t s = T.left_off[P];
        for (int i = threadIdx.x; i < T.left_len[P]; i += TT) {
            double v = (double)T.lval[s + i];
            if constexpr (VLO) v += (double)T.llo[s + i];
            f(r0 + T.lrow[s + i], (int64_t)T.lcol[s + i], v);
        }
    }
}

struct CooOut {
    int32_t* p;
    int32_t* q;
    double* v;
    unsigned long long* count;
    unsigned long long cap;
    __device__ void operator()(int64_t pp, int64_t qq, double vv) const {
        const unsigned long long e = atomicAdd(count, 1ull);
        if (e < cap) {
            p[e] = (int32_t)pp;
            q[e] = (int32_t)qq;
            v[e] = vv;
        }
    }
};

struct SelfEnergyAdd {
    const double* diag;
    double energy, gmin;
    double* out;
    __device__ void operator()(int64_t pp, int64_t qq, double vv) const {
        const double v2 = vv * vv;
        atomicAdd(out + pp, -v2 / fmax(diag[qq] - energy, gmin));
        atomicAdd(out + qq, -v2 / fmax(diag[pp] - energy, gmin));
    }
};

// Stored pairs that touch a marked row (bitmap over internal indices), in the caller's
// indices, both orientations: (row, column, value) with the row marked.
struct RowFilter {
    const uint32_t* mark;
    const int32_t* orig;
    int64_t* out_r;
    int64_t* out_c;
    double* out_v;
    unsigned long long* count;
    unsigned long long cap;
    __device__ void emit(int64_t r, int64_t c, double v) const {
        const unsigned long long k = atomicAdd(count, 1ull);
        if (k < cap) {
            out_r[k] = orig[r];
            out_c[k] = orig[c];
            out_v[k] = v;
        }
    }
    __device__ void operator()(int64_t pp, int64_t qq, double vv) const {
        if ((mark[pp >> 5] >> (pp & 31)) & 1u) emit(pp, qq, vv);
        if ((mark[qq >> 5] >> (qq & 31)) & 1u) emit(qq, pp, vv);
    }
};

template <typename V>
TileView<V> tile_view(risqgpu* h, const V* lval, const float* llo) {
    TileView<V> T;
    T.rb = h->tile_rb;
    T.cb = h->tile_cb;
    T.wb = std::min(h->tile_rb, h->tile_cb);
    T.panel_tile = h->d_panel_tile;
    T.tile_win = h->d_tile_win;
    T.tile_blk = h->d_tile_blk;
    T.tile_bound = h->d_tile_bound;
    T.blocks = h->d_tile_blocks;
    T.chunks = h->d_chunk_tab;
    T.left_off = h->d_left_off;
    T.left_len = h->d_left_len;
    T.lcol = h->d_left_col;
    T.lrow = h->d_left_row;
    T.lval = lval;
    T.llo = llo;
    T.row_left = h->d_row_left;
    T.row_nleft = h->d_row_nleft;
    return T;
}

template <typename F>
int tiles_each(risqgpu* h, F f) {
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(h->part_p_hi - h->part_p_lo, (int64_t)num_sms(h) * 8));
    const int64_t N = (int64_t)h->N, lo = h->part_p_lo, hi = h->part_p_hi;
    if (h->tile_list) {
        if (h->precision == RISQGPU_FP64)
            k_list_each<double, false, F><<<grid, TT, 0, h->stream>>>(N, lo, hi, list_view<double>(h), f);
        else if (h->precision == RISQGPU_MIXED)
            k_list_each<float, true, F><<<grid, TT, 0, h->stream>>>(N, lo, hi, list_view<float>(h), f);
        else
            k_list_each<float, false, F><<<grid, TT, 0, h->stream>>>(N, lo, hi, list_view<float>(h), f);
        return check_launch(h, "tiled pairs");
    }
    if (h->precision == RISQGPU_FP64)
        k_tiles_each<double, false, F><<<grid, TT, 0, h->stream>>>(
            N, lo, hi, tile_view<double>(h, h->d_left64, nullptr), f);
    else if (h->precision == RISQGPU_MIXED)
        k_tiles_each<float, true, F><<<grid, TT, 0, h->stream>>>(
            N, lo, hi, tile_view<float>(h, h->d_left32, h->d_left_lo), f);
    else
        k_tiles_each<float, false, F><<<grid, TT, 0, h->stream>>>(
            N, lo, hi, tile_view<float>(h, h->d_left32, nullptr), f);
    return check_launch(h, "tiled pairs");
}

inline int grid_n(risqgpu* h, int64_t n) {
    return (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, (int64_t)num_sms(h) * 16));
}

template <typename X, typename V, bool EXACT, typename K, typename T_>
int launch_sigma(risqgpu* h, const X* x, X* y, K kern, size_t smem, const T_& T) {
    using Y = typename std::conditional<EXACT, long long, X>::type;
    const int64_t N = (int64_t)h->N;
    RQ_TRY(allow_smem(h, kern, smem));
    int occ = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, ST, smem);
    // FP32 sums: N columns, then the rows' in fixed point
    long long* const acc_row = EXACT ? nullptr : h->d_acc + (N + 1) / 2;
    const int grid =
        (int)std::max<int64_t>(1, std::min<int64_t>(h->n_units, (int64_t)num_sms(h) * std::max(occ, 1)));
    k_sigma_prep<X, Y><<<(int)(((N - 1) >> T.wb) + 1), 256, 0, h->stream>>>(
        x, N, T.wb, reinterpret_cast<Y*>(h->d_acc), acc_row, h->d_wmax, h->h_row_abs_max,
        std::is_same<X, float>::value ? 100 : 1000, 61, h->d_sig_scalars, h->stop_flag);
    kern<<<grid, ST, smem, h->stream>>>(N, h->n_units, h->d_units, T, x, h->d_wmax, h->d_acc,
                                        reinterpret_cast<unsigned long long*>(EXACT ? h->d_acc : acc_row),
                                        h->d_sig_scalars, h->stop_flag);
    RQ_TRY(check_launch(h, "sigma (tiles)"));
    // with a row-block partition every rank summed its own panels: the exact integer
    // sums are added across the ranks
    if (EXACT && h->part_n > 1) RQ_TRY(part_allreduce(h, h->d_acc, (size_t)N));
    k_fixed_finish<X, Y><<<grid_n(h, N), 256, 0, h->stream>>>(N, h->d_diag, x, reinterpret_cast<const Y*>(h->d_acc),
                                                             acc_row, h->d_sig_scalars, y);
    return check_launch(h, "sigma (tiles)");
}

template <typename X, typename V, bool VLO, bool EXACT>
int launch_fx(risqgpu* h, const X* x, X* y, const V* lval, const float* llo) {
    if (h->tile_list) {
        const size_t smem = ((size_t)(8 + 2 * sizeof(X)) << h->tile_rb) + ((size_t)(2 * sizeof(X)) << h->tile_cb);
        return launch_sigma<X, V, EXACT>(h, x, y, k_sigma_list<X, V, VLO, EXACT>, smem, list_view<V>(h));
    }
    // x and the accumulators of a window; FP64 values: the row sums of a panel
    const size_t smem = (((size_t)2 * sizeof(X)) << h->tile_cb) + (sizeof(V) == 8 ? (size_t)8 << h->tile_rb : 0);
    return launch_sigma<X, V, EXACT>(h, x, y, k_sigma_fx<X, V, VLO, EXACT>, smem, tile_view<V>(h, lval, llo));
}

}  // namespace

int part_allreduce(risqgpu* h, void* buf_dev, size_t count) {
    if (!h->part_reduce) {
        h->err = "partitioned handle without a reduce function";
        return RISQGPU_ERR_INVALID;
    }
    if (h->part_reduce(buf_dev, count, (void*)h->stream, h->part_user) != 0) {
        h->err = "the caller's all-reduce failed";
        return RISQGPU_ERR_CUDA;
    }
    return check_launch(h, "all-reduce");
}

int part_agree(risqgpu* h, int rc) {
    if (h->part_n <= 1) return rc;
    // out of memory counts one, any other failure 2^32
    const unsigned long long mine = rc == RISQGPU_OK ? 0ull : rc == RISQGPU_ERR_OOM ? 1ull : 1ull << 32;
    unsigned long long all = 0;
    RQ_CUDA(h, cudaMemcpyAsync(h->d_agree, &mine, sizeof(mine), cudaMemcpyHostToDevice, h->stream));
    RQ_TRY(part_allreduce(h, h->d_agree, 1));
    RQ_CUDA(h, cudaMemcpyAsync(&all, h->d_agree, sizeof(all), cudaMemcpyDeviceToHost, h->stream));
    RQ_TRY(sync(h, "agreement of the ranks"));
    if (rc != RISQGPU_OK && rc != RISQGPU_ERR_OOM) return rc;
    if (all >> 32) { h->err = "another rank's build failed"; return RISQGPU_ERR_INVALID; }
    if (all && rc == RISQGPU_OK) h->err = "another rank is out of device memory";
    return all ? RISQGPU_ERR_OOM : RISQGPU_OK;
}

namespace {

// The device's table of the element arrays.
int chunk_table(risqgpu* h) {
    RQ_TRY(dalloc(h, h->d_chunk_tab, h->chunks.size()));
    if (!h->chunks.empty())
        RQ_CUDA(h, cudaMemcpyAsync(h->d_chunk_tab, h->chunks.data(), sizeof(TileChunk) * h->chunks.size(),
                                   cudaMemcpyHostToDevice, h->stream));
    return RISQGPU_OK;
}

// The handle's units: by weight in steps of an eighth of the target, falling.
int set_units(risqgpu* h, const std::vector<SigmaUnit>& us, const std::vector<int64_t>& weight, int64_t target) {
    constexpr size_t NB = 512;
    std::vector<size_t> start(NB + 2, 0);
    auto bucket = [&](int64_t w) { return NB - (size_t)std::min<int64_t>((int64_t)NB, w * 8 / target); };
    for (int64_t w : weight) start[bucket(w) + 1]++;
    for (size_t b = 1; b < start.size(); b++) start[b] += start[b - 1];
    std::vector<SigmaUnit> ordered(us.size());
    for (size_t i = 0; i < us.size(); i++) ordered[start[bucket(weight[i])]++] = us[i];
    h->n_units = (int64_t)us.size();
    if (!us.empty()) {
        RQ_TRY(dalloc(h, h->d_units, ordered.size()));
        RQ_CUDA(h, cudaMemcpyAsync(h->d_units, ordered.data(), sizeof(SigmaUnit) * ordered.size(), cudaMemcpyHostToDevice,
                                   h->stream));
        RQ_TRY(sync(h, "sigma units"));
    }
    return RISQGPU_OK;
}

// Units of the leftovers of panel P's rows (nl of each row), about a quarter of the target
// each, since one costs about four dense pairs.
void left_units(std::vector<SigmaUnit>& us, std::vector<int64_t>& weight, const std::vector<int32_t>& nl, int64_t P,
                int64_t R, int64_t N, int64_t target) {
    const int64_t r0 = P * R, r1 = std::min(N, r0 + R);
    int64_t lo = r0, acc = 0;
    for (int64_t r = r0; r < r1; r++) {
        acc += nl[(size_t)r];
        if ((acc >= target / 4 || r + 1 == r1) && acc > 0) {
            us.push_back({-1, (int32_t)P, (int32_t)(lo - r0), (int32_t)(r + 1 - r0), 0});
            weight.push_back(4 * acc);
            lo = r + 1;
            acc = 0;
        }
    }
}

}  // namespace

int tile_shape(int64_t N, int& rb, int& cb, int& kb) {
    // Windows of 4096 columns, or fewer while there would be under 1,200 bins of 256 rows
    // (a work unit is at least one): a wide window makes long rows in a bin, so less
    // padding and fewer group headers.  Panels of up to 2048 rows, at least 32 of them: a
    // tile's scale comes from its panel's largest |x| and the sums of its 256-row blocks'
    // column bounds.
    cb = 12;
    while (cb > 8 && (double)N * (double)N / ((double)((int64_t)256 << cb) * 2) < 1200.0) cb--;
    rb = 11;
    while (rb > 8 && (N >> rb) < 32) rb--;
    // blocks of 256 rows (a bin's elements fit shared memory), of more once the table of
    // bins would exceed 2^25 entries
    kb = 8;
    while (kb < std::min(rb, cb) && (double)N * (double)N / ((double)((int64_t)1 << (kb + cb)) * 2) > (double)(1 << 25)) kb++;
    // columns in a window and the length of a row in a tile are coded in 16 bits
    while (cb < 15 && ((N + ((int64_t)1 << cb) - 1) >> cb) > 16384) cb++;
    return ((N + ((int64_t)1 << cb) - 1) >> cb) <= 65536 ? RISQGPU_OK : RISQGPU_ERR_INVALID;
}

int tile_shape64(int64_t N, int64_t pairs, int& rb, int& cb) {
    rb = 10;  // 1024 rows per panel
    // 2048 columns per window; 4096 where a row has less than one pair in such a window on
    // average, since a row's slot, x_p and row sum cost as much as several pairs: 9,150,723
    // determinants (0.54 pairs), FP64 sigma 63.3 ms at 2048, 56.7 at 4096.  Sets of up to
    // 551,147 determinants have 4 and more.
    const int64_t half = ((N + 2047) >> 11) / 2;
    cb = pairs < N * half ? 12 : 11;
    while (cb < 16 && ((N + ((int64_t)1 << cb) - 1) >> cb) > MAX_BINS) cb++;
    return ((N + ((int64_t)1 << cb) - 1) >> cb) <= MAX_BINS ? RISQGPU_OK : RISQGPU_ERR_INVALID;
}

int tile_shape_list(int64_t N, int& rb, int& cb) {
    rb = 10;
    cb = 11;
    while (cb < 16 && ((N + ((int64_t)1 << cb) - 1) >> cb) > MAX_BINS) cb++;
    return ((N + ((int64_t)1 << cb) - 1) >> cb) <= MAX_BINS ? RISQGPU_OK : RISQGPU_ERR_INVALID;
}

int TileBuilder::plan(risqgpu* h_, const uint32_t* hist, const int64_t* bin_off, int64_t n_blocks_) {
    h = h_;
    n_blocks = n_blocks_;
    const int64_t N = (int64_t)h->N, np = h->n_panels;
    counts.resize((size_t)np);
    PanelCount* d = nullptr;
    ScopedFree<1> release(d);
    RQ_TRY(dalloc(h, d, (size_t)np));
    k_panel_count<<<(int)std::min<int64_t>(np, (int64_t)num_sms(h) * 8), TT, 0, h->stream>>>(
        N, np, n_blocks, h->tile_rb, h->tile_cb, h->tile_kb, hist, bin_off, d);
    RQ_TRY(check_launch(h, "panel counts"));
    RQ_CUDA(h, cudaMemcpyAsync(counts.data(), d, sizeof(PanelCount) * np, cudaMemcpyDeviceToHost, h->stream));
    return sync(h, "panel counts");
}

// Sizes and allocates the arrays of the panels [p_lo, p_hi) and plans every bin.
int TileBuilder::begin(int64_t p_lo, int64_t p_hi, int precision, const uint32_t* hist, const int64_t* bin_off,
                       unsigned long long* cur) {
    const int64_t N = (int64_t)h->N, np = h->n_panels;
    const bool lo = precision == RISQGPU_MIXED;
    base.assign((size_t)np + 1, PanelBase{0, 0, 0});
    panel_chunk.assign((size_t)np, 0);
    std::vector<int64_t> loff((size_t)np, 0), pt((size_t)np + 1, 0);
    left = 0;
    PanelBase b{0, 0, 0};
    for (int64_t P = 0; P <= np; P++) {
        base[(size_t)P] = b;
        pt[(size_t)P] = b.tile;
        if (P == np) break;
        loff[(size_t)P] = left;
        if (P < p_lo || P >= p_hi) continue;
        const PanelCount& c = counts[(size_t)P];
        b.el += c.dense;
        b.tile += c.tiles;
        b.block += c.blocks;
        left += c.left;
    }
    const int64_t nt = b.tile, nb = b.block;
    if (nt >= INT32_MAX || nb >= INT32_MAX) { h->err = "too many tiles"; return RISQGPU_ERR_INVALID; }
    h->n_tiles = nt;
    RQ_TRY(dalloc(h, h->d_panel_tile, (size_t)np + 1));
    RQ_TRY(dalloc(h, h->d_tile_win, (size_t)nt));
    RQ_TRY(dalloc(h, h->d_tile_blk, (size_t)nt + 1));
    RQ_TRY(dalloc(h, h->d_tile_bound, (size_t)nt));
    RQ_TRY(dalloc(h, h->d_tile_blocks, (size_t)nb));
    RQ_TRY(dalloc(h, h->d_left_off, (size_t)np));
    RQ_TRY(dalloc(h, h->d_left_len, (size_t)np));
    RQ_TRY(dalloc(h, h->d_left_col, (size_t)left));
    RQ_TRY(dalloc(h, h->d_left_row, (size_t)left));
    RQ_TRY(dalloc(h, h->d_left32, (size_t)left));
    if (lo) RQ_TRY(dalloc(h, h->d_left_lo, (size_t)left));
    RQ_TRY(dalloc_reduced(h, h->d_acc, (size_t)(N + (N + 1) / 2)));
    RQ_TRY(dalloc(h, h->d_sig_scalars, 5));
    RQ_TRY(dalloc(h, h->d_wmax, (size_t)((N - 1) >> std::min(h->tile_rb, h->tile_cb)) + 1));
    RQ_TRY(dalloc(h, left_cur, (size_t)np));
    RQ_TRY(dalloc_reduced(h, sums, (size_t)(np + ((N - 1) >> h->tile_cb) + 1)));
    RQ_TRY(dalloc(h, counters, 5));
    RQ_CUDA(h, cudaMemsetAsync(h->d_sig_scalars, 0, sizeof(double) * 5, h->stream));
    RQ_CUDA(h, cudaMemsetAsync(h->d_left_len, 0, sizeof(int32_t) * np, h->stream));
    RQ_CUDA(h, cudaMemsetAsync(sums, 0, sizeof(unsigned long long) * (np + ((N - 1) >> h->tile_cb) + 1), h->stream));
    RQ_CUDA(h, cudaMemsetAsync(counters, 0, sizeof(unsigned long long) * 5, h->stream));
    PanelBase* db = nullptr;
    ScopedFree<1> release(db);
    RQ_TRY(dalloc(h, db, (size_t)np + 1));
    RQ_CUDA(h, cudaMemcpyAsync(db, base.data(), sizeof(PanelBase) * (np + 1), cudaMemcpyHostToDevice, h->stream));
    RQ_CUDA(h, cudaMemcpyAsync(h->d_panel_tile, pt.data(), sizeof(int64_t) * (np + 1), cudaMemcpyHostToDevice, h->stream));
    RQ_CUDA(h, cudaMemcpyAsync(h->d_left_off, loff.data(), sizeof(int64_t) * np, cudaMemcpyHostToDevice, h->stream));
    RQ_CUDA(h, cudaMemcpyAsync(left_cur, loff.data(), sizeof(int64_t) * np, cudaMemcpyHostToDevice, h->stream));
    const int32_t end = (int32_t)nb;
    RQ_CUDA(h, cudaMemcpyAsync(h->d_tile_blk + nt, &end, sizeof(int32_t), cudaMemcpyHostToDevice, h->stream));
    if (p_hi > p_lo)
        k_panel_plan<<<(int)std::min<int64_t>(p_hi - p_lo, (int64_t)num_sms(h) * 8), TT, 0, h->stream>>>(
            N, p_lo, p_hi, n_blocks, h->tile_rb, h->tile_cb, h->tile_kb, hist, bin_off, db, h->d_tile_win,
            h->d_tile_blk, h->d_tile_blocks, cur);
    RQ_TRY(check_launch(h, "panel plan"));
    return sync(h, "panel plan");
}

namespace {

// The elements of the bins blocks[k_lo, k_hi) (in code / vin / lin, bins starting at their
// `el` minus el0) into arrays of just the size they need, appended to the handle's chunks.
template <typename V>
int arrange_bins(risqgpu* h, TileBlock* blocks, int64_t k_lo, int64_t k_hi, int64_t el0, const unsigned long long* cur,
                 const uint32_t* code, const V* vin, const float* lin, unsigned long long* counters) {
    const int B = 1 << h->tile_kb, C = 1 << h->tile_cb;
    const int64_t nb = k_hi - k_lo;
    h->chunks.emplace_back();
    if (nb <= 0) return RISQGPU_OK;
    uint16_t* row_cnt = nullptr;
    ScopedFree<1> release(row_cnt);
    RQ_TRY(dalloc(h, row_cnt, (size_t)nb * B));
    auto grid_of = [&](auto kern, size_t smem) {
        int occ = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, AT, smem);
        return (int)std::min<int64_t>(nb, (int64_t)num_sms(h) * std::max(occ, 1));
    };
    RQ_CUDA(h, cudaMemsetAsync(counters, 0, sizeof(unsigned long long) * 3, h->stream));
    const size_t smem1 = sizeof(int) * (size_t)(3 * B + B / 32 + 4);
    RQ_TRY(allow_smem(h, k_tile_size, smem1));
    k_tile_size<<<grid_of(k_tile_size, smem1), AT, smem1, h->stream>>>(k_lo, k_hi, h->tile_rb, h->tile_cb, h->tile_kb, el0,
                                                                       blocks, cur, code, row_cnt, counters);
    RQ_TRY(check_launch(h, "tile sizes"));
    unsigned long long c[2] = {0, 0};
    RQ_CUDA(h, cudaMemcpyAsync(c, counters, sizeof(c), cudaMemcpyDeviceToHost, h->stream));
    RQ_TRY(sync(h, "tile sizes"));
    TileChunk& ch = h->chunks.back();
    V* val = nullptr;
    RQ_TRY(dalloc(h, ch.grp_off, (size_t)c[1]));
    RQ_TRY(dalloc(h, ch.slots, (size_t)c[1] * 32));
    RQ_TRY(dalloc(h, ch.col, (size_t)c[0] * 2));
    RQ_TRY(dalloc(h, val, (size_t)c[0] * 2));
    ch.val = val;
    if (lin) RQ_TRY(dalloc(h, ch.lo, (size_t)c[0] * 2));
    RQ_CUDA(h, cudaMemsetAsync(counters + 2, 0, sizeof(unsigned long long), h->stream));
    const size_t fixed = sizeof(uint32_t) * (size_t)((sizeof(V) == 8 ? C : 0) + 5 * B + B / 32 + 4);
    const size_t per = 2 + sizeof(V) + (lin ? 4 : 0);
    // two CTAs per SM
    const int cap = (int)((((size_t)110 << 10) - std::min(fixed, (size_t)100 << 10)) / per) & ~63;
    const size_t smem = fixed + (size_t)cap * per;
    auto go = [&](auto kern) -> int {
        RQ_TRY(allow_smem(h, kern, smem));
        kern<<<grid_of(kern, smem), AT, smem, h->stream>>>(k_lo, k_hi, h->tile_rb, h->tile_cb, h->tile_kb, el0, blocks,
                                                           code, vin, lin, row_cnt, cap, counters, ch.slots, ch.grp_off,
                                                           ch.col, val, ch.lo);
        return check_launch(h, "tile arrangement");
    };
    if constexpr (std::is_same<V, double>::value) return go(k_tile_arrange<double, false>);
    else if (lin) return go(k_tile_arrange<float, true>);
    else return go(k_tile_arrange<float, false>);
}

}  // namespace

// Arranges the panels [p_lo, p_hi), whose candidates the fill has put into the temporary
// arrays (chunk_el0: the chunk's first element).
int TileBuilder::chunk(int64_t p_lo, int64_t p_hi, int64_t chunk_el0, const unsigned long long* cur,
                       const uint32_t* code, const float* vin, const float* lin) {
    const int64_t np = p_hi - p_lo;
    if (np <= 0) return RISQGPU_OK;
    const PanelBase a = base[(size_t)p_lo], z = base[(size_t)p_hi];
    RQ_TRY(arrange_bins<float>(h, h->d_tile_blocks, a.block, z.block, chunk_el0, cur, code, vin, lin, counters));
    const int32_t id = (int32_t)h->chunks.size() - 1;
    for (int64_t P = p_lo; P < p_hi; P++) panel_chunk[(size_t)P] = id;
    if (z.tile > a.tile) {
        const int64_t nt = z.tile - a.tile;
        const size_t smem = sizeof(uint32_t) << h->tile_cb;
        auto go = [&](auto kern) -> int {
            RQ_TRY(allow_smem(h, kern, smem));
            kern<<<(int)std::min<int64_t>(nt, (int64_t)num_sms(h) * 64), TT, smem, h->stream>>>(
                a.tile, z.tile, z.block, h->tile_rb, h->tile_cb, h->n_panels, id, chunk_el0, h->d_tile_blocks, h->d_tile_blk,
                h->d_tile_win, code, vin, h->d_tile_bound, sums, counters + 3);
            return check_launch(h, "tile bounds");
        };
        RQ_TRY(lin ? go(k_tile_finish<true>) : go(k_tile_finish<false>));
    }
    k_left_len<<<grid_n(h, np), 256, 0, h->stream>>>(p_lo, p_hi, left_cur, h->d_left_off, h->d_left_len);
    const int grid = (int)std::min<int64_t>(np, (int64_t)num_sms(h) * 8);
    if (lin)
        k_left_sums<true><<<grid, 256, 0, h->stream>>>(p_lo, p_hi, h->tile_cb, h->n_panels, h->d_left_off, h->d_left_len,
                                                       h->d_left_col, h->d_left32, sums, counters + 4);
    else
        k_left_sums<false><<<grid, 256, 0, h->stream>>>(p_lo, p_hi, h->tile_cb, h->n_panels, h->d_left_off, h->d_left_len,
                                                        h->d_left_col, h->d_left32, sums, counters + 4);
    return check_launch(h, "leftover sums");
}

int TileBuilder::finish() {
    const int64_t N = (int64_t)h->N, np = h->n_panels, nw = ((N - 1) >> h->tile_cb) + 1;
    // bounds on the row sums of |H| over both triangles: with a partition each rank holds
    // part of them, so the integer sums are added across the ranks first
    if (h->part_n > 1) RQ_TRY(part_allreduce(h, sums, (size_t)(np + nw)));
    std::vector<unsigned long long> s((size_t)(np + nw));
    unsigned long long c[5] = {0, 0, 0, 0, 0};
    RQ_CUDA(h, cudaMemcpyAsync(s.data(), sums, sizeof(unsigned long long) * s.size(), cudaMemcpyDeviceToHost, h->stream));
    RQ_CUDA(h, cudaMemcpyAsync(c, counters, sizeof(c), cudaMemcpyDeviceToHost, h->stream));
    RQ_TRY(sync(h, "row sums"));
    const unsigned long long row = *std::max_element(s.begin(), s.begin() + np);
    const unsigned long long col = *std::max_element(s.begin() + np, s.end());
    h->h_row_abs_max = 1.01 * ((double)(row + col) / 1048576.0) + 1e-6;
    h->n_dense_el = c[3];
    stored = (int64_t)(c[3] + c[4]);
    RQ_TRY(chunk_table(h));
    h->tiled = true;
    return make_units();
}

// Sigma work units: every tile's row blocks in runs of at most about `target` pairs, every
// panel's leftovers in runs of that many, the large ones first, so that the CTAs that take
// units from a counter finish together.
int TileBuilder::make_units() {
    const int64_t p_lo = h->part_p_lo, p_hi = h->part_p_hi, nt = h->n_tiles, nb = base[(size_t)h->n_panels].block;
    std::vector<int32_t> tblk((size_t)nt + 1), ll((size_t)h->n_panels), bl((size_t)nb);
    int32_t* dbl = nullptr;
    ScopedFree<1> release(dbl);
    RQ_TRY(dalloc(h, dbl, (size_t)nb));
    if (nb > 0) k_block_len<<<grid_n(h, nb), 256, 0, h->stream>>>(nb, h->d_tile_blocks, dbl);
    RQ_TRY(check_launch(h, "sigma units"));
    RQ_CUDA(h, cudaMemcpyAsync(bl.data(), dbl, sizeof(int32_t) * nb, cudaMemcpyDeviceToHost, h->stream));
    RQ_CUDA(h, cudaMemcpyAsync(tblk.data(), h->d_tile_blk, sizeof(int32_t) * (nt + 1), cudaMemcpyDeviceToHost, h->stream));
    RQ_CUDA(h, cudaMemcpyAsync(ll.data(), h->d_left_len, sizeof(int32_t) * ll.size(), cudaMemcpyDeviceToHost, h->stream));
    RQ_TRY(sync(h, "sigma units"));
    const int64_t target = std::max<int64_t>(16384, stored / ((int64_t)num_sms(h) * 32));
    std::vector<SigmaUnit> us;
    std::vector<int64_t> weight;
    for (int64_t P = p_lo; P < p_hi; P++) {
        for (int64_t t = base[(size_t)P].tile; t < base[(size_t)P + 1].tile; t++) {
            int32_t lo = tblk[(size_t)t];
            const int32_t end = tblk[(size_t)t + 1];
            int64_t acc = 0;
            for (int32_t k = lo; k < end; k++) {
                acc += bl[(size_t)k];
                if (acc >= target || k + 1 == end || k + 1 - lo == 32) {
                    if (acc > 0) {
                        us.push_back({(int32_t)t, (int32_t)P, lo, k + 1, panel_chunk[(size_t)P]});
                        weight.push_back(acc);
                    }
                    lo = k + 1;
                    acc = 0;
                }
            }
        }
        // a leftover pair costs about four dense ones
        for (int64_t i = 0; i < ll[(size_t)P]; i += target / 4) {
            const int64_t e = std::min<int64_t>(ll[(size_t)P], i + target / 4);
            us.push_back({-1, (int32_t)P, (int32_t)i, (int32_t)e, 0});
            weight.push_back(4 * (e - i));
        }
    }
    return set_units(h, us, weight, target);
}

int Tiles64Builder::begin(risqgpu* h_) {
    h = h_;
    const int64_t N = (int64_t)h->N;
    panel_tile.assign((size_t)h->n_panels + 1, 0);
    RQ_TRY(dalloc(h, h->d_row_left, (size_t)N));
    RQ_TRY(dalloc(h, h->d_row_nleft, (size_t)N));
    RQ_TRY(dalloc_reduced(h, row_abs, (size_t)N));
    RQ_TRY(dalloc(h, absmax, 1));
    RQ_TRY(dalloc(h, counters, 4));
    RQ_CUDA(h, cudaMemsetAsync(h->d_row_nleft, 0, sizeof(int32_t) * N, h->stream));
    RQ_CUDA(h, cudaMemsetAsync(row_abs, 0, sizeof(unsigned long long) * N, h->stream));
    RQ_CUDA(h, cudaMemsetAsync(absmax, 0, sizeof(unsigned long long), h->stream));
    RQ_CUDA(h, cudaMemsetAsync(counters, 0, sizeof(unsigned long long) * 4, h->stream));
    return RISQGPU_OK;
}

int Tiles64Builder::chunk(int64_t p_lo, int64_t p_hi, const int64_t* row_start, int64_t base, const int32_t* row_len,
                          const int32_t* cols, const double* vin, uint32_t* code, double* val, int64_t cap) {
    const int64_t N = (int64_t)h->N, np = p_hi - p_lo;
    if (np <= 0) return RISQGPU_OK;
    PanelCount* dc = nullptr;
    PanelBase* db = nullptr;
    ScopedFree<2> release(dc, db);
    RQ_TRY(dalloc(h, dc, (size_t)np));
    RQ_TRY(dalloc(h, db, (size_t)np));
    const int rb = h->tile_rb, cb = h->tile_cb;
    const size_t smem_count = sizeof(int32_t) * MAX_BINS;
    const size_t smem_scatter = sizeof(int32_t) * (MAX_BINS + ((size_t)1 << rb));
    RQ_TRY(allow_smem(h, k_tile_count, smem_count));
    RQ_TRY((allow_smem(h, k_tile_scatter<double, false>, smem_scatter)));
    const int grid = (int)std::min<int64_t>(np, (int64_t)num_sms(h) * 2);
    k_tile_count<<<grid, CT, smem_count, h->stream>>>(N, p_lo, p_hi, rb, cb, row_start, base, row_len, cols, dc,
                                                      h->d_row_nleft);
    RQ_TRY(check_launch(h, "tile count"));
    std::vector<PanelCount> pc((size_t)np);
    RQ_CUDA(h, cudaMemcpyAsync(pc.data(), dc, sizeof(PanelCount) * np, cudaMemcpyDeviceToHost, h->stream));
    RQ_TRY(sync(h, "tile count"));
    // first element, tile and (as `block`) leftover of every panel, in the chunk's arrays
    std::vector<PanelBase> pb((size_t)np);
    PanelBase b{0, 0, 0};
    for (int64_t P = 0; P < np; P++) {
        pb[(size_t)P] = b;
        panel_tile[(size_t)(p_lo + P)] = tiles + b.tile;
        b.el += pc[(size_t)P].dense;
        b.tile += pc[(size_t)P].tiles;
        b.block += pc[(size_t)P].left;
    }
    if (b.el > cap) {
        h->err = "tiled layout: " + std::to_string(b.el) + " elements exceed the " + std::to_string(cap) + " slots counted";
        return RISQGPU_ERR_INVALID;
    }
    RQ_CUDA(h, cudaMemcpyAsync(db, pb.data(), sizeof(PanelBase) * np, cudaMemcpyHostToDevice, h->stream));
    parts.push_back({p_lo, p_hi, b.tile, b.block, nullptr, nullptr, nullptr, nullptr, nullptr});
    Chunk& c = parts.back();
    RQ_TRY(dalloc(h, c.blocks, (size_t)b.tile));
    RQ_TRY(dalloc(h, c.win, (size_t)b.tile));
    RQ_TRY(dalloc(h, c.bound, (size_t)b.tile));
    RQ_TRY(dalloc(h, c.lcol, (size_t)b.block));
    RQ_TRY(dalloc(h, c.lval, (size_t)b.block));
    k_tile_scatter<double, false><<<grid, CT, smem_scatter, h->stream>>>(
        N, p_lo, p_hi, rb, cb, row_start, base, row_len, cols, vin, nullptr, db, left, h->d_row_nleft, c.win, c.blocks, nullptr,
        nullptr, h->d_row_left, code, val, nullptr, c.lcol, c.lval, nullptr, row_abs);
    RQ_TRY(check_launch(h, "tile scatter"));
    RQ_TRY(arrange_bins<double>(h, c.blocks, 0, b.tile, 0, nullptr, code, val, nullptr, counters));
    if (b.tile > 0) {
        k_tile_finish64<<<grid_n(h, b.tile), 256, 0, h->stream>>>(b.tile, (int32_t)h->chunks.size() - 1, c.blocks, c.bound,
                                                                  counters + 3);
        RQ_TRY(check_launch(h, "tile bounds"));
    }
    tiles += b.tile;
    left += b.block;
    return RISQGPU_OK;
}

int Tiles64Builder::gather() {
    const int64_t np = h->n_panels;
    for (int64_t P = h->part_p_hi; P <= np; P++) panel_tile[(size_t)P] = tiles;
    if (tiles >= INT32_MAX) { h->err = "too many tiles"; return RISQGPU_ERR_INVALID; }
    h->n_tiles = tiles;
    // the chunks' tile records and leftovers in one array each
    auto gather = [&](auto*& dst, auto Chunk::*src, int64_t n, int64_t Chunk::*count) -> int {
        using E = typename std::remove_pointer<typename std::remove_reference<decltype(dst)>::type>::type;
        if (parts.size() == 1) {
            dfree(dst);
            dst = parts[0].*src;
            parts[0].*src = nullptr;
            return RISQGPU_OK;
        }
        RQ_TRY(dalloc(h, dst, (size_t)n));
        int64_t at = 0;
        for (Chunk& c : parts) {
            if (c.*count > 0)
                RQ_CUDA(h, cudaMemcpyAsync(dst + at, c.*src, sizeof(E) * (c.*count), cudaMemcpyDeviceToDevice, h->stream));
            at += c.*count;
            dfree(c.*src);
        }
        return RISQGPU_OK;
    };
    RQ_TRY(gather(h->d_tile_blocks, &Chunk::blocks, tiles, &Chunk::tiles));
    RQ_TRY(gather(h->d_tile_win, &Chunk::win, tiles, &Chunk::tiles));
    RQ_TRY(gather(h->d_tile_bound, &Chunk::bound, tiles, &Chunk::tiles));
    RQ_TRY(gather(h->d_left_col, &Chunk::lcol, left, &Chunk::left));
    return gather(h->d_left64, &Chunk::lval, left, &Chunk::left);
}

int Tiles64Builder::finish() {
    const int64_t N = (int64_t)h->N, np = h->n_panels;
    std::vector<int32_t> tblk((size_t)tiles + 1);
    for (int64_t t = 0; t <= tiles; t++) tblk[(size_t)t] = (int32_t)t;  // a tile is one block
    RQ_TRY(dalloc(h, h->d_panel_tile, (size_t)np + 1));
    RQ_TRY(dalloc(h, h->d_tile_blk, (size_t)tiles + 1));
    RQ_CUDA(h, cudaMemcpyAsync(h->d_panel_tile, panel_tile.data(), sizeof(int64_t) * (np + 1), cudaMemcpyHostToDevice,
                               h->stream));
    RQ_CUDA(h, cudaMemcpyAsync(h->d_tile_blk, tblk.data(), sizeof(int32_t) * (tiles + 1), cudaMemcpyHostToDevice,
                               h->stream));
    // row sums of |H| over both triangles: with a partition each rank holds part of every
    // row's sum, so the exact integer sums are added across the ranks first
    if (h->part_n > 1) RQ_TRY(part_allreduce(h, row_abs, (size_t)N));
    k_max_u64<<<grid_n(h, N), 256, 0, h->stream>>>(row_abs, N, absmax);
    unsigned long long mi = 0, dense = 0;
    std::vector<TileBlock> tb((size_t)tiles);
    std::vector<int32_t> nl((size_t)N);
    RQ_CUDA(h, cudaMemcpyAsync(&mi, absmax, sizeof(mi), cudaMemcpyDeviceToHost, h->stream));
    RQ_CUDA(h, cudaMemcpyAsync(&dense, counters + 3, sizeof(dense), cudaMemcpyDeviceToHost, h->stream));
    if (tiles > 0)
        RQ_CUDA(h, cudaMemcpyAsync(tb.data(), h->d_tile_blocks, sizeof(TileBlock) * tiles, cudaMemcpyDeviceToHost, h->stream));
    RQ_CUDA(h, cudaMemcpyAsync(nl.data(), h->d_row_nleft, sizeof(int32_t) * N, cudaMemcpyDeviceToHost, h->stream));
    RQ_TRY(dalloc_reduced(h, h->d_acc, (size_t)N));
    RQ_TRY(dalloc(h, h->d_sig_scalars, 5));
    RQ_TRY(dalloc(h, h->d_wmax, (size_t)((N - 1) >> std::min(h->tile_rb, h->tile_cb)) + 1));
    RQ_CUDA(h, cudaMemsetAsync(h->d_sig_scalars, 0, sizeof(double) * 5, h->stream));
    RQ_TRY(sync(h, "row sums"));
    // each |H_pq| was rounded to a multiple of 2^-32: the margin covers that rounding
    h->h_row_abs_max = 1.01 * ((double)mi / 4294967296.0) + 1e-6;
    h->n_dense_el = dense;
    stored = (int64_t)dense + left;
    RQ_TRY(chunk_table(h));
    h->tiled = true;
    // units: whole tiles (a tile's sums are rounded together), and rows with leftovers
    std::vector<SigmaUnit> us;
    std::vector<int64_t> weight;
    const int64_t R = (int64_t)1 << h->tile_rb, target = 32768;
    for (int64_t P = h->part_p_lo; P < h->part_p_hi; P++) {
        for (int64_t t = panel_tile[(size_t)P]; t < panel_tile[(size_t)P + 1]; t++) {
            us.push_back({(int32_t)t, (int32_t)P, (int32_t)t, (int32_t)t + 1, tb[(size_t)t].chunk});
            weight.push_back(tb[(size_t)t].len);
        }
        left_units(us, weight, nl, P, R, N, target);
    }
    return set_units(h, us, weight, target);
}

Tiles64Builder::~Tiles64Builder() {
    dfree(row_abs);
    dfree(absmax);
    dfree(counters);
    for (Chunk& c : parts) {
        dfree(c.blocks);
        dfree(c.win);
        dfree(c.bound);
        dfree(c.lcol);
        dfree(c.lval);
    }
}

int TileListBuilder::begin(risqgpu* h_, int precision_, int64_t cap_) {
    h = h_;
    precision = precision_;
    cap = cap_;
    const int64_t N = (int64_t)h->N;
    panel_tile.assign((size_t)h->n_panels + 1, 0);
    RQ_TRY(dalloc(h, h->d_row_left, (size_t)N));
    RQ_TRY(dalloc(h, h->d_row_nleft, (size_t)N));
    RQ_TRY(dalloc_reduced(h, row_abs, (size_t)N));
    RQ_TRY(dalloc(h, absmax, 1));
    RQ_TRY(dalloc(h, h->d_el_idx, (size_t)cap));
    if (precision == RISQGPU_FP64) RQ_TRY(dalloc(h, h->d_val64, (size_t)cap));
    else RQ_TRY(dalloc(h, h->d_val32, (size_t)cap));
    if (precision == RISQGPU_MIXED) RQ_TRY(dalloc(h, h->d_val_lo, (size_t)cap));
    RQ_CUDA(h, cudaMemsetAsync(h->d_row_nleft, 0, sizeof(int32_t) * N, h->stream));
    RQ_CUDA(h, cudaMemsetAsync(row_abs, 0, sizeof(unsigned long long) * N, h->stream));
    RQ_CUDA(h, cudaMemsetAsync(absmax, 0, sizeof(unsigned long long), h->stream));
    return RISQGPU_OK;
}

int TileListBuilder::chunk(int64_t p_lo, int64_t p_hi, const int64_t* row_start, int64_t base, const int32_t* row_len,
                           const int32_t* cols, const double* v64, const float* v32, const float* vlo) {
    const int64_t N = (int64_t)h->N, np = p_hi - p_lo;
    if (np <= 0) return RISQGPU_OK;
    PanelCount* dc = nullptr;
    PanelBase* db = nullptr;
    ScopedFree<2> release(dc, db);
    RQ_TRY(dalloc(h, dc, (size_t)np));
    RQ_TRY(dalloc(h, db, (size_t)np));
    const int rb = h->tile_rb, cb = h->tile_cb;
    const size_t smem_count = sizeof(int32_t) * MAX_BINS;
    const size_t smem_scatter = sizeof(int32_t) * (MAX_BINS + ((size_t)1 << rb));
    RQ_TRY(allow_smem(h, k_tile_count, smem_count));
    const int grid = (int)std::min<int64_t>(np, (int64_t)num_sms(h) * 2);
    k_tile_count<<<grid, CT, smem_count, h->stream>>>(N, p_lo, p_hi, rb, cb, row_start, base, row_len, cols, dc,
                                                      h->d_row_nleft);
    RQ_TRY(check_launch(h, "tile count"));
    std::vector<PanelCount> pc((size_t)np);
    RQ_CUDA(h, cudaMemcpyAsync(pc.data(), dc, sizeof(PanelCount) * np, cudaMemcpyDeviceToHost, h->stream));
    RQ_TRY(sync(h, "tile count"));
    // a panel: its tiles' pairs, then its leftovers (their first one as `block`)
    std::vector<PanelBase> pb((size_t)np);
    int64_t nt = 0;
    for (int64_t P = 0; P < np; P++) {
        const PanelCount& c = pc[(size_t)P];
        pb[(size_t)P] = PanelBase{stored, nt, stored + c.dense};
        panel_tile[(size_t)(p_lo + P)] = tiles + nt;
        stored += c.dense + c.left;
        dense += c.dense;
        nt += c.tiles;
    }
    if (stored > cap) {
        h->err = "tiled layout: " + std::to_string(stored) + " elements exceed the " + std::to_string(cap) + " slots counted";
        return RISQGPU_ERR_INVALID;
    }
    RQ_CUDA(h, cudaMemcpyAsync(db, pb.data(), sizeof(PanelBase) * np, cudaMemcpyHostToDevice, h->stream));
    parts.push_back({nt, nullptr, nullptr, nullptr, nullptr});
    Part& c = parts.back();
    RQ_TRY(dalloc(h, c.win, (size_t)nt));
    RQ_TRY(dalloc(h, c.off, (size_t)nt));
    RQ_TRY(dalloc(h, c.len, (size_t)nt));
    RQ_TRY(dalloc(h, c.bound, (size_t)nt));
    auto go = [&](auto scatter, auto bounds, auto* vin, auto* val) -> int {
        RQ_TRY(allow_smem(h, scatter, smem_scatter));
        scatter<<<grid, CT, smem_scatter, h->stream>>>(N, p_lo, p_hi, rb, cb, row_start, base, row_len, cols, vin, vlo, db, 0,
                                                       h->d_row_nleft, c.win, nullptr, c.off, c.len, h->d_row_left,
                                                       h->d_el_idx, val, h->d_val_lo, h->d_el_idx, val, h->d_val_lo, row_abs);
        RQ_TRY(check_launch(h, "tile scatter"));
        if (nt == 0) return RISQGPU_OK;
        const size_t smem = (sizeof(uint32_t) << rb) + (sizeof(uint32_t) << cb);
        RQ_TRY(allow_smem(h, bounds, smem));
        bounds<<<(int)std::min<int64_t>(nt, (int64_t)num_sms(h) * 64), TT, smem, h->stream>>>(nt, rb, cb, c.off, c.len,
                                                                                          h->d_el_idx, val, c.bound);
        return check_launch(h, "tile bounds");
    };
    if (precision == RISQGPU_FP64) RQ_TRY(go(k_tile_scatter<double, false>, k_list_bounds<double, false>, v64, h->d_val64));
    else if (precision == RISQGPU_MIXED)
        RQ_TRY(go(k_tile_scatter<float, true>, k_list_bounds<float, true>, v32, h->d_val32));
    else RQ_TRY(go(k_tile_scatter<float, false>, k_list_bounds<float, false>, v32, h->d_val32));
    tiles += nt;
    return RISQGPU_OK;
}

// The chunks' tile records in one array each, and the work space of sigma.
int TileListBuilder::gather() {
    const int64_t N = (int64_t)h->N, np = h->n_panels;
    for (int64_t P = h->part_p_hi; P <= np; P++) panel_tile[(size_t)P] = tiles;
    if (tiles >= INT32_MAX) { h->err = "too many tiles"; return RISQGPU_ERR_INVALID; }
    h->n_tiles = tiles;
    auto gather = [&](auto*& dst, auto Part::*src) -> int {
        using E = typename std::remove_pointer<typename std::remove_reference<decltype(dst)>::type>::type;
        RQ_TRY(dalloc(h, dst, (size_t)tiles));
        int64_t at = 0;
        for (Part& c : parts) {
            if (c.tiles > 0)
                RQ_CUDA(h, cudaMemcpyAsync(dst + at, c.*src, sizeof(E) * c.tiles, cudaMemcpyDeviceToDevice, h->stream));
            at += c.tiles;
            dfree(c.*src);
        }
        return RISQGPU_OK;
    };
    RQ_TRY(gather(h->d_tile_win, &Part::win));
    RQ_TRY(gather(h->d_tile_off, &Part::off));
    RQ_TRY(gather(h->d_tile_len, &Part::len));
    RQ_TRY(gather(h->d_tile_bound, &Part::bound));
    RQ_TRY(dalloc(h, h->d_panel_tile, (size_t)np + 1));
    const bool f64 = precision == RISQGPU_FP64;
    RQ_TRY(dalloc_reduced(h, h->d_acc, (size_t)(f64 ? N : N + (N + 1) / 2)));
    RQ_TRY(dalloc(h, h->d_sig_scalars, 5));
    return dalloc(h, h->d_wmax, (size_t)((N - 1) >> std::min(h->tile_rb, h->tile_cb)) + 1);
}

int TileListBuilder::finish() {
    const int64_t N = (int64_t)h->N, np = h->n_panels;
    RQ_CUDA(h, cudaMemcpyAsync(h->d_panel_tile, panel_tile.data(), sizeof(int64_t) * (np + 1), cudaMemcpyHostToDevice,
                               h->stream));
    RQ_CUDA(h, cudaMemsetAsync(h->d_sig_scalars, 0, sizeof(double) * 5, h->stream));
    // row sums of |H| over both triangles: with a partition each rank holds part of every
    // row's sum, so the exact integer sums are added across the ranks first
    if (h->part_n > 1) RQ_TRY(part_allreduce(h, row_abs, (size_t)N));
    k_max_u64<<<grid_n(h, N), 256, 0, h->stream>>>(row_abs, N, absmax);
    RQ_TRY(check_launch(h, "row sums"));
    unsigned long long mi = 0;
    std::vector<int32_t> len((size_t)tiles), nl((size_t)N);
    RQ_CUDA(h, cudaMemcpyAsync(&mi, absmax, sizeof(mi), cudaMemcpyDeviceToHost, h->stream));
    RQ_CUDA(h, cudaMemcpyAsync(len.data(), h->d_tile_len, sizeof(int32_t) * tiles, cudaMemcpyDeviceToHost, h->stream));
    RQ_CUDA(h, cudaMemcpyAsync(nl.data(), h->d_row_nleft, sizeof(int32_t) * N, cudaMemcpyDeviceToHost, h->stream));
    RQ_TRY(sync(h, "row sums"));
    // each |H_pq| was rounded to a multiple of 2^-32: the margin covers that rounding
    h->h_row_abs_max = 1.01 * ((double)mi / 4294967296.0) + 1e-6;
    h->n_dense_el = (uint64_t)dense;
    h->tiled = h->tile_list = true;
    // units: runs of a panel's tiles of about `target` pairs, and rows with leftovers
    std::vector<SigmaUnit> us;
    std::vector<int64_t> weight;
    const int64_t R = (int64_t)1 << h->tile_rb, target = std::max<int64_t>(32768, stored / ((int64_t)num_sms(h) * 64));
    for (int64_t P = h->part_p_lo; P < h->part_p_hi; P++) {
        int64_t acc = 0;
        int32_t lo = (int32_t)panel_tile[(size_t)P];
        const int32_t end = (int32_t)panel_tile[(size_t)P + 1];
        for (int32_t t = lo; t < end; t++) {
            acc += len[(size_t)t];
            if (acc < target && t + 1 < end) continue;
            us.push_back({lo, (int32_t)P, lo, t + 1, 0});
            weight.push_back(acc);
            lo = t + 1;
            acc = 0;
        }
        left_units(us, weight, nl, P, R, N, target);
    }
    return set_units(h, us, weight, target);
}

TileListBuilder::~TileListBuilder() {
    dfree(row_abs);
    dfree(absmax);
    for (Part& c : parts) {
        dfree(c.win);
        dfree(c.off);
        dfree(c.len);
        dfree(c.bound);
    }
}

TileBuilder::~TileBuilder() {
    dfree(left_cur);
    dfree(sums);
    dfree(counters);
}

// sigma over tiled storage; kind 0: FP64 vectors (FP64 values, or FP32 + remainder),
// 1: FP32 vectors with the FP32 values.  FP32 vectors sum across tiles in FP32 unless the
// handle asked for reproducible sums or is partitioned (the ranks' sums must add exactly).
int sigma_tiles(risqgpu* h, const void* x, void* y, int kind) {
    if (kind == 0) {
        if (h->precision == RISQGPU_FP64)
            return launch_fx<double, double, false, true>(h, (const double*)x, (double*)y, h->d_left64, nullptr);
        if (h->precision == RISQGPU_MIXED)
            return launch_fx<double, float, true, true>(h, (const double*)x, (double*)y, h->d_left32, h->d_left_lo);
        h->err = "FP64 sigma needs FP64 or FP32 + remainder values";
        return RISQGPU_ERR_INVALID;
    }
    if (h->precision == RISQGPU_FP64) {
        h->err = "FP32 sigma needs FP32 values";
        return RISQGPU_ERR_INVALID;
    }
    if (!h->reproducible && h->part_n == 1)
        return launch_fx<float, float, false, false>(h, (const float*)x, (float*)y, h->d_left32, nullptr);
    return launch_fx<float, float, false, true>(h, (const float*)x, (float*)y, h->d_left32, nullptr);
}

// Every stored pair of a tiled build as (p, q, value), internal indices, in no particular
// order (nnz_upper entries each).
int tiles_coo(risqgpu* h, int32_t* p, int32_t* q, double* v) {
    unsigned long long* count = nullptr;
    ScopedFree<1> release(count);
    RQ_TRY(dalloc(h, count, 1));
    RQ_CUDA(h, cudaMemsetAsync(count, 0, sizeof(unsigned long long), h->stream));
    return tiles_each(h, CooOut{p, q, v, count, h->nnz_upper});
}

// out[i] -= sum_j H_ij^2 / max(H_jj - E, gmin) over the stored pairs (out zeroed by the caller).
int tiles_self_energy(risqgpu* h, double energy, double gmin, double* out) {
    return tiles_each(h, SelfEnergyAdd{h->d_diag, energy, gmin, out});
}

int tiles_rows(risqgpu* h, const uint32_t* mark, int64_t* out_r, int64_t* out_c, double* out_v,
               unsigned long long* count, unsigned long long cap) {
    return tiles_each(h, RowFilter{mark, h->d_orig, out_r, out_c, out_v, count, cap});
}

void free_tiles(risqgpu* h) {
    dfree(h->d_panel_tile);
    dfree(h->d_tile_bound);
    dfree(h->d_units);
    h->n_units = 0;
    dfree(h->d_tile_win);
    dfree(h->d_tile_blk);
    dfree(h->d_tile_blocks);
    dfree(h->d_tile_off);
    dfree(h->d_tile_len);
    dfree(h->d_el_idx);
    for (TileChunk& ch : h->chunks) {
        dfree(ch.grp_off);
        dfree(ch.slots);
        dfree(ch.col);
        dfree(ch.val);
        dfree(ch.lo);
    }
    h->chunks.clear();
    dfree(h->d_chunk_tab);
    dfree(h->d_left_off);
    dfree(h->d_left_len);
    dfree(h->d_left_col);
    dfree(h->d_left_row);
    dfree(h->d_left64);
    dfree(h->d_row_left);
    dfree(h->d_row_nleft);
    dfree(h->d_left32);
    dfree(h->d_left_lo);
    dfree(h->d_acc);
    dfree(h->d_wmax);
    dfree(h->d_sig_scalars);
    h->tiled = h->tile_list = false;
    h->n_panels = h->n_tiles = 0;
    h->n_dense_el = 0;
    h->h_row_abs_max = 0.0;
}

}  // namespace risq
