// Upper-triangle tiles as plain pair lists (included by tiles.cu).
//
// The layout of tiles.cu pads short rows and heads every group of 32 slots, so a set whose
// tiles hold few pairs a row takes up to 24 bytes a pair there.  Where that does not fit, the
// tiles are lists of pairs instead, coded (row in panel << cb | column in window): 4 bytes and
// the value, whatever the set.  Nothing is arranged, so a build needs besides the lists only
// a chunk of CSR rows.  A pair costs two shared loads and, for FP32 vectors, two shared
// atomics (one for each row of a lane's four pairs) instead of one each.  Sigma, against the
// groups: 551,147 determinants FP32 893 us (692), FP32 + remainder 1740 us (1180); 8,300,003
// determinants 27.5 ms (24.6) and 57.4 ms (43.3).
#pragma once

template <typename V>
struct ListView {
    int rb, cb, wb;  // log2 of the rows of a panel, the columns of a window, the entries per max |x|
    const int64_t* __restrict__ panel_tile;
    const int32_t* __restrict__ win;
    const int64_t* __restrict__ off;     // first pair and pairs of each tile
    const int32_t* __restrict__ len;
    const float2* __restrict__ bound;    // largest row and column sum of |H| of each tile
    const int64_t* __restrict__ row_left;  // leftovers of each row
    const int32_t* __restrict__ row_nleft;
    const uint32_t* __restrict__ code;   // of a leftover: its column
    const V* __restrict__ val;
    const float* __restrict__ lo;
};

// Largest row and column sum of |H| of every tile, in integers, every element rounded up.
template <typename V, bool VLO>
__global__ void __launch_bounds__(TT) k_list_bounds(int64_t nt, int rb, int cb, const int64_t* __restrict__ off,
                                                    const int32_t* __restrict__ len, const uint32_t* __restrict__ code,
                                                    const V* __restrict__ val, float2* __restrict__ bound) {
    extern __shared__ __align__(16) unsigned char sm[];
    uint32_t* sum = reinterpret_cast<uint32_t*>(sm);  // R row sums, C column sums
    __shared__ uint32_t s_max[3];
    const int R = 1 << rb, C = 1 << cb;
    for (int64_t t = blockIdx.x; t < nt; t += gridDim.x) {
        for (int i = threadIdx.x; i < R + C; i += TT) sum[i] = 0;
        if (threadIdx.x < 3) s_max[threadIdx.x] = 0;
        __syncthreads();
        const int64_t e0 = off[t];
        const int E = len[t];
        float vmax = 0.f;
        for (int i = threadIdx.x; i < E; i += TT) vmax = fmaxf(vmax, __double2float_ru(fabs((double)val[e0 + i])));
        const uint32_t bits = __reduce_max_sync(FULL, __float_as_uint(vmax));
        if ((threadIdx.x & 31) == 0) atomicMax(s_max + 2, bits);
        __syncthreads();
        vmax = __uint_as_float(s_max[2]);
        int ex = 0;
        if (vmax > 0.f) frexpf(vmax, &ex);
        const int u = 31 - max(rb, cb) - 1 - ex;
        const double unit = ldexp(1.0, u);
        for (int i = threadIdx.x; i < E; i += TT) {
            const uint32_t cd = code[e0 + i];
            const uint32_t a = (uint32_t)__double2ll_ru(fabs((double)val[e0 + i]) * unit) + (VLO ? 1u : 0u);
            atomicAdd(sum + (cd >> cb), a);
            atomicAdd(sum + R + (cd & ((uint32_t)C - 1u)), a);
        }
        __syncthreads();
        uint32_t rm = 0, cm = 0;
        for (int i = threadIdx.x; i < R; i += TT) rm = max(rm, sum[i]);
        for (int i = threadIdx.x; i < C; i += TT) cm = max(cm, sum[R + i]);
        rm = __reduce_max_sync(FULL, rm);
        cm = __reduce_max_sync(FULL, cm);
        if ((threadIdx.x & 31) == 0) {
            atomicMax(s_max, rm);
            atomicMax(s_max + 1, cm);
        }
        __syncthreads();
        if (threadIdx.x == 0)
            bound[t] = make_float2(__double2float_ru(ldexp((double)s_max[0], -u)), __double2float_ru(ldexp((double)s_max[1], -u)));
        __syncthreads();
    }
}

// Sigma over the lists: as k_sigma_fx, with the row sums of a tile in shared memory too (FP64
// vectors: high parts and low lbr bits apart, like the columns').  A work unit is a run of a
// panel's tiles, whose row sums gather at the scale 2^S, or rows of a panel's leftovers.
template <typename X, typename V, bool VLO, bool EXACT>
__global__ void __launch_bounds__(ST, sizeof(X) == 4 ? 4 : 2)
    k_sigma_list(int64_t N, int64_t n_units, const SigmaUnit* __restrict__ units, ListView<V> T, const X* __restrict__ x,
                 const double* __restrict__ wmax, void* __restrict__ acc_out, unsigned long long* __restrict__ acc_row,
                 double* __restrict__ scalars, const int* __restrict__ stop) {
    if (stop && *stop) return;
    constexpr bool DBL = std::is_same<X, double>::value;
    extern __shared__ __align__(16) unsigned char sm[];
    const int R = 1 << T.rb, C = 1 << T.cb, lb = 32 - T.rb, lbr = 32 - T.cb;
    X* xP = reinterpret_cast<X*>(sm);
    X* xJ = xP + R;
    long long* yP = reinterpret_cast<long long*>(xJ + C);  // row sums of the unit
    int* yRa = reinterpret_cast<int*>(yP + R);
    int* yJa = yRa + R;
    unsigned* yRb = reinterpret_cast<unsigned*>(yJa + C);  // FP64 vectors
    unsigned* yJb = yRb + R;
    __shared__ long long s_unit;
    const int lane = threadIdx.x & 31;
    const double gscale = scalars[1];  // 2^S
    const int S = ilogb(gscale);
    unsigned long long* counter = reinterpret_cast<unsigned long long*>(scalars) + 3;
    unsigned long long* acc_ll = reinterpret_cast<unsigned long long*>(acc_out);
    X* acc_x = reinterpret_cast<X*>(acc_out);
    auto max_of = [&](int64_t i0, int64_t i1) {
        double m = 0.0;
        for (int64_t b = i0 >> T.wb; b << T.wb < i1; b++) m = fmax(m, wmax[b]);
        return m;
    };
    for (;;) {
        if (threadIdx.x == 0) s_unit = (long long)atomicAdd(counter, 1ull);
        __syncthreads();
        if (s_unit >= n_units) break;
        const SigmaUnit u = units[s_unit];
        const int64_t r0 = (int64_t)u.panel << T.rb;
        if (u.tile < 0) {
            // leftover pairs: one warp per row, private row sum, column sums of the rounded products
            for (int64_t p = r0 + u.lo + (threadIdx.x >> 5); p < r0 + u.hi; p += ST / 32) {
                const int64_t s = T.row_left[p];
                const int len = T.row_nleft[p];
                if (len == 0) continue;
                const X xp = __ldg(x + p);
                double rs = 0.0;
                for (int k = lane; k < len; k += 32) {
                    const uint32_t q = __ldcs(T.code + s + k);
                    X v = (X)__ldcs(T.val + s + k);
                    if constexpr (VLO) v += (X)__ldcs(T.lo + s + k);
                    rs += (double)(v * __ldg(x + q));
                    if constexpr (EXACT) atomicAdd(acc_ll + q, (unsigned long long)llrint((double)(v * xp) * gscale));
                    else atomicAdd(acc_x + q, v * xp);
                }
                // fixed lane order: the warp sum does not depend on timing
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) rs += __shfl_xor_sync(FULL, rs, o);
                if (lane == 0) atomicAdd(acc_row + p, (unsigned long long)llrint(rs * gscale));
            }
            __syncthreads();
            continue;
        }
        const int nr = (int)min((int64_t)R, N - r0);
        const double xm = max_of(r0, r0 + nr);
        stage_window<X>(xP, x + r0, nr);
        for (int i = threadIdx.x; i < R; i += ST) {
            yP[i] = 0;
            yRa[i] = 0;
            if constexpr (DBL) yRb[i] = 0u;
        }
        for (int t = u.lo; t < u.hi; t++) {
            const int64_t c0 = (int64_t)T.win[t] << T.cb;
            const int w = (int)min((int64_t)C, N - c0);
            const float2 bound = T.bound[t];
            int sh = fixed_shift32((double)bound.y * xm, DBL ? 800 : 120);
            const int rsh = min(DBL ? S - lbr : S, fixed_shift32((double)bound.x * max_of(c0, c0 + w), DBL ? 800 : 120));
            if constexpr (EXACT) sh = min(sh, DBL ? S - lb : S);
            const X csc = (X)ldexp(1.0, DBL ? sh + lb : sh), rsc = (X)ldexp(1.0, DBL ? rsh + lbr : rsh);
            stage_window<X>(xJ, x + c0, w);
            for (int i = threadIdx.x; i < w; i += ST) {
                yJa[i] = 0;
                if constexpr (DBL) yJb[i] = 0u;
            }
            __syncthreads();
            const int64_t e0 = T.off[t];
            const int E = T.len[t];
            const uint32_t cmask = (uint32_t)C - 1u;
            using RS = typename std::conditional<DBL, long long, int>::type;
            auto add_row = [&](uint32_t r, RS q) {
                if constexpr (DBL) {
                    atomicAdd(yRa + r, (int)(q >> lbr));
                    atomicAdd(yRb + r, (unsigned)q & ((1u << lbr) - 1u));
                } else atomicAdd(yRa + r, q);
            };
            // a pair's column sum; returns its part of the row sum
            auto add_col = [&](uint32_t cd, X v) -> RS {
                const uint32_t r = cd >> T.cb, c = cd & cmask;
                if constexpr (DBL) {
                    const long long q = __double2ll_rn(v * (xP[r] * csc));
                    atomicAdd(yJa + c, (int)(q >> lb));
                    atomicAdd(yJb + c, (unsigned)q & ((1u << lb) - 1u));
                    return __double2ll_rn(v * xJ[c] * rsc);
                } else {
                    atomicAdd(yJa + c, __float2int_rn(v * (xP[r] * csc)));
                    return __float2int_rn(v * xJ[c] * rsc);
                }
            };
            // Pairs of a row follow one another: a lane takes four, and adds what falls in one row
            // at once.  Aligned vectors of four, those before and after them one by one.
            const int head = min(E, (int)((4 - (e0 & 3)) & 3)), nblk = (E - head) >> 2, rest = E - head - 4 * nblk;
            if ((int)threadIdx.x < head + rest) {
                const int64_t e = (int)threadIdx.x < head ? e0 + threadIdx.x : e0 + 4 * nblk + threadIdx.x;
                const uint32_t cd = __ldcs(T.code + e);
                X v = (X)__ldcs(T.val + e);
                if constexpr (VLO) v += (X)__ldcs(T.lo + e);
                add_row(cd >> T.cb, add_col(cd, v));
            }
            auto four = [&](const uint4 c4, const X (&v)[4]) {
                const uint32_t cd[4] = {c4.x, c4.y, c4.z, c4.w};
                uint32_t r = cd[0] >> T.cb;
                RS sum = 0;
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const RS q = add_col(cd[k], v[k]);
                    if (cd[k] >> T.cb != r) {
                        add_row(r, sum);
                        r = cd[k] >> T.cb;
                        sum = 0;
                    }
                    sum += q;
                }
                add_row(r, sum);
            };
            auto load4 = [&](int64_t e, X (&v)[4]) {
                X a[2], b[2];
                load2<V, X, VLO>(T.val + e, T.lo + (VLO ? e : 0), a);
                load2<V, X, VLO>(T.val + e + 2, T.lo + (VLO ? e + 2 : 0), b);
                v[0] = a[0];
                v[1] = a[1];
                v[2] = b[0];
                v[3] = b[1];
            };
            for (int bk = threadIdx.x; bk < nblk; bk += 2 * ST) {
                const int64_t e1 = e0 + head + 4 * (int64_t)bk, e2 = e1 + 4 * ST;
                const bool two = bk + ST < nblk;
                X v1[4], v2[4];
                const uint4 c1 = __ldcs(reinterpret_cast<const uint4*>(T.code + e1));
                load4(e1, v1);
                uint4 c2;
                if (two) {
                    c2 = __ldcs(reinterpret_cast<const uint4*>(T.code + e2));
                    load4(e2, v2);
                }
                four(c1, v1);
                if (two) four(c2, v2);
            }
            __syncthreads();
            for (int i = threadIdx.x; i < nr; i += ST) {
                long long q = yRa[i];
                if constexpr (DBL) q = (q << lbr) + (long long)yRb[i];
                if (q != 0) {
                    yP[i] += q << (DBL ? S - rsh - lbr : S - rsh);
                    yRa[i] = 0;
                    if constexpr (DBL) yRb[i] = 0u;
                }
            }
            const float inv = ldexpf(1.f, EXACT ? 0 : -sh);
            for (int i = threadIdx.x; i < w; i += ST) {
                if constexpr (EXACT) {
                    long long q = yJa[i];
                    if constexpr (DBL) q = (q << lb) + (long long)yJb[i];
                    if (q != 0) atomicAdd(acc_ll + c0 + i, (unsigned long long)(q << (DBL ? S - sh - lb : S - sh)));
                } else {
                    if (yJa[i] != 0) atomicAdd(acc_x + c0 + i, (float)yJa[i] * inv);
                }
            }
            __syncthreads();
        }
        for (int i = threadIdx.x; i < nr; i += ST)
            if (yP[i] != 0) atomicAdd(acc_row + r0 + i, (unsigned long long)yP[i]);
        __syncthreads();
    }
}

// Calls f(p, q, v) for every stored pair (as k_tiles_each).
template <typename V, bool VLO, typename F>
__global__ void __launch_bounds__(TT) k_list_each(int64_t N, int64_t p_lo, int64_t p_hi, ListView<V> T, F f) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto value = [&](int64_t e) {
        double v = (double)T.val[e];
        if constexpr (VLO) v += (double)T.lo[e];
        return v;
    };
    for (int64_t P = p_lo + blockIdx.x; P < p_hi; P += gridDim.x) {
        const int64_t r0 = P << T.rb;
        for (int64_t t = T.panel_tile[P]; t < T.panel_tile[P + 1]; t++) {
            const int64_t c0 = (int64_t)T.win[t] << T.cb;
            for (int i = threadIdx.x; i < T.len[t]; i += TT) {
                const uint32_t cd = T.code[T.off[t] + i];
                f(r0 + (cd >> T.cb), c0 + (cd & ((1u << T.cb) - 1u)), value(T.off[t] + i));
            }
        }
        for (int64_t p = r0 + warp; p < min(N, r0 + ((int64_t)1 << T.rb)); p += TT / 32)
            for (int k = lane; k < T.row_nleft[p]; k += 32)
                f(p, (int64_t)T.code[T.row_left[p] + k], value(T.row_left[p] + k));
    }
}

template <typename V>
ListView<V> list_view(risqgpu* h) {
    const V* val;
    if constexpr (std::is_same<V, double>::value) val = h->d_val64;
    else val = h->d_val32;
    return ListView<V>{h->tile_rb, h->tile_cb, std::min(h->tile_rb, h->tile_cb), h->d_panel_tile, h->d_tile_win,
                       h->d_tile_off, h->d_tile_len, h->d_tile_bound, h->d_row_left, h->d_row_nleft, h->d_el_idx, val,
                       h->d_val_lo};
}
