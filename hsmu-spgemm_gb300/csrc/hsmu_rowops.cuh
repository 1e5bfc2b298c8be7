// Per-row routines for rows with few intermediate products ("tiny" rows:
// at most TINY_MAX products), one thread per row.
//
// The AMG Galerkin operands (A*P: <= 7 products per row, P^T*(AP): <= 32)
// and the 2-D Laplacian (<= 25) consist of such rows only; a warp per row
// would leave most lanes idle.  The count pass and the fill pass need no B
// tiles: a thread lists its row's products in the oracle's order (A entry,
// then B entry) and sorts them by column in registers, stable by product.
// Every product is added to its column's sum in that order: 0.0 + p_1 + p_2
// + ... (arithmetic per step as in hsmu_products.cuh), bit-identical to the
// host oracle.  The batched engine's general rows, and matrices of more
// columns than a sort key holds, keep sorted insertion lists instead.
//
// The per-thread lists live in shared memory laid out element-major
// ([TINY_MAX][threads]) so that neighbouring threads hit neighbouring banks.
//
// B's row k is given as entries brp[k] .. bre[k]-1 (bre = brp + 1 for a CSR
// row pointer).
#pragma once
#include "hsmu_products.cuh"

namespace hsmu {

constexpr int TINY_MAX = 32;

// Batcher's odd-even merge sort of N keys in registers: the pairs that are compared
template <int N>
struct SortNet {
    int n = 0, x[8 * N] = {}, y[8 * N] = {};
    constexpr SortNet() {
        for (int p = 1; p < N; p *= 2)
            for (int k = p; k >= 1; k /= 2)
                for (int j = k % p; j + k < N; j += 2 * k)
                    for (int i = 0; i < k && i + j + k < N; i++)
                        if ((i + j) / (2 * p) == (i + j + k) / (2 * p)) {
                            x[n] = i + j;
                            y[n] = i + j + k;
                            n++;
                        }
    }
};
template <int N>
__device__ __forceinline__ void sort_keys(unsigned (&key)[N]) {
    constexpr SortNet<N> NET{};
    constexpr int SIZE = NET.n;
#pragma unroll
    for (int c = 0; c < SIZE; c++) {
        const unsigned lo = min(key[NET.x[c]], key[NET.y[c]]), hi = max(key[NET.x[c]], key[NET.y[c]]);
        key[NET.x[c]] = lo;
        key[NET.y[c]] = hi;
    }
}

// A entries of a tiny row handled per batch: their column ids, B row bounds
// and first B entries are fetched in three rounds of independent loads
// before any of them is used (a thread would otherwise wait for ~3 dependent
// memory round trips per A entry)
constexpr int TINY_BATCH = 8;

template <bool NC, bool VALS>
struct TinyFetch {
    int qs[TINY_BATCH], qe[TINY_BATCH], j0[TINY_BATCH];
    double a[TINY_BATCH], b0[TINY_BATCH];

    __device__ __forceinline__ void load(int p0, int a_hi, const int *__restrict__ acol,
                                         const double *__restrict__ aval, const int *__restrict__ brp,
                                         const int *__restrict__ bre, const int *__restrict__ bcol,
                                         const double *__restrict__ bval) {
        int k[TINY_BATCH];
#pragma unroll
        for (int u = 0; u < TINY_BATCH; u++) {
            k[u] = p0 + u < a_hi ? ldx<NC>(acol + p0 + u) : -1;
            if (VALS) a[u] = p0 + u < a_hi ? ldx<NC>(aval + p0 + u) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < TINY_BATCH; u++) {
            qs[u] = qe[u] = 0;
            if (k[u] >= 0) {
                qs[u] = ldx<NC>(brp + k[u]);
                qe[u] = ldx<NC>(bre + k[u]);
            }
        }
#pragma unroll
        for (int u = 0; u < TINY_BATCH; u++) {
            j0[u] = 0;
            b0[u] = 0.0;
            if (qs[u] < qe[u]) {
                j0[u] = ldx<NC>(bcol + qs[u]);
                if (VALS) b0[u] = ldx<NC>(bval + qs[u]);
            }
        }
    }
};

// A warp's rows as flat product lists, one row per lane (element-major, as above): tiny_list writes every
// product's place in B and the A value, then all products are loaded at once and their columns sorted by a
// network of the size that the warp's longest row needs.  An insertion list costs a chain of shared-memory
// steps per product, and every entry of a B row after the first is a memory round trip of its own
// (150,001 random rows of 12 entries on average: fill 83 -> 26 us, count 45 -> 6.5; 2-D Laplacian of side 256,
// 25 products per row: 21.5 -> 18.0 and 7.9 -> 5.7: the fill there is FP64 issue, 6 us, and
// each lane's stores to its own row).
template <int AR>
struct TinySmem {
    double t[TINY_MAX][WARP];  // the A value, then add_term's term, of every product
    double a[AR == AR_FMA ? TINY_MAX : 1][WARP];  // its A value (fused multiply-add)
    int q[TINY_MAX][WARP];     // its entry of B
};
// sort keys are column << 5 | product, below the empty key
constexpr int TINY_KEY_COLS = (1 << 27) - 1;

// the number of products of the lane's row, listed; more than TINY_MAX if there are more
template <bool VALS>
__device__ __forceinline__ int tiny_list(int a_lo, int a_hi, const int *__restrict__ acol,
                                         const double *__restrict__ aval, const int *__restrict__ brp,
                                         int (*qs)[WARP], double (*t)[WARP]) {
    const int lane = lane_id();
    int n = 0;
    for (int p0 = a_lo; p0 < a_hi && n <= TINY_MAX; p0 += TINY_BATCH) {
        int s[TINY_BATCH], e[TINY_BATCH];
        double a[TINY_BATCH];
#pragma unroll
        for (int u = 0; u < TINY_BATCH; u++) {
            s[u] = p0 + u < a_hi ? __ldg(acol + p0 + u) : -1;
            if (VALS) a[u] = p0 + u < a_hi ? __ldg(aval + p0 + u) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < TINY_BATCH; u++) {
            const int k = s[u];
            s[u] = e[u] = 0;
            if (k >= 0) {
                s[u] = __ldg(brp + k);
                e[u] = __ldg(brp + k + 1);
            }
        }
#pragma unroll
        for (int u = 0; u < TINY_BATCH; u++) {
            const int m = min(e[u] - s[u], TINY_MAX - n);
            for (int i = 0; i < m; i++) {
                qs[n + i][lane] = s[u] + i;
                if (VALS) t[n + i][lane] = a[u];
            }
            n += e[u] - s[u];
        }
    }
    return n;
}

// distinct columns of the lane's n <= N listed products
template <int N>
__device__ __forceinline__ int tiny_list_count(int n, const int *__restrict__ bcol, const int (*qs)[WARP]) {
    unsigned key[N];
#pragma unroll
    for (int u = 0; u < N; u++) key[u] = u < n ? (unsigned)__ldg(bcol + qs[u][lane_id()]) : ~0u;
    sort_keys<N>(key);
    int c = 0;
#pragma unroll
    for (int u = 0; u < N; u++) c += key[u] != ~0u && (u == 0 || key[u] != key[u - 1]);
    return c;
}

// The lane's n <= N listed products sorted by column (stable by product), summed run by run and written,
// at most cap entries; returns the distinct columns.
template <int AR, int N>
__device__ __forceinline__ int tiny_list_fill(int n, const int *__restrict__ bcol, const double *__restrict__ bval,
                                              TinySmem<AR> &S, int cap, int *__restrict__ oc,
                                              double *__restrict__ ov) {
    const int lane = lane_id();
    unsigned key[N];
#pragma unroll
    for (int u = 0; u < N; u++) key[u] = u < n ? ((unsigned)__ldg(bcol + S.q[u][lane]) << 5) | (unsigned)u : ~0u;
#pragma unroll
    for (int u0 = 0; u0 < N; u0 += 8) {
        double b[8];
#pragma unroll
        for (int i = 0; i < 8; i++) b[i] = u0 + i < n ? __ldg(bval + S.q[u0 + i][lane]) : 0.0;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            if (u0 + i < n) {
                const double a = S.t[u0 + i][lane];
                if (AR == AR_FMA) S.a[u0 + i][lane] = a;
                S.t[u0 + i][lane] = term<AR>(a, b[i]);
            }
        }
    }
    sort_keys<N>(key);
    int at = -1;
    double acc = 0.0;
#pragma unroll
    for (int u = 0; u < N; u++) {
        if (key[u] != ~0u) {
            const bool head = u == 0 || key[u] >> 5 != key[u - 1] >> 5;
            const int o = (int)(key[u] & 31u);
            at += head;
            acc = add_term<AR>(head ? 0.0 : acc, AR == AR_FMA ? S.a[o][lane] : 0.0, S.t[o][lane]);
            if ((u == N - 1 || key[u + 1 < N ? u + 1 : u] >> 5 != key[u] >> 5) && at < cap) {
                oc[at] = (int)(key[u] >> 5);
                ov[at] = acc;
            }
        }
    }
    return at + 1;
}

// A row with one entry of A (value a): its B row [s, e), already in order, is the row of C.  Writes at most cap
// entries; returns the row's number.  Where a warp has only such rows nothing is listed or sorted (three million
// rows that each take one of 27 entries: count 136 -> 27 us, fill 1,505 -> 1,141; two million of 15 on average:
// 88 -> 16 and 644 -> 458; insertion lists took 226 and 1,141, and 114 and 526).
template <int AR>
__device__ __forceinline__ int tiny_copy_fill(int s, int e, double a, const int *__restrict__ bcol,
                                              const double *__restrict__ bval, int cap, int *__restrict__ oc,
                                              double *__restrict__ ov) {
    const int n = e - s, m = min(n, cap);
    for (int u0 = 0; u0 < m; u0 += 8) {
        int c[8];
        double b[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            c[i] = u0 + i < m ? __ldg(bcol + s + u0 + i) : 0;
            b[i] = u0 + i < m ? __ldg(bval + s + u0 + i) : 0.0;
        }
#pragma unroll
        for (int i = 0; i < 8; i++) {
            if (u0 + i < m) {
                oc[u0 + i] = c[i];
                ov[u0 + i] = add_term<AR>(0.0, a, term<AR>(a, b[i]));
            }
        }
    }
    return n;
}

// Builds the row's sorted distinct columns and their accumulated values in
// the thread's list (cols/acc, element stride `stride`, TINY_MAX entries) and
// returns its length; returns -1 (list contents undefined) when the row has
// more than `limit` products (limit <= TINY_MAX).
template <int AR, bool NC = true>
__device__ __forceinline__ int tiny_row_build(int a_lo, int a_hi, const int *__restrict__ acol,
                                              const double *__restrict__ aval, const int *__restrict__ brp,
                                              const int *__restrict__ bre, const int *__restrict__ bcol,
                                              const double *__restrict__ bval, int *cols, double *acc, int stride,
                                              int limit) {
    int n = 0, seen = 0;
    for (int p0 = a_lo; p0 < a_hi; p0 += TINY_BATCH) {
        TinyFetch<NC, true> F;
        F.load(p0, a_hi, acol, aval, brp, bre, bcol, bval);
#pragma unroll
        for (int u = 0; u < TINY_BATCH; u++) {
            const double a = F.a[u];
            for (int q = F.qs[u]; q < F.qe[u]; q++) {
                if (++seen > limit) return -1;
                const bool first = q == F.qs[u];
                const int j = first ? F.j0[u] : ldx<NC>(bcol + q);
                const double pr = term<AR>(a, first ? F.b0[u] : ldx<NC>(bval + q));
                int pos = n;
                while (pos > 0 && cols[(pos - 1) * stride] > j) pos--;
                if (pos > 0 && cols[(pos - 1) * stride] == j) {
                    acc[(pos - 1) * stride] = add_term<AR>(acc[(pos - 1) * stride], a, pr);
                    continue;
                }
                for (int t = n; t > pos; t--) {
                    cols[t * stride] = cols[(t - 1) * stride];
                    acc[t * stride] = acc[(t - 1) * stride];
                }
                cols[pos * stride] = j;
                acc[pos * stride] = add_term<AR>(0.0, a, pr);
                n++;
            }
        }
    }
    return n;
}

// copies a list built by tiny_row_build to out_col/out_val
__device__ __forceinline__ void tiny_row_write(const int *cols, const double *acc, int stride, int n,
                                               int *__restrict__ out_col, double *__restrict__ out_val) {
    for (int t = 0; t < n; t++) {
        out_col[t] = cols[t * stride];
        out_val[t] = acc[t * stride];
    }
}

// Fills the row's sorted columns and values at out_col/out_val and returns
// its nnz; returns -1 on an inconsistency (more than TINY_MAX products, or
// more than `cap` distinct columns).
template <int AR, bool NC = true>
__device__ __forceinline__ int tiny_row_fill(int a_lo, int a_hi, const int *__restrict__ acol,
                                             const double *__restrict__ aval, const int *__restrict__ brp,
                                             const int *__restrict__ bre, const int *__restrict__ bcol,
                                             const double *__restrict__ bval, int *cols, double *acc, int stride,
                                             int cap, int *__restrict__ out_col,
                                             double *__restrict__ out_val) {
    const int n = tiny_row_build<AR, NC>(a_lo, a_hi, acol, aval, brp, bre, bcol, bval, cols, acc, stride, TINY_MAX);
    if (n < 0 || n > cap) return -1;
    tiny_row_write(cols, acc, stride, n, out_col, out_val);
    return n;
}

// ---------------------------------------------------------------------------
// Warp-per-row routines on a dense span table, driven by B's entries (no B
// tiles): used by the batched engine, where B may be produced inside the same
// launch.  msk[] holds SPAN_T u64 masks, base[] SPAN_T ints, acc[] `cap`
// doubles, all private to the warp.

// first and last column of row (a_lo..a_hi) of A*B: min/max over the first /
// last entries of the referenced (sorted) B rows; returns products too.
template <bool NC = true>
__device__ __forceinline__ void warp_row_extent(int a_lo, int a_hi, const int *__restrict__ acol,
                                                const int *__restrict__ brp, const int *__restrict__ bre,
                                                const int *__restrict__ bcol, int &cmin, int &cmax, int &prod) {
    cmin = 0x7fffffff;
    cmax = -1;
    prod = 0;
    for (int p = a_lo + lane_id(); p < a_hi; p += WARP) {
        const int k = ldx<NC>(acol + p);
        const int s = ldx<NC>(brp + k), e = ldx<NC>(bre + k);
        if (e > s) {
            cmin = min(cmin, ldx<NC>(bcol + s));
            cmax = max(cmax, ldx<NC>(bcol + e - 1));
            prod += e - s;
        }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        cmin = min(cmin, __shfl_xor_sync(FULL, cmin, d));
        cmax = max(cmax, __shfl_xor_sync(FULL, cmax, d));
        prod += __shfl_xor_sync(FULL, prod, d);
    }
}

// OR the row's columns into msk[0..span) (tile t0 + i at msk[i]).  Without
// CLIP a column outside the span is an error (returns false); with CLIP each
// B row is first cut to the span's columns (two binary searches), so a wide
// row can be taken one column window at a time.
template <bool NC = true, bool CLIP = false>
__device__ __forceinline__ bool warp_row_masks(int a_lo, int a_hi, const int *__restrict__ acol,
                                               const int *__restrict__ brp, const int *__restrict__ bre,
                                               const int *__restrict__ bcol, int t0,
                                               int span, unsigned long long *msk) {
    for (int t = lane_id(); t < span; t += WARP) msk[t] = 0ull;
    __syncwarp();
    bool bad = false;
    const int c0 = CLIP ? t0 << 6 : 0;
    const int c1 = CLIP ? (int)min((long long)(t0 + span) << 6, (long long)INT_MAX) : 0;
    warp_walk_tiles<CLIP, NC>(a_lo, a_hi, 0, WARP, acol, brp, bre, bcol, c0, c1, [&](int q) {
        const int j = ldx<NC>(bcol + q);
        const int t = (j >> 6) - t0;
        if (t >= 0 && t < span) smem_setbit64(msk + t, j & 63);
        else bad = true;
    });
    __syncwarp();
    return !__any_sync(FULL, bad);
}

// nnz of the masks
__device__ __forceinline__ int warp_mask_count(const unsigned long long *msk, int span) {
    int c = 0;
    for (int t = lane_id(); t < span; t += WARP) c += popc64(msk[t]);
    return warp_sum(c);
}

// Given the row's masks: write its sorted columns to out_col, accumulate the
// products (oracle order) in acc and write the values to out_val.  nnz must
// equal the masks' popcount and be <= cap.  Returns false on inconsistency.
// CLIP: the masks cover one column window [t0*64, (t0+span)*64) of the row;
// each B row is cut to it, and the output is that window's part of the row.
template <int AR, bool NC = true, bool CLIP = false>
__device__ __forceinline__ bool warp_row_fill(int a_lo, int a_hi, const int *__restrict__ acol,
                                              const double *__restrict__ aval, const int *__restrict__ brp,
                                              const int *__restrict__ bre, const int *__restrict__ bcol,
                                              const double *__restrict__ bval, int t0, int span, const unsigned long long *msk, int *base,
                                              double *acc, int nnz, int *__restrict__ out_col,
                                              double *__restrict__ out_val) {
    const int lane = lane_id();
    const int per = (span + WARP - 1) / WARP;
    const int lo = min(span, lane * per), hi = min(span, lo + per);
    int sum = 0;
    for (int t = lo; t < hi; t++) sum += popc64(msk[t]);
    const int incl = warp_incl_scan(sum);
    if (__shfl_sync(FULL, incl, WARP - 1) != nnz) return false;
    int run = incl - sum;
    for (int t = lo; t < hi; t++) {
        unsigned long long m = msk[t];
        base[t] = run;
        int pos = run;
        const int cb = (t0 + t) << 6;
        run += popc64(m);
        while (m) {
            out_col[pos++] = cb + (__ffsll((long long)m) - 1);
            m &= m - 1ull;
        }
    }
    for (int q = lane; q < nnz; q += WARP) acc[q] = 0.0;
    __syncwarp();
    const int c0 = CLIP ? t0 << 6 : 0;
    const int c1 = CLIP ? (int)min((long long)(t0 + span) << 6, (long long)INT_MAX) : 0;
    auto seg = [&](int, int k, int &elo, int &ehi) {
        elo = ldx<NC>(brp + k);
        ehi = ldx<NC>(bre + k);
        if (CLIP) {
            elo = lower_bound_x<NC>(bcol, elo, ehi, c0);
            ehi = lower_bound_x<NC>(bcol, elo, ehi, c1);
        }
    };
    auto lookup = [&](int j) -> int {
        const int t = (j >> 6) - t0;
        if ((unsigned)t >= (unsigned)span) return -1;
        return tile_slot(msk[t], base[t], j);
    };
    bool bad = false;
    warp_accumulate<AR, NC>(a_lo, a_hi, acol, aval, brp, bcol, bval, seg, lookup, acc, bad);
    __syncwarp();
    for (int q = lane; q < nnz; q += WARP) out_val[q] = acc[q];
    __syncwarp();
    return !__any_sync(FULL, bad);
}

}  // namespace hsmu
