// Batched persistent engine: many independent SpGEMMs (C_p = A_p * B_p) or
// AMG Galerkin triple products (C_p = Pt_p * (A_p * P_p)) in one graph launch
// of one kernel, or of two.
//
// The reference runs each product separately, with ~10 blocking host round
// trips and several cudaMalloc calls per product
// (src/compressed/compressed_NHC_spgemm.cu:22-248); for hundreds of small
// products that overhead, not the arithmetic, sets the time.  Here all rows of
// all products form one flattened row space, cut into tiles of 32 rows that
// never span two products, and a cooperative, persistent kernel takes every
// row in one pass:
//   * a warp computes its tile's rows (thread per row with a sorted list in
//     shared memory; warp per row with a dense tile table for rows with more
//     products), so the tile's entry count is known;
//   * one atomic on the product's allocation counter gives the tile a
//     contiguous block of the product's region of the output pool (regions
//     sized by the products' nnz bounds when the batch is made), and the rows
//     are written there, compact, with no count pass and no wait on any other
//     tile.
// Products whose right rows hold one entry (a piecewise-constant prolongator)
// have their first round's tiles done by a launch of its own ahead of that
// kernel, which such batches alone pay for (k_batch_select).
//
// The intermediate A*P of a Galerkin product is read in that form (every row
// has a start and an end); the second product (Pt * (AP)) runs the same way
// after one grid barrier.  The last product is put in row order at the end:
// a device-wide scan of the tile counts gives every tile its place in its
// product, and each tile is copied there as one block with its row pointers.
// No host synchronisation happens inside; the launch is captured once in a
// CUDA graph and replayed.
//
// Wide rows (more than B_FUSE_CAP entries, or a column span of more than
// SPAN_T tiles) are counted by their tile's warp one column window at a time
// and listed; after the tiles, a wide-row phase of the same launch gives each
// listed row to a warp, which writes it window by window (windows of whole
// tiles with fewer than B_FUSE_CAP entries).
//
// Grid barriers spin on a generation counter with an iteration limit: a
// barrier that gives up sets an error bit (HSMU_ERR_TIMEOUT) and every block
// returns, so a fault in one block can never hang the GPU.
//
// Tuning: the thread-per-row product limit (`tiny`) and the grid size are
// parameters of the launch; hsmu_batch_autotune times the candidates on the
// actual batch and keeps the fastest.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstring>
#include <new>
#include <vector>

#include "hsmu_gb.h"
#include "hsmu_kernels.h"
#include "hsmu_rowops.cuh"
#include "hsmu_steps.cuh"

namespace hsmu {

constexpr int B_FUSE_CAP = 512;           // entries of a row (or a column window) written from one table
constexpr int SUB_NNZ = B_FUSE_CAP - 64;  // window cut: tiles whose first entry lies in one block of SUB_NNZ
constexpr int TILE_ROWS = WARP;           // rows per tile (one warp)
constexpr int WIDE_LIST = 1 << 16;        // listed wide rows per round (more are written in place)
constexpr unsigned long long SPIN_LIMIT = 1ull << 25;
enum BatchErr : int { BERR_TIMEOUT = 16, BERR_CAPACITY = 64, BERR_INTERNAL = 128 };

struct BOp {  // one CSR operand on the device; row k is rp[k] .. re[k]-1
    int M, N;
    const int *rp;
    const int *re;
    const int *col;
    const double *val;
};

// A round: one product of every entry of the batch (one round for plain products;
// two for Galerkin entries, A*P and then Pt*(AP)).
struct BRound {
    int nprod;
    const BOp *A;            // left operand per product
    const BOp *B;            // right operand per product (unused when b_from_prev)
    int b_from_prev;         // B_p = C_p of the previous round
    int last;                // the round whose output is returned (put in row order)
    const long long *row0;   // [nprod+1] flattened row offsets
    const long long *rpo;    // [nprod+1] offsets of each product's row pointers in rp_pool / rs / re
    const long long *tile0;  // [nprod+1] offsets of each product's tiles
    const long long *reg;    // [nprod+1] each product's region of the pools
    long long R, T;          // rows, tiles
    unsigned long long *alloc;  // [nprod] entries handed out in each region (zeroed before every launch)
    int *nwide;              // wide rows listed (zeroed before every launch)
    long long *wide;         // [2*WIDE_LIST] (flattened row, pool offset) of listed wide rows
    int *col_pool;           // [reg[nprod]] rows as the tiles wrote them
    double *val_pool;
    // intermediate rounds: every row's start and end in its region
    int *rs, *re;            // [rpo[nprod]]
    // the last round: tile counts and places, then the output in row order
    int *tbase, *tcnt;       // [T] a tile's block in its region, its entry count
    long long *tex;          // [T+1] exclusive scan of tcnt over all tiles of the round
    int *rp_pool;            // [rpo[nprod]] row pointers, 0-based within the product (row counts before)
    int *out_col;            // [reg[nprod]]
    double *out_val;
};

struct GridBar {
    unsigned count;
    unsigned gen;
};

struct BParams {
    BRound rnd[2];
    int nrounds;
    int tiny;              // products limit of the thread-per-row path
    long long *bsum;       // [gridDim.x + 1] block sums of the tile-count scan
    GridBar *bar;
    int *err;
    int arith;             // hsmu_opts.arith of the batch
    const unsigned char *sel_done;  // first round: tiles that k_batch_select has finished (nullable)
    const int *sel_left;            // the number it has not
    unsigned long long spin_limit;  // polls of a grid barrier before it gives up
};

// grid-wide barrier; false (every block returns) when a wait gave up or any
// error bit is set, so no later phase reads what an unfinished phase left
__device__ bool grid_sync(GridBar *gb, int *err, unsigned long long spin_limit) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        int ok = 1;
        volatile unsigned *vgen = &gb->gen;
        const unsigned g = *vgen;
        __threadfence();
        const unsigned arrived = atomicAdd(&gb->count, 1u);
        if (arrived == gridDim.x - 1) {
            atomicExch(&gb->count, 0u);
            __threadfence();
            atomicAdd(&gb->gen, 1u);
        } else {
            unsigned long long it = 0;
            while (*vgen == g) {
                if (++it > spin_limit) {
                    atomicOr(err, BERR_TIMEOUT);
                    ok = 0;
                    break;
                }
                __nanosleep(64);
            }
        }
        __threadfence();
        if (*(volatile int *)err) ok = 0;
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// product owning flattened index i of an ascending offset array (off[lo] <= i < off[lo+1])
__device__ __forceinline__ int find_prod(const long long *off, int n, long long i) {
    int lo = 0, hi = n;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(off + mid) <= i) lo = mid; else hi = mid;
    }
    return lo;
}

// the B operand of product p in round r (C of the previous round for Galerkin)
__device__ __forceinline__ BOp b_operand(const BParams &P, int r, int p) {
    const BRound &R = P.rnd[r];
    if (!R.b_from_prev) return R.B[p];
    const BRound &Q = P.rnd[r - 1];
    const long long base = __ldg(Q.reg + p), ro = __ldg(Q.rpo + p);
    BOp b;
    b.M = (int)(__ldg(Q.row0 + p + 1) - __ldg(Q.row0 + p));
    b.N = __ldg(&Q.B[p].N);
    b.rp = Q.rs + ro;
    b.re = Q.re + ro;
    b.col = Q.col_pool + base;
    b.val = Q.val_pool + base;
    return b;
}

constexpr int BW = 8;  // warps per block (launch uses BW*32 threads)

struct BWarpSmem {
    union {
        struct {
            unsigned long long msk[SPAN_T];
            int base[SPAN_T];
            double acc[B_FUSE_CAP];
        } w;
        struct {
            int cols[TINY_MAX * WARP];
            double acc[TINY_MAX * WARP];
        } t;
    };
};

// exclusive prefix of the masks' popcounts into base[0..span); returns the total
__device__ __forceinline__ int mask_prefix(const unsigned long long *msk, int span, int *base) {
    const int lane = lane_id();
    const int per = (span + WARP - 1) / WARP;
    const int lo = min(span, lane * per), hi = min(span, lo + per);
    int sum = 0;
    for (int t = lo; t < hi; t++) sum += popc64(msk[t]);
    const int incl = warp_incl_scan(sum);
    int run = incl - sum;
    for (int t = lo; t < hi; t++) {
        base[t] = run;
        run += popc64(msk[t]);
    }
    __syncwarp();
    return __shfl_sync(FULL, incl, WARP - 1);
}

// first index in [lo, hi) with base[idx] >= key (base ascending, shared memory)
__device__ __forceinline__ int smem_lower_bound(const int *base, int lo, int hi, int key) {
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (base[mid] < key) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// Entry count of a row that fails the thread path (warp-wide).  Rows of span
// <= SPAN_T tiles take one pass over their products; wider ones one pass per
// SPAN_T-tile column window.  `wide` is set for rows that the warp-row fill
// cannot write in one table (more than B_FUSE_CAP entries or a wide span).
template <bool NC>
__device__ int big_row_count(int a_lo, int a_hi, const BOp &A, const BOp &B, BWarpSmem &S, bool &wide, bool &bad) {
    int cmin, cmax, prod;
    warp_row_extent<NC>(a_lo, a_hi, A.col, B.rp, B.re, B.col, cmin, cmax, prod);
    wide = false;
    if (cmax < 0) return 0;
    const int t_lo = cmin >> 6, t_hi = cmax >> 6;
    if (t_hi - t_lo < SPAN_T) {
        const int span = t_hi - t_lo + 1;
        if (!warp_row_masks<NC>(a_lo, a_hi, A.col, B.rp, B.re, B.col, t_lo, span, S.w.msk)) bad = true;
        const int c = warp_mask_count(S.w.msk, span);
        __syncwarp();
        wide = c > B_FUSE_CAP;
        return c;
    }
    wide = true;
    long long c = 0;
    for (int c0 = t_lo; c0 <= t_hi; c0 += SPAN_T) {
        const int span = min(SPAN_T, t_hi - c0 + 1);
        if (!warp_row_masks<NC, true>(a_lo, a_hi, A.col, B.rp, B.re, B.col, c0, span, S.w.msk)) bad = true;
        c += warp_mask_count(S.w.msk, span);
        __syncwarp();
    }
    if (c > INT_MAX) bad = true;
    return (int)c;
}

// Writes a wide row of `nnz` entries at out_col/out_val (warp-wide): one
// SPAN_T-tile column window at a time, each cut into windows of whole tiles
// whose first entries lie in one block of SUB_NNZ entries (fewer than
// B_FUSE_CAP entries each), written by the warp-row fill on clipped B rows.
template <int AR, bool NC>
__device__ bool wide_row_fill(int a_lo, int a_hi, const BOp &A, const BOp &B, BWarpSmem &S, int nnz,
                              int *__restrict__ out_col, double *__restrict__ out_val) {
    int cmin, cmax, prod;
    warp_row_extent<NC>(a_lo, a_hi, A.col, B.rp, B.re, B.col, cmin, cmax, prod);
    if (cmax < 0) return nnz == 0;
    const int t_lo = cmin >> 6, t_hi = cmax >> 6;
    long long done = 0;
    for (int c0 = t_lo; c0 <= t_hi; c0 += SPAN_T) {
        const int span = min(SPAN_T, t_hi - c0 + 1);
        if (!warp_row_masks<NC, true>(a_lo, a_hi, A.col, B.rp, B.re, B.col, c0, span, S.w.msk)) return false;
        const int total = mask_prefix(S.w.msk, span, S.w.base);
        if (done + total > nnz) return false;
        int s0 = 0;
        for (int w0 = 0; w0 < total; w0 += SUB_NNZ) {
            // tiles [s0, s1): base in [w0, w0 + SUB_NNZ); base[s0..) is read before the
            // fill below rewrites base[s0..s1) with the window's own offsets
            const int s1 = smem_lower_bound(S.w.base, s0, span, w0 + SUB_NNZ);
            const int first = s0 < span ? S.w.base[s0] : total;
            const int n = (s1 < span ? S.w.base[s1] : total) - first;
            __syncwarp();
            if (n > 0 && !warp_row_fill<AR, NC, true>(a_lo, a_hi, A.col, A.val, B.rp, B.re, B.col, B.val, c0 + s0,
                                                      s1 - s0, S.w.msk + s0, S.w.base + s0, S.w.acc, n,
                                                      out_col + done + first, out_val + done + first))
                return false;
            s0 = s1;
        }
        done += total;
    }
    return done == nnz;
}

// A tile's block of its product's region: agg entries from the offset that take_block gives lane 0 (one
// atomic, whose answer is waited for where place_tile uses it), and the row's place in it: cnt entries
// after `before` of the tile's.  ro: the product's rows in the pools; li: the lane's row in the product.
// The whole warp calls both; place_tile gives false (an error is set) when the region is full.
__device__ __forceinline__ unsigned long long take_block(const BRound &R, int p, int agg) {
    return lane_id() == 0 && agg ? atomicAdd(R.alloc + p, (unsigned long long)agg) : 0;
}
__device__ __forceinline__ bool place_tile(const BRound &R, int *err, unsigned long long tb, long long ro, long long region,
                                           long long t, int li, bool valid, int cnt, int before, int agg, int &off) {
    const int lane = lane_id();
    tb = __shfl_sync(FULL, tb, 0);
    if ((long long)tb + agg > region) {
        if (lane == 0) atomicOr(err, BERR_CAPACITY);
        return false;
    }
    off = (int)tb + before;  // within the region
    if (R.last) {
        if (valid) R.rp_pool[ro + li] = cnt;
        if (lane == 0) {
            R.tbase[t] = (int)tb;
            R.tcnt[t] = agg;
        }
    } else if (valid) {
        R.rs[ro + li] = off;
        R.re[ro + li] = off + cnt;
    }
    return true;
}

// Selecting tiles: rows of at most SEL_MAX entries of A whose B rows hold at most one entry each (a
// piecewise-constant prolongator): every entry of A is at most one product, so a row's products are
// sorted by column in a thread's registers -- a network over column << 3 | entry, stable by the entry
// number -- and summed run by run, one multiply and one add per product.  The tile's block is taken as
// soon as the distinct columns are counted, and the rows leave through shared memory, 32 consecutive
// entries per store.  The tile's entries of A, one stretch of the CSR arrays, are copied to shared memory
// while the tile before is computed (in registers they spill).
// They have a launch of their own ahead of the persistent one, at 24 warps per SM where its registers
// allow 16.  That alone gave nothing: the L1 pipe was 61 % busy, with each lane copying its own row and
// the operands' descriptions read for every tile.  With one stretch per tile, the descriptions held until
// the product changes and staging that skips a slot in 16 (strides of 2^k entries meet in few banks
// otherwise) it took 355 us instead of 457 (20 Galerkin products of sides 16..96, 1.13 GB of DRAM
// traffic), a contiguous range of tiles per warp 397 (neighbouring tiles share lines of B).  The whole
// batch: 1.045 ms with these tiles on the lists, 0.743 within the persistent launch, 0.673 so, 0.662 with
// the block asked for before the sums; 0.78 at 16 warps per SM, 0.70 at 20.
constexpr int SEL_MAX = 8;
constexpr int SEL_COLS = 1 << 28;  // B columns a key can hold
constexpr int SEL_TILE = SEL_MAX * WARP;

__device__ __forceinline__ int skew8(int i) { return i + (i >> 4); }  // of 8-byte entries
__device__ __forceinline__ int skew4(int i) { return i + (i >> 5); }  // of 4-byte entries

template <int AR>
struct SelSmem {
    double t[SEL_MAX][WARP];   // add_term's term of every product
    double a[AR == AR_FMA ? SEL_MAX : 1][WARP];  // and its A value
    double val[SEL_TILE + SEL_TILE / 16];  // the tile's entries
    double na[SEL_TILE + SEL_TILE / 16];   // entries of A, copied here while the tile before is computed
    int col[SEL_TILE + SEL_TILE / 32];
    int nk[SEL_TILE + SEL_TILE / 32];
};
// start the copy of a tile's entries of A, [first, end) (at most SEL_TILE)
template <int AR>
__device__ __forceinline__ void sel_copy(int first, int end, const BOp &A, SelSmem<AR> &S) {
#pragma unroll
    for (int u = 0; u < SEL_MAX; u++) {
        const int i = u * WARP + lane_id();
        if (i < end - first) {
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(&S.nk[skew4(i)])), "l"(A.col + first + i)
                         : "memory");
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(&S.na[skew8(i)])), "l"(A.val + first + i)
                         : "memory");
        }
    }
}

constexpr int SELK_WARPS = 4, SELK_CTAS_PER_SM = 6;
static_assert(SELK_CTAS_PER_SM * (SELK_WARPS * sizeof(SelSmem<AR_RN>) + 1024) <= 228 * 1024, "CTAs per SM");

// The selecting tiles of the first round (sel_prod: products that can have them), tile t by global warp
// t mod (warps in the grid).  done[t]: whether the tile is finished; *nleft: tiles that are not (the
// persistent launch does those).
template <int AR>
__global__ void __launch_bounds__(SELK_WARPS * 32, AR == AR_FMA ? 4 : SELK_CTAS_PER_SM)
    k_batch_select(BRound R, const unsigned char *__restrict__ sel_prod, unsigned char *__restrict__ done, int *nleft,
                   int *err) {
    extern __shared__ unsigned long long s_dyn[];
    SelSmem<AR> &S = reinterpret_cast<SelSmem<AR> *>(s_dyn)[threadIdx.x >> 5];
    const int lane = lane_id();
    const long long nw = (long long)gridDim.x * SELK_WARPS;
    // the product of the tile in hand: held until a tile of another one
    int p = 0;
    long long p_t0 = 0, p_t1 = 0, reg0 = 0, rpo = 0;  // its tiles, its place in the pools
    int region = 0;
    bool psel = false;
    BOp A{}, B{};
    auto product_of = [&](long long t) {
        if (t < p_t1) return;
        while (__ldg(R.tile0 + p + 1) <= t) p++;
        p_t0 = __ldg(R.tile0 + p);
        p_t1 = __ldg(R.tile0 + p + 1);
        reg0 = __ldg(R.reg + p);
        region = (int)min((long long)INT_MAX, __ldg(R.reg + p + 1) - reg0);
        rpo = __ldg(R.rpo + p);
        psel = sel_prod[p];
        A = R.A[p];
        B = R.B[p];
    };
    long long t = (long long)blockIdx.x * SELK_WARPS + (threadIdx.x >> 5);
    int left = 0, lo = 0, hi = 0;
    bool ahead = false;  // lo, hi and the copy belong to tile t
    if (t < R.T) p = find_prod(R.tile0, R.nprod, t);
    for (; t < R.T; t += nw) {
        product_of(t);
        if (!psel) {
            if (lane == 0) done[t] = 0;
            left++;
            continue;
        }
        const int li = (int)(t - p_t0) * TILE_ROWS + lane;
        if (!ahead) {
            lo = __ldg(A.rp + min(li, A.M));
            hi = __ldg(A.rp + min(li + 1, A.M));
        }
        const int first = __shfl_sync(FULL, lo, 0), len = hi - lo;
        const bool rows_ok = __all_sync(FULL, len <= SEL_MAX);
        if (!ahead && rows_ok) sel_copy(first, __shfl_sync(FULL, hi, WARP - 1), A, S);
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
        ahead = false;
        unsigned key[SEL_MAX];
        double b[SEL_MAX];
        int s[SEL_MAX], e[SEL_MAX];
        bool one = rows_ok;
        if (rows_ok) {
#pragma unroll
            for (int u = 0; u < SEL_MAX; u++) {
                s[u] = e[u] = 0;
                if (u < len) {
                    const int k = S.nk[skew4(lo - first + u)];
                    s[u] = __ldg(B.rp + k);
                    e[u] = __ldg(B.re + k);
                }
            }
#pragma unroll
            for (int u = 0; u < SEL_MAX; u++) one = one && e[u] - s[u] <= 1;
            one = __all_sync(FULL, one);
        }
        if (!one) {
            if (lane == 0) done[t] = 0;
            left++;
            continue;
        }
#pragma unroll
        for (int u = 0; u < SEL_MAX; u++) {
            key[u] = ~0u;
            b[u] = 0.0;
            if (e[u] > s[u]) {
                key[u] = ((unsigned)__ldg(B.col + s[u]) << 3) | (unsigned)u;
                b[u] = __ldg(B.val + s[u]);
            }
        }
        // the next tile's rows, if it is one of this product's
        int nlo = 0, nhi = 0;
        if (t + nw < p_t1) {
            nlo = __ldg(A.rp + min(li + (int)nw * TILE_ROWS, A.M));
            nhi = __ldg(A.rp + min(li + (int)nw * TILE_ROWS + 1, A.M));
        }
#pragma unroll
        for (int u = 0; u < SEL_MAX; u++) {
            const double a = u < len ? S.na[skew8(lo - first + u)] : 0.0;
            S.t[u][lane] = term<AR>(a, b[u]);
            if (AR == AR_FMA) S.a[u][lane] = a;
        }
        __syncwarp();
        if (t + nw < p_t1 && __all_sync(FULL, nhi - nlo <= SEL_MAX)) {
            sel_copy(__shfl_sync(FULL, nlo, 0), __shfl_sync(FULL, nhi, WARP - 1), A, S);
            ahead = true;
        }
        sort_keys<SEL_MAX>(key);
        int n = 0;
#pragma unroll
        for (int u = 0; u < SEL_MAX; u++) n += key[u] != ~0u && (u == 0 || key[u] >> 3 != key[u - 1] >> 3);
        const int incl = warp_incl_scan(n), before = incl - n;
        const int agg = __shfl_sync(FULL, incl, WARP - 1);
        const unsigned long long tb = take_block(R, p, agg);
        int at = before - 1;
        double acc = 0.0;
#pragma unroll
        for (int u = 0; u < SEL_MAX; u++) {
            if (key[u] != ~0u) {
                const bool head = u == 0 || key[u] >> 3 != key[u - 1] >> 3;
                const int o = (int)(key[u] & 7u);
                at += head;
                acc = add_term<AR>(head ? 0.0 : acc, AR == AR_FMA ? S.a[o][lane] : 0.0, S.t[o][lane]);
                if (u == SEL_MAX - 1 || key[u + 1] >> 3 != key[u] >> 3) {  // the run's last product
                    S.col[skew4(at)] = (int)(key[u] >> 3);
                    S.val[skew8(at)] = acc;
                }
            }
        }
        __syncwarp();
        int off = 0;
        if (place_tile(R, err, tb, rpo, region, t, li, li < A.M, n, before, agg, off)) {
            int *oc = R.col_pool + reg0 + (off - before);
            double *ov = R.val_pool + reg0 + (off - before);
            for (int q = lane; q < agg; q += WARP) {
                oc[q] = S.col[skew4(q)];
                ov[q] = S.val[skew8(q)];
            }
        }
        if (lane == 0) done[t] = 1;
        lo = nlo;
        hi = nhi;
        __syncwarp();
    }
    if (lane == 0 && left) atomicAdd(nleft, left);
}

// Short tiles: rows of at most SHORT_A entries of A whose B rows hold at most SHORT_B entries each (the
// second product of an aggregation: eight fine rows of four coarse columns).  All of a tile's products
// are loaded at once, 32 per thread, sorted by column in registers as above and summed run by run.  In
// the insertion lists every entry of a B row after the first was a memory round trip of its own
// (36 us per tile); 20 Galerkin products of sides 16..96: launch 0.864 -> 0.807 ms.
constexpr int SHORT_A = 8, SHORT_B = 4, SHORT_P = SHORT_A * SHORT_B;
constexpr int SHORT_COLS = (1 << 27) - 1;  // column << 5 | product stays below the empty key

struct ShortSmem {
    double t[SHORT_P][WARP];  // add_term's term of every product
    double a[SHORT_A][WARP];  // its A value (fused multiply-add)
};
static_assert(sizeof(ShortSmem) <= sizeof(BWarpSmem), "short tiles use the warp's shared memory");

// One tile, a row per lane; as in k_batch_select, but each lane writes its own row (take gives the pointers of
// the tile's block).
template <int AR, bool NC, class Take>
__device__ __forceinline__ int short_tile(int a_lo, int a_hi, const BOp &A, const BOp &B, ShortSmem &S, Take take) {
    const int lane = lane_id(), len = a_hi - a_lo;
    if (!__all_sync(FULL, len <= SHORT_A)) return -1;
    int s[SHORT_A], e[SHORT_A];
    double a[SHORT_A];
#pragma unroll
    for (int u = 0; u < SHORT_A; u++) {
        s[u] = u < len ? ldx<NC>(A.col + a_lo + u) : -1;
        a[u] = u < len ? ldx<NC>(A.val + a_lo + u) : 0.0;
    }
    bool fits = true;
#pragma unroll
    for (int u = 0; u < SHORT_A; u++) {
        const int k = s[u];
        s[u] = e[u] = 0;
        if (k >= 0) {
            s[u] = ldx<NC>(B.rp + k);
            e[u] = ldx<NC>(B.re + k);
        }
    }
#pragma unroll
    for (int u = 0; u < SHORT_A; u++) fits = fits && e[u] - s[u] <= SHORT_B;
    if (!__all_sync(FULL, fits)) return -1;
    __syncwarp();
    unsigned key[SHORT_P];
#pragma unroll
    for (int q = 0; q < SHORT_P; q++) {
        const int u = q / SHORT_B, i = q % SHORT_B;
        key[q] = ~0u;
        if (s[u] + i < e[u]) key[q] = ((unsigned)ldx<NC>(B.col + s[u] + i) << 5) | (unsigned)q;
    }
#pragma unroll
    for (int u = 0; u < SHORT_A; u++) {
        double b[SHORT_B];
#pragma unroll
        for (int i = 0; i < SHORT_B; i++) b[i] = s[u] + i < e[u] ? ldx<NC>(B.val + s[u] + i) : 0.0;
#pragma unroll
        for (int i = 0; i < SHORT_B; i++) S.t[u * SHORT_B + i][lane] = term<AR>(a[u], b[i]);
        if (AR == AR_FMA) S.a[u][lane] = a[u];
    }
    sort_keys<SHORT_P>(key);
    int n = 0;
#pragma unroll
    for (int q = 0; q < SHORT_P; q++) n += key[q] != ~0u && (q == 0 || key[q] >> 5 != key[q - 1] >> 5);
    const int incl = warp_incl_scan(n);
    const int agg = __shfl_sync(FULL, incl, WARP - 1);
    int *ocol;
    double *oval;
    take(incl - n, n, agg, ocol, oval);
    int at = incl - n - 1;
    double acc = 0.0;
#pragma unroll
    for (int q = 0; q < SHORT_P; q++) {
        if (key[q] != ~0u) {
            const bool head = q == 0 || key[q] >> 5 != key[q - 1] >> 5;
            const int o = (int)(key[q] & 31u);
            at += head;
            acc = add_term<AR>(head ? 0.0 : acc, AR == AR_FMA ? S.a[o / SHORT_B][lane] : 0.0, S.t[o][lane]);
            if ((q == SHORT_P - 1 || key[q + 1] >> 5 != key[q] >> 5) && ocol) {
                ocol[at] = (int)(key[q] >> 5);
                oval[at] = acc;
            }
        }
    }
    __syncwarp();
    return n;
}

enum RowKind { RK_THREAD = 0, RK_WARP = 1, RK_WIDE = 2 };

// All tiles of round r, tile t by global warp t mod (warps in the grid).  A
// tile's rows are computed, the tile takes a block of its product's region
// (one atomic) and the rows are written there in row order.
template <int AR, bool NC>
__device__ void phase_tiles(const BParams &P, int r, BWarpSmem &S) {
    const BRound &R = P.rnd[r];
    const int lane = lane_id();
    const long long nw = (long long)gridDim.x * BW;
    const long long gw = (long long)blockIdx.x * BW + (threadIdx.x >> 5);
    int p = gw < R.T ? find_prod(R.tile0, R.nprod, gw) : 0;
    int no_short = -1;  // the product whose tiles turned out not to be short ones
    // tiles finished by k_batch_select
    const unsigned char *done = r == 0 ? P.sel_done : nullptr;
    if (done && *(volatile int *)P.sel_left == 0) return;
    for (long long t = gw; t < R.T; t += nw) {
        if (done && done[t]) continue;
        while (__ldg(R.tile0 + p + 1) <= t) p++;
        const long long tfirst = __ldg(R.tile0 + p), prow0 = __ldg(R.row0 + p);
        const int M = (int)(__ldg(R.row0 + p + 1) - prow0);
        const int li = (int)(t - tfirst) * TILE_ROWS + lane;
        const bool valid = li < M;
        const BOp A = R.A[p];
        const BOp B = b_operand(P, r, p);
        const int a_lo = valid ? ldx<true>(A.rp + li) : 0, a_hi = valid ? ldx<true>(A.rp + li + 1) : 0;
        const long long base = __ldg(R.reg + p), region = __ldg(R.reg + p + 1) - base, ro = __ldg(R.rpo + p);
        auto take = [&](int before, int cnt, int agg, int *&oc, double *&ov) {
            int off = 0;
            const bool fits = place_tile(R, P.err, take_block(R, p, agg), ro, region, t, li, valid, cnt, before, agg, off);
            oc = fits ? R.col_pool + base + (off - before) : nullptr;
            ov = R.val_pool + base + (off - before);
        };
        // (rows of one entry of A are in order as they are: the lists append them)
        if (P.tiny >= SHORT_P && p != no_short && B.N <= SHORT_COLS && !__all_sync(FULL, a_hi - a_lo <= 1)) {
            if (short_tile<AR, NC>(a_lo, a_hi, A, B, reinterpret_cast<ShortSmem &>(S), take) >= 0) continue;
            no_short = p;
        }
        // thread path: the row's list is built in shared memory; rows with more
        // than `tiny` products give up (nothing written) and go to the warp
        int cnt = tiny_row_build<AR, NC>(a_lo, a_hi, A.col, A.val, B.rp, B.re, B.col, B.val, S.t.cols + lane,
                                         S.t.acc + lane, WARP, P.tiny);
        int kind = RK_THREAD;
        if (cnt < 0) kind = RK_WARP;
        unsigned bigs = __ballot_sync(FULL, kind != RK_THREAD);
        const bool had_big = bigs != 0;
        bool bad = false;
        while (bigs) {  // counts of the other rows, one row at a time (the lists are lost)
            const int src = __ffs(bigs) - 1;
            bigs &= bigs - 1;
            const int lo = __shfl_sync(FULL, a_lo, src), hi = __shfl_sync(FULL, a_hi, src);
            bool wide;
            const int c = big_row_count<NC>(lo, hi, A, B, S, wide, bad);
            if (lane == src) {
                cnt = c;
                kind = wide ? RK_WIDE : RK_WARP;
            }
        }
        if (!valid) cnt = 0;
        const int incl = warp_incl_scan(cnt);
        const int agg = __shfl_sync(FULL, incl, WARP - 1);
        int off = 0;
        if (!place_tile(R, P.err, take_block(R, p, agg), ro, region, t, li, valid, cnt, incl - cnt, agg, off)) continue;
        int *ocol = R.col_pool + base;
        double *oval = R.val_pool + base;
        if (!had_big) {
            if (valid) tiny_row_write(S.t.cols + lane, S.t.acc + lane, WARP, cnt, ocol + off, oval + off);
            continue;
        }
        // a tile with other rows: thread rows are built again, then the others one at a time
        if (valid && kind == RK_THREAD) {
            if (tiny_row_build<AR, NC>(a_lo, a_hi, A.col, A.val, B.rp, B.re, B.col, B.val, S.t.cols + lane,
                                       S.t.acc + lane, WARP, P.tiny) == cnt)
                tiny_row_write(S.t.cols + lane, S.t.acc + lane, WARP, cnt, ocol + off, oval + off);
            else
                bad = true;
        }
        __syncwarp();
        unsigned warps = __ballot_sync(FULL, valid && kind == RK_WARP);
        while (warps) {
            const int src = __ffs(warps) - 1;
            warps &= warps - 1;
            const int lo = __shfl_sync(FULL, a_lo, src), hi = __shfl_sync(FULL, a_hi, src);
            const int n = __shfl_sync(FULL, cnt, src), o = __shfl_sync(FULL, off, src);
            if (n == 0) continue;
            int cmin, cmax, prod;
            warp_row_extent<NC>(lo, hi, A.col, B.rp, B.re, B.col, cmin, cmax, prod);
            const int t0 = cmin >> 6, span = (cmax >> 6) - t0 + 1;
            if (span > SPAN_T || !warp_row_masks<NC>(lo, hi, A.col, B.rp, B.re, B.col, t0, span, S.w.msk) ||
                !warp_row_fill<AR, NC>(lo, hi, A.col, A.val, B.rp, B.re, B.col, B.val, t0, span, S.w.msk, S.w.base,
                                       S.w.acc, n, ocol + o, oval + o))
                bad = true;
            __syncwarp();
        }
        unsigned wides = __ballot_sync(FULL, valid && kind == RK_WIDE);
        while (wides) {
            const int src = __ffs(wides) - 1;
            wides &= wides - 1;
            const int o = __shfl_sync(FULL, off, src);
            int slot = 0;
            if (lane == 0) slot = atomicAdd(R.nwide, 1);
            slot = __shfl_sync(FULL, slot, 0);
            if (slot < WIDE_LIST) {  // written in the wide-row phase
                if (lane == 0) {
                    R.wide[2 * slot] = prow0 + (t - tfirst) * TILE_ROWS + src;
                    R.wide[2 * slot + 1] = base + o;
                }
                continue;
            }
            const int lo = __shfl_sync(FULL, a_lo, src), hi = __shfl_sync(FULL, a_hi, src);
            const int n = __shfl_sync(FULL, cnt, src);
            if (!wide_row_fill<AR, NC>(lo, hi, A, B, S, n, ocol + o, oval + o)) bad = true;
            __syncwarp();
        }
        if (__any_sync(FULL, bad) && lane == 0) atomicOr(P.err, BERR_INTERNAL);
    }
}

// the listed wide rows of round r, one per warp (after a grid barrier: every
// row's count is stored)
template <int AR, bool NC>
__device__ void phase_wide(const BParams &P, int r, BWarpSmem &S, int n) {
    const BRound &R = P.rnd[r];
    const long long nw = (long long)gridDim.x * BW;
    for (long long e = (long long)blockIdx.x * BW + (threadIdx.x >> 5); e < n; e += nw) {
        const long long i = ldx<false>(R.wide + 2 * e), o = ldx<false>(R.wide + 2 * e + 1);
        const int p = find_prod(R.row0, R.nprod, i);
        const int li = (int)(i - __ldg(R.row0 + p));
        const long long ro = __ldg(R.rpo + p);
        const BOp A = R.A[p];
        const BOp B = b_operand(P, r, p);
        const int nnz = R.last ? ldx<false>(R.rp_pool + ro + li) : ldx<false>(R.re + ro + li) - ldx<false>(R.rs + ro + li);
        if (!wide_row_fill<AR, NC>(ldx<true>(A.rp + li), ldx<true>(A.rp + li + 1), A, B, S, nnz, R.col_pool + o,
                                   R.val_pool + o) &&
            lane_id() == 0)
            atomicOr(P.err, BERR_INTERNAL);
        __syncwarp();
    }
}

// block sums of the last round's tile counts (first step of a device-wide
// exclusive scan of tcnt into tex; the blocks take equal ranges of tiles)
__device__ void scan_block_sums(const BParams &P, const BRound &R) {
    __shared__ long long s_tmp[BW + 1];
    const long long per = (R.T + gridDim.x - 1) / gridDim.x;
    const long long lo = min((long long)blockIdx.x * per, R.T), hi = min(lo + per, R.T);
    long long v = 0;
    for (long long i = lo + threadIdx.x; i < hi; i += blockDim.x) v += ldx<false>(R.tcnt + i);
    long long tot;
    block_excl_sum<BW * 32>(v, s_tmp, tot);
    if (threadIdx.x == 0) P.bsum[blockIdx.x] = tot;
}

// block 0: exclusive scan of the block sums
__device__ void scan_top(const BParams &P, const BRound &R) {
    __shared__ long long s_tmp[BW + 1];
    if (blockIdx.x != 0) return;
    long long carry = 0;
    for (int b0 = 0; b0 < (int)gridDim.x; b0 += blockDim.x) {
        const int b = b0 + threadIdx.x;
        const long long x = b < (int)gridDim.x ? ldx<false>(P.bsum + b) : 0;
        long long t2;
        const long long ex = block_excl_sum<BW * 32>(x, s_tmp, t2);
        if (b < (int)gridDim.x) P.bsum[b] = ex + carry;
        carry += t2;
    }
    if (threadIdx.x == 0) R.tex[R.T] = carry;
}

// the block's range of tiles scanned from its block sum, SCAN_RUN tiles per thread
__device__ void scan_blocks(const BParams &P, const BRound &R) {
    __shared__ long long s_tmp[BW + 1];
    constexpr int SCAN_RUN = 16;
    const long long per = (R.T + gridDim.x - 1) / gridDim.x;
    const long long lo = min((long long)blockIdx.x * per, R.T), hi = min(lo + per, R.T);
    long long run = ldx<false>(P.bsum + blockIdx.x);
    for (long long b = lo; b < hi; b += (long long)blockDim.x * SCAN_RUN) {
        const long long i0 = b + (long long)threadIdx.x * SCAN_RUN;
        int x[SCAN_RUN];
        long long sum = 0;
#pragma unroll
        for (int u = 0; u < SCAN_RUN; u++) {
            x[u] = i0 + u < hi ? ldx<false>(R.tcnt + i0 + u) : 0;
            sum += x[u];
        }
        long long t2;
        long long e = run + block_excl_sum<BW * 32>(sum, s_tmp, t2);
#pragma unroll
        for (int u = 0; u < SCAN_RUN; u++) {
            if (i0 + u < hi) R.tex[i0 + u] = e;
            e += x[u];
        }
        run += t2;
    }
}

// the last round in row order: every tile's block copied to its place in the
// product (scanned tile counts) and its rows' pointers written
// PLACE_U steps of a block are read before any is written: a step at a time each
// waits for its own round trip, seven for a tile of 7-entry rows (20 Galerkin products
// of sides 16..96, whole launch: 0.662 -> 0.603 ms).
constexpr int PLACE_U = 8;

__device__ void phase_place(const BParams &P, const BRound &R) {
    const int lane = lane_id();
    const long long nw = (long long)gridDim.x * BW;
    const long long gw = (long long)blockIdx.x * BW + (threadIdx.x >> 5);
    int p = gw < R.T ? find_prod(R.tile0, R.nprod, gw) : 0;
    for (long long t = gw; t < R.T; t += nw) {
        while (__ldg(R.tile0 + p + 1) <= t) p++;
        const long long tfirst = __ldg(R.tile0 + p);
        const int M = (int)(__ldg(R.row0 + p + 1) - __ldg(R.row0 + p));
        const int li = (int)(t - tfirst) * TILE_ROWS + lane;
        const long long ro = __ldg(R.rpo + p), base = __ldg(R.reg + p);
        const long long dst = ldx<false>(R.tex + t) - ldx<false>(R.tex + tfirst);  // within the product
        const int n = ldx<false>(R.tcnt + t);
        const int src = ldx<false>(R.tbase + t);
        const int c = li < M ? ldx<false>(R.rp_pool + ro + li) : 0;
        const int incl = warp_incl_scan(c);
        if (li < M) {
            R.rp_pool[ro + li] = (int)dst + incl - c;
            if (li == M - 1) R.rp_pool[ro + M] = (int)dst + incl;
        }
        const int *sc = R.col_pool + base + src;
        const double *sv = R.val_pool + base + src;
        int *dc = R.out_col + base + dst;
        double *dv = R.out_val + base + dst;
        for (StepPos q0 = lane; step_in(q0, 0, n); q0 += PLACE_U * WARP) {
            int c8[PLACE_U];
            double v8[PLACE_U];
#pragma unroll
            for (int u = 0; u < PLACE_U; u++) {
                const bool in = step_in(q0, u * WARP, n);
                c8[u] = in ? ldx<false>(sc + q0 + u * WARP) : 0;
                v8[u] = in ? ldx<false>(sv + q0 + u * WARP) : 0.0;
            }
#pragma unroll
            for (int u = 0; u < PLACE_U; u++) {
                if (step_in(q0, u * WARP, n)) {
                    dc[q0 + u * WARP] = c8[u];
                    dv[q0 + u * WARP] = v8[u];
                }
            }
        }
    }
}

template <int AR>
__global__ void __launch_bounds__(BW * 32, 2) k_batch(BParams P) {
    extern __shared__ unsigned long long s_dyn[];
    BWarpSmem &S = reinterpret_cast<BWarpSmem *>(s_dyn)[threadIdx.x >> 5];
    for (int r = 0; r < P.nrounds; r++) {
        // the first product reads only the caller's operands (read-only path); the second
        // reads the first one's output, ordered by the barrier's fences
        if (r == 0) phase_tiles<AR, true>(P, r, S);
        else phase_tiles<AR, false>(P, r, S);
        if (!grid_sync(P.bar, P.err, P.spin_limit)) return;
        const BRound &R = P.rnd[r];
        const int nwide = min(*(volatile int *)R.nwide, WIDE_LIST);
        if (nwide > 0) {
            if (r == 0) phase_wide<AR, true>(P, r, S, nwide);
            else phase_wide<AR, false>(P, r, S, nwide);
        }
        if (!R.last) {
            if (nwide > 0 && !grid_sync(P.bar, P.err, P.spin_limit)) return;
            continue;
        }
        scan_block_sums(P, R);
        if (!grid_sync(P.bar, P.err, P.spin_limit)) return;
        scan_top(P, R);
        if (!grid_sync(P.bar, P.err, P.spin_limit)) return;
        scan_blocks(P, R);
        if (!grid_sync(P.bar, P.err, P.spin_limit)) return;
        phase_place(P, R);
    }
}

// ---------------------------------------------------------------- sizing
// per row of the first product: products and the bound min(products, N) on its nnz,
// summed per product; `rowbound` keeps the uncapped products of each row for
// the second product's bound; `unfit` counts each product's rows that keep their
// tile from being a selecting one (nullable)
__device__ __forceinline__ void add_per_product(unsigned long long *pbound, int p, unsigned long long v) {
    const int p0 = __shfl_sync(FULL, p, 0);
    if (__all_sync(FULL, p == p0)) {
        v = warp_sum(v);
        if (lane_id() == 0 && v) atomicAdd(pbound + p0, v);
    } else if (v) {
        atomicAdd(pbound + p, v);
    }
}

__global__ void k_batch_bound(const BOp *A, const BOp *B, const long long *row0, int nprod, long long R,
                              long long *rowbound, unsigned long long *pbound, unsigned long long *unfit) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    // every lane runs the same number of iterations (the warp-wide sums below)
    for (long long i0 = blockIdx.x * (long long)blockDim.x; i0 < R; i0 += stride) {
        const long long i = i0 + threadIdx.x;
        int p = 0;
        unsigned long long bnd = 0;
        bool fits = true;
        if (i < R) {
            p = find_prod(row0, nprod, i);
            const BOp a = A[p], b = B[p];
            const int li = (int)(i - row0[p]);
            long long prod = 0;
            for (int q = a.rp[li]; q < a.rp[li + 1]; q++) {
                const int k = a.col[q];
                const int len = b.rp[k + 1] - b.rp[k];
                prod += len;
                fits = fits && len <= 1;
            }
            fits = fits && a.rp[li + 1] - a.rp[li] <= SEL_MAX;
            if (rowbound) rowbound[i] = prod;
            bnd = (unsigned long long)(prod < b.N ? prod : b.N);
        }
        add_per_product(pbound, p, bnd);
        if (unfit) add_per_product(unfit, p, !fits);
    }
}

// bound of a row of Pt * (A*P): the sum over its entries of the A*P row bounds, capped by N
__global__ void k_batch_bound2(const BOp *Pt, const long long *row0_2, const long long *row0_1, int nprod,
                               long long R, const long long *rowbound1, const int *ncols,
                               unsigned long long *pbound) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i0 = blockIdx.x * (long long)blockDim.x; i0 < R; i0 += stride) {
        const long long i = i0 + threadIdx.x;
        int p = 0;
        unsigned long long bnd = 0;
        if (i < R) {
            p = find_prod(row0_2, nprod, i);
            const BOp a = Pt[p];
            const int li = (int)(i - row0_2[p]);
            long long prod = 0;
            for (int q = a.rp[li]; q < a.rp[li + 1]; q++)
                prod += min(rowbound1[row0_1[p] + a.col[q]], (long long)ncols[p]);
            bnd = (unsigned long long)(prod < ncols[p] ? prod : ncols[p]);
        }
        add_per_product(pbound, p, bnd);
    }
}

}  // namespace hsmu

using namespace hsmu;

struct hsmu_batch_s {
    int kind, nprod;
    int nsm, grid, threads, tiny, arith;
    size_t smem;
    unsigned char *sel_prod, *sel_done;  // products that can have selecting tiles (null: none has), tiles
    int *sel_left;
    BParams P;
    std::vector<void *> allocs;
    std::vector<long long> row0[2], rpo[2], reg[2];
    std::vector<int> ncol[2];
    void *reset;          // zeroed before every launch: barrier, error word, wide-row counters, tiles left, allocation counters
    size_t reset_bytes;
    cudaGraph_t graph;
    cudaGraphExec_t gexec;
};

namespace {

template <class T>
cudaError_t balloc(hsmu_batch_s *b, T **p, size_t n) {
    *p = nullptr;
    cudaError_t e = cudaMalloc(reinterpret_cast<void **>(p), std::max<size_t>(n, 1) * sizeof(T));
    if (e == cudaSuccess) b->allocs.push_back(*p);
    return e;
}

template <class T>
cudaError_t bupload(hsmu_batch_s *b, T **p, const std::vector<T> &h) {
    cudaError_t e = balloc(b, p, h.size());
    if (e == cudaSuccess) e = cudaMemcpy(*p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice);
    return e;
}

template <int AR>
int launch_select(hsmu_batch_s *b, cudaStream_t st) {
    const int per_sm = AR == AR_FMA ? 4 : SELK_CTAS_PER_SM;
    const BRound &R = b->P.rnd[0];
    k_batch_select<AR><<<grid_for(b->nsm * per_sm, R.T, SELK_WARPS), SELK_WARPS * 32, SELK_WARPS * sizeof(SelSmem<AR>), st>>>(
        R, b->sel_prod, b->sel_done, b->sel_left, b->P.err);
    return cudaGetLastError() == cudaSuccess ? HSMU_OK : HSMU_ERR_CUDA;
}

int launch_batch(hsmu_batch_s *b, cudaStream_t st) {
    if (cudaMemsetAsync(b->reset, 0, b->reset_bytes, st) != cudaSuccess) return HSMU_ERR_CUDA;
    b->P.tiny = b->tiny;
    const bool sel = b->sel_prod && b->tiny >= SEL_MAX;
    b->P.sel_done = sel ? b->sel_done : nullptr;
    b->P.sel_left = b->sel_left;
    if (sel) {
        const int rc = b->arith == AR_IMUL  ? launch_select<AR_IMUL>(b, st)
                       : b->arith == AR_FMA ? launch_select<AR_FMA>(b, st)
                                            : launch_select<AR_RN>(b, st);
        if (rc) return rc;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(b->grid);
    cfg.blockDim = dim3(b->threads);
    cfg.dynamicSmemBytes = b->smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t e = b->arith == AR_IMUL  ? cudaLaunchKernelEx(&cfg, k_batch<AR_IMUL>, b->P)
                    : b->arith == AR_FMA ? cudaLaunchKernelEx(&cfg, k_batch<AR_FMA>, b->P)
                                         : cudaLaunchKernelEx(&cfg, k_batch<AR_RN>, b->P);
    return e == cudaSuccess ? HSMU_OK : HSMU_ERR_CUDA;
}

int configure_batch(hsmu_batch_s *b, int dev) {
    b->threads = BW * 32;
    b->smem = BW * sizeof(BWarpSmem);
    for (auto k : {k_batch<AR_RN>, k_batch<AR_FMA>, k_batch<AR_IMUL>})
        if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)b->smem) != cudaSuccess)
            return HSMU_ERR_CUDA;
    if (cudaFuncSetAttribute(k_batch_select<AR_RN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             SELK_WARPS * (int)sizeof(SelSmem<AR_RN>)) != cudaSuccess ||
        cudaFuncSetAttribute(k_batch_select<AR_FMA>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             SELK_WARPS * (int)sizeof(SelSmem<AR_FMA>)) != cudaSuccess ||
        cudaFuncSetAttribute(k_batch_select<AR_IMUL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             SELK_WARPS * (int)sizeof(SelSmem<AR_IMUL>)) != cudaSuccess)
        return HSMU_ERR_CUDA;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_batch<AR_RN>, b->threads, b->smem) != cudaSuccess ||
        per_sm < 1)
        return HSMU_ERR_CUDA;
    int coop = 0;
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    if (!coop) return HSMU_ERR_NO_DEVICE;
    b->grid = b->nsm * per_sm;
    return HSMU_OK;
}

}  // namespace

extern "C" {

int hsmu_batch_create(hsmu_handle h, int kind, int n, const hsmu_csr *A, const hsmu_csr *B, const hsmu_csr *Pt,
                      const hsmu_opts *opts, hsmu_batch *out, void *stream) {
    if (!h || !out || n <= 0 || !A || !B) return HSMU_ERR_INVALID;
    if (kind != HSMU_BATCH_PRODUCT && kind != HSMU_BATCH_GALERKIN) return HSMU_ERR_INVALID;
    if (kind == HSMU_BATCH_GALERKIN && !Pt) return HSMU_ERR_INVALID;
    if (opts && (opts->arith < HSMU_ARITH_RN || opts->arith > HSMU_ARITH_IMUL)) return HSMU_ERR_INVALID;
    *out = nullptr;
    for (int p = 0; p < n; p++) {
        if (A[p].N != B[p].M || !A[p].row_ptr || !B[p].row_ptr) return HSMU_ERR_INVALID;
        if (kind == HSMU_BATCH_GALERKIN && (Pt[p].N != A[p].M || !Pt[p].row_ptr)) return HSMU_ERR_INVALID;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    hsmu_batch_s *b = new (std::nothrow) hsmu_batch_s();
    if (!b) return HSMU_ERR_ALLOC;
    b->kind = kind;
    b->nprod = n;
    b->arith = opts ? opts->arith : AR_RN;
    // test hook: barriers and look-backs that give up after opts->wait_polls polls
    b->P.spin_limit = (opts && opts->wait_polls > 0) ? (unsigned long long)opts->wait_polls : SPIN_LIMIT;
    b->tiny = TINY_MAX;
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&b->nsm, cudaDevAttrMultiProcessorCount, dev);
    int rc = configure_batch(b, dev);
    const int nr = kind == HSMU_BATCH_GALERKIN ? 2 : 1;
    long long *rowbound = nullptr;
    int *dncol = nullptr;
    unsigned long long *dpb = nullptr;
    std::vector<unsigned long long> hpb;
    std::vector<unsigned char> sel((size_t)n, 0);
    bool any_sel = false;
    std::vector<long long> tiles[2];
    std::vector<BOp> hA(n), hB(n);
    if (rc) goto fail;
    b->P.nrounds = nr;
    // operand tables, row, row-pointer and tile offsets
    for (int r = 0; r < nr; r++) {
        const hsmu_csr *L = (r == 0) ? A : Pt;
        b->row0[r].assign(n + 1, 0);
        b->rpo[r].assign(n + 1, 0);
        tiles[r].assign(n + 1, 0);
        b->ncol[r].assign(n, 0);
        for (int p = 0; p < n; p++) {
            b->row0[r][p + 1] = b->row0[r][p] + L[p].M;
            b->rpo[r][p + 1] = b->rpo[r][p] + L[p].M + 1;
            tiles[r][p + 1] = tiles[r][p] + (L[p].M + TILE_ROWS - 1) / TILE_ROWS;
            b->ncol[r][p] = B[p].N;
        }
        for (int p = 0; p < n; p++) {
            hA[p] = BOp{L[p].M, L[p].N, L[p].row_ptr, L[p].row_ptr + 1, L[p].col, L[p].val};
            hB[p] = BOp{B[p].M, B[p].N, B[p].row_ptr, B[p].row_ptr + 1, B[p].col, B[p].val};
        }
        BRound &R = b->P.rnd[r];
        BOp *dA = nullptr, *dB = nullptr;
        long long *drow0 = nullptr, *drpo = nullptr, *dtile0 = nullptr;
        if (bupload(b, &dA, hA) || bupload(b, &dB, hB) || bupload(b, &drow0, b->row0[r]) ||
            bupload(b, &drpo, b->rpo[r]) || bupload(b, &dtile0, tiles[r])) {
            rc = HSMU_ERR_ALLOC;
            goto fail;
        }
        R.nprod = n;
        R.A = dA;
        R.B = (r == 0) ? dB : nullptr;
        R.b_from_prev = r > 0;
        R.row0 = drow0;
        R.rpo = drpo;
        R.tile0 = dtile0;
        R.R = b->row0[r][n];
        R.T = tiles[r][n];
    }
    // products that can have selecting tiles: single-entry right rows, short left rows, columns that a
    // sort key holds (and few enough rows that do not fit: counted by the sizing pass)
    for (int p = 0; p < n; p++) {
        sel[(size_t)p] = B[p].nnz <= B[p].M && A[p].nnz <= (long long)SEL_MAX * A[p].M && B[p].N <= SEL_COLS;
        any_sel |= sel[(size_t)p] != 0;
    }
    // nnz bound of every product (one sizing pass and one host read): min(products, N) per row of
    // the first product; for Galerkin, per row of the second the sum of its A*P rows' bounds
    if (balloc(b, &dpb, (size_t)n * (nr + 1)) || (nr == 2 && balloc(b, &rowbound, (size_t)b->P.rnd[0].R))) {
        rc = HSMU_ERR_ALLOC;
        goto fail;
    }
    cudaMemsetAsync(dpb, 0, sizeof(unsigned long long) * n * (nr + 1), st);
    k_batch_bound<<<b->nsm * 8, 256, 0, st>>>(b->P.rnd[0].A, b->P.rnd[0].B, b->P.rnd[0].row0, n, b->P.rnd[0].R,
                                              rowbound, dpb, any_sel ? dpb + (size_t)n * nr : nullptr);
    if (nr == 2) {
        if (bupload(b, &dncol, b->ncol[1])) {
            rc = HSMU_ERR_ALLOC;
            goto fail;
        }
        k_batch_bound2<<<b->nsm * 8, 256, 0, st>>>(b->P.rnd[1].A, b->P.rnd[1].row0, b->P.rnd[0].row0, n,
                                                   b->P.rnd[1].R, rowbound, dncol, dpb + n);
    }
    hpb.assign((size_t)n * (nr + 1), 0);
    if (cudaGetLastError() != cudaSuccess ||
        cudaMemcpyAsync(hpb.data(), dpb, sizeof(unsigned long long) * n * (nr + 1), cudaMemcpyDeviceToHost, st) ||
        cudaStreamSynchronize(st)) {
        rc = HSMU_ERR_CUDA;
        goto fail;
    }
    for (void *q : {(void *)rowbound, (void *)dpb, (void *)dncol}) {  // only needed for sizing
        if (!q) continue;
        cudaFree(q);
        b->allocs.erase(std::find(b->allocs.begin(), b->allocs.end(), q));
    }
    // A product whose unfit rows may spoil half of its tiles goes without selecting tiles: where no product
    // has them their launch is saved (sixteen products of 5,000 rows of 4 to 9 entries: 70.7 -> 68 us).
    {
        bool any = false;
        for (int p = 0; p < n; p++) {
            const long long tiles = (b->row0[0][p + 1] - b->row0[0][p] + TILE_ROWS - 1) / TILE_ROWS;
            if (2 * hpb[(size_t)n * nr + p] > (unsigned long long)tiles) sel[(size_t)p] = 0;
            any |= sel[(size_t)p] != 0;
        }
        if (any && (bupload(b, &b->sel_prod, sel) || balloc(b, &b->sel_done, (size_t)b->P.rnd[0].T))) {
            rc = HSMU_ERR_ALLOC;
            goto fail;
        }
    }
    // output regions (a product's entries are indexed by int: its region is capped there; a
    // product that needs more reports HSMU_ERR_OVERFLOW), pools, row starts / row pointers
    for (int r = 0; r < nr; r++) {
        BRound &R = b->P.rnd[r];
        R.last = r == nr - 1;
        b->reg[r].assign(n + 1, 0);
        for (int p = 0; p < n; p++)
            b->reg[r][p + 1] = b->reg[r][p] + (long long)std::min<unsigned long long>(hpb[(size_t)r * n + p], INT_MAX);
        const size_t cap = (size_t)b->reg[r][n], nrp = (size_t)b->rpo[r][n];
        long long *dreg = nullptr;
        if (bupload(b, &dreg, b->reg[r]) || balloc(b, &R.col_pool, cap) || balloc(b, &R.val_pool, cap) ||
            balloc(b, &R.wide, 2 * (size_t)WIDE_LIST)) {
            rc = HSMU_ERR_ALLOC;
            goto fail;
        }
        R.reg = dreg;
        if (!R.last) {
            if (balloc(b, &R.rs, nrp) || balloc(b, &R.re, nrp)) {
                rc = HSMU_ERR_ALLOC;
                goto fail;
            }
            continue;
        }
        if (balloc(b, &R.tbase, (size_t)R.T) || balloc(b, &R.tcnt, (size_t)R.T) || balloc(b, &R.tex, (size_t)R.T + 1) ||
            balloc(b, &R.rp_pool, nrp) || balloc(b, &R.out_col, cap) || balloc(b, &R.out_val, cap)) {
            rc = HSMU_ERR_ALLOC;
            goto fail;
        }
        // row pointers of products without rows are never written by a tile
        if (cudaMemset(R.rp_pool, 0, sizeof(int) * nrp) != cudaSuccess) {
            rc = HSMU_ERR_CUDA;
            goto fail;
        }
    }
    {
        int per_sm = 0;  // the scan's block sums, for the largest grid a launch can have
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_batch<AR_RN>, b->threads, b->smem);
        if (balloc(b, &b->P.bsum, (size_t)b->nsm * per_sm + 1)) {
            rc = HSMU_ERR_ALLOC;
            goto fail;
        }
    }
    // the block zeroed before every launch: barrier, error word, wide-row counters, allocation counters
    {
        size_t o = 0;
        const size_t o_bar = o;
        o += sizeof(GridBar);
        const size_t o_err = o;
        o += sizeof(int);
        const size_t o_nwide = o;
        o += 2 * sizeof(int);
        const size_t o_left = o;
        o += sizeof(int);
        o = (o + 15) & ~size_t(15);
        size_t o_alloc[2] = {0, 0};
        for (int r = 0; r < nr; r++) {
            o_alloc[r] = o;
            o += sizeof(unsigned long long) * (size_t)n;
        }
        unsigned char *rb = nullptr;
        if (balloc(b, &rb, o)) {
            rc = HSMU_ERR_ALLOC;
            goto fail;
        }
        b->reset = rb;
        b->reset_bytes = o;
        b->P.bar = reinterpret_cast<GridBar *>(rb + o_bar);
        b->P.err = reinterpret_cast<int *>(rb + o_err);
        b->sel_left = reinterpret_cast<int *>(rb + o_left);
        for (int r = 0; r < nr; r++) {
            b->P.rnd[r].nwide = reinterpret_cast<int *>(rb + o_nwide) + r;
            b->P.rnd[r].alloc = reinterpret_cast<unsigned long long *>(rb + o_alloc[r]);
        }
    }
    b->P.arith = b->arith;
    *out = b;
    return HSMU_OK;
fail:
    hsmu_batch_destroy(b);
    return rc;
}

int hsmu_batch_execute(hsmu_batch b, void *stream) {
    if (!b) return HSMU_ERR_INVALID;
    return launch_batch(b, static_cast<cudaStream_t>(stream));
}

int hsmu_batch_graph_launch(hsmu_batch b, void *stream) {
    if (!b) return HSMU_ERR_INVALID;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (!b->gexec) {
        cudaStream_t cap;
        if (cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking) != cudaSuccess) return HSMU_ERR_CUDA;
        int rc = HSMU_OK;
        if (cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal) != cudaSuccess) rc = HSMU_ERR_CUDA;
        if (!rc) rc = launch_batch(b, cap);
        cudaGraph_t g = nullptr;
        const cudaError_t ee = cudaStreamEndCapture(cap, &g);
        if (!rc && ee != cudaSuccess) rc = HSMU_ERR_CUDA;
        if (!rc && cudaGraphInstantiate(&b->gexec, g, 0) != cudaSuccess) rc = HSMU_ERR_CUDA;
        if (g) b->graph = g;
        cudaStreamDestroy(cap);
        if (rc) {
            cudaGetLastError();
            return rc;
        }
    }
    return cudaGraphLaunch(b->gexec, st) == cudaSuccess ? HSMU_OK : HSMU_ERR_CUDA;
}

int hsmu_batch_status(hsmu_batch b, void *stream) {
    if (!b) return HSMU_ERR_INVALID;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    int err = 0;
    if (cudaMemcpyAsync(&err, b->P.err, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return HSMU_ERR_CUDA;
    if (err & BERR_TIMEOUT) return HSMU_ERR_TIMEOUT;
    if (err & BERR_CAPACITY) return HSMU_ERR_OVERFLOW;
    if (err) return HSMU_ERR_INTERNAL;
    return HSMU_OK;
}

int hsmu_batch_result(hsmu_batch b, int p, hsmu_csr *C) {
    if (!b || !C || p < 0 || p >= b->nprod) return HSMU_ERR_INVALID;
    const int r = b->P.nrounds - 1;
    const BRound &R = b->P.rnd[r];
    const int M = (int)(b->row0[r][p + 1] - b->row0[r][p]);
    int nnz = 0;
    if (cudaMemcpy(&nnz, R.rp_pool + b->rpo[r][p] + M, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess)
        return HSMU_ERR_CUDA;
    C->M = M;
    C->N = b->ncol[r][p];
    C->nnz = nnz;
    C->owned = 0;
    C->row_ptr = R.rp_pool + b->rpo[r][p];
    C->col = R.out_col + b->reg[r][p];
    C->val = R.out_val + b->reg[r][p];
    return HSMU_OK;
}

int hsmu_batch_set_params(hsmu_batch b, int tiny, int grid) {
    if (!b || tiny < 0 || tiny > TINY_MAX || grid < 0) return HSMU_ERR_INVALID;
    b->tiny = tiny;
    if (grid > 0) {
        int per_sm = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_batch<AR_RN>, b->threads, b->smem);
        if (grid > b->nsm * per_sm) return HSMU_ERR_INVALID;  // cooperative launch needs all blocks resident
        b->grid = grid;
    }
    if (b->gexec) {
        cudaGraphExecDestroy(b->gexec);
        b->gexec = nullptr;
    }
    if (b->graph) {
        cudaGraphDestroy(b->graph);
        b->graph = nullptr;
    }
    return HSMU_OK;
}

int hsmu_batch_autotune(hsmu_batch b, void *stream, int *best_tiny, int *best_grid, float *best_ms) {
    if (!b) return HSMU_ERR_INVALID;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_batch<AR_RN>, b->threads, b->smem);
    const int tinies[] = {8, 16, 32};
    std::vector<int> grids = {b->nsm * per_sm};
    if (per_sm > 1) grids.push_back(b->nsm);
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    float best = 1e30f;
    int bt = b->tiny, bg = b->grid, rc = HSMU_OK;
    for (int t : tinies)
        for (int g : grids) {
            if ((rc = hsmu_batch_set_params(b, t, g))) break;
            if ((rc = launch_batch(b, st))) break;  // warm-up
            cudaEventRecord(e0, st);
            for (int k = 0; k < 2 && !rc; k++) rc = launch_batch(b, st);
            cudaEventRecord(e1, st);
            if (cudaEventSynchronize(e1) != cudaSuccess) rc = HSMU_ERR_CUDA;
            if (rc) break;
            if ((rc = hsmu_batch_status(b, st))) break;
            float ms = 0.f;
            cudaEventElapsedTime(&ms, e0, e1);
            ms *= 0.5f;
            if (ms < best) {
                best = ms;
                bt = t;
                bg = g;
            }
        }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (rc) return rc;
    rc = hsmu_batch_set_params(b, bt, bg);
    if (best_tiny) *best_tiny = bt;
    if (best_grid) *best_grid = bg;
    if (best_ms) *best_ms = best;
    return rc;
}

int hsmu_batch_destroy(hsmu_batch b) {
    if (!b) return HSMU_OK;
    if (b->gexec) cudaGraphExecDestroy(b->gexec);
    if (b->graph) cudaGraphDestroy(b->graph);
    for (void *p : b->allocs) cudaFree(p);
    delete b;
    return HSMU_OK;
}

}  // extern "C"
