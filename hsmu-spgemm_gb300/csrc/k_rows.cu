// Stage 2: per-row bounds + row binning, and the device exclusive scan.
//
// Bounds: for every A row, the number of intermediate products
// sum_{k in A(i,:)} nnz(B(k,:)) (64-bit; the reference counts it on the host,
// src/NHC_spgemm.cuh:37-42, and bounds C tiles per row with k_compute_flop,
// src/small/mask.cuh:14-51) and the exact first/last C tile of the row (the
// min/max over the 64-column tiles of every referenced B row's first and last
// column -- read from B itself, so this pass does not wait for B's tiles and
// runs beside their construction).  The tile span decides the row class
// (one warp with a dense span table, or one CTA with a chunked table), which
// replaces the reference's host-round-trip binning (src/bining.cuh:1-207):
// rows are binned on the device by a stable single-pass compaction, so every bin
// lists its rows in ascending order and the rows of a row panel are one
// contiguous slice of each bin.
//
// Scan: one launch with a look-back over the earlier tiles' sums, 64-bit running
// totals; replaces cub::DeviceScan::ExclusiveSum plus the full-array D2H copies
// of the reference (src/compressed/compressed_tileOR.cuh:620-622).
#include <climits>

#include "hsmu_common.cuh"
#include "hsmu_kernels.h"
#include "hsmu_lookback.cuh"
#include "hsmu_rowops.cuh"
#include "hsmu_rowsums.cuh"

namespace hsmu {

// the most tiles and products of a warp row
struct ClassLine {
    float tiles;
    long long products;
};

// What a block adds up over its rows for the control block: one thread per sum sends it there.
enum BoundsSum { BS_PROD, BS_WB, BS_CB, BS_CBD, BS_WDP, BS_SPAN, BS_BIN, BS_N = BS_BIN + NBIN };
struct BoundsSmem {
    unsigned long long sum[BS_N];
};

// a thread's part of them
struct BoundsSums {
    unsigned long long t_prod = 0, t_wb = 0, t_cb = 0, t_cbd = 0, t_wdp = 0, t_span = 0;
    int cnt[NBIN] = {};

    // one row's products, tile span and class
    __device__ __forceinline__ void row(int i, int len, const RowSums<true> &sums, int N, const RowInfo &ri,
                                        ClassLine line) {
        const long long prod = sums.prod;
        const int tmin = sums.cmin == INT_MAX ? INT_MAX : sums.cmin >> 6, tmax = sums.cmax >> 6;
        ri.prod[i] = prod;
        ri.tmin[i] = tmin;
        ri.tmax[i] = tmax;
        int bin = -1;
        if (prod == 0) {
            ri.cnnz[i] = 0;
        } else {
            const int span = tmax - tmin + 1;
            const bool scattered = prod <= H_MAX && span <= H_SPAN && len <= H_ROW;
            const bool narrow = span <= SPAN_T && sums.tiles <= line.tiles && prod <= line.products;
            bin = prod <= TINY_MAX ? BIN_TINY : narrow ? BIN_DS : scattered ? BIN_H : BIN_L;
            t_prod += (unsigned long long)prod;
            const long long cap = prod < (long long)N ? prod : (long long)N;
            // windows per row <= slot cuts + tile-rank cuts + span cuts + 1
            const long long tl = cap < (long long)span ? cap : (long long)span;
            const unsigned long long wb = (unsigned long long)(cap / WIN_CUT + tl / WIN_TCAP + (span - 1) / WIN_SPAN + 1);
            // rows that can reach the window pass: the large class, and warp rows above FUSE_CAP
            if (bin == BIN_L) {
                t_wb += wb;
                t_cb += wb * (unsigned long long)len;
                t_span += (unsigned long long)span;
            }
            if (bin == BIN_DS && prod > FUSE_CAP) {
                t_wb += wb;
                t_cbd += wb * (unsigned long long)len;
                t_wdp += (unsigned long long)prod;
            }
        }
        ri.cls[i] = (signed char)bin;
#pragma unroll
        for (int k = 0; k < NBIN; k++) cnt[k] += bin == k;
    }

    // every thread of the block
    __device__ __forceinline__ void flush(BoundsSmem &S, Ctl *ctl) {
        if (threadIdx.x < BS_N) S.sum[threadIdx.x] = 0;
        __syncthreads();
        auto add = [&](int k, unsigned long long v) {
            v = warp_sum(v);
            if (lane_id() == 0 && v) atomicAdd(&S.sum[k], v);
        };
        add(BS_PROD, t_prod);
        add(BS_WB, t_wb);
        add(BS_CB, t_cb);
        add(BS_CBD, t_cbd);
        add(BS_WDP, t_wdp);
        add(BS_SPAN, t_span);
#pragma unroll
        for (int k = 0; k < NBIN; k++) add(BS_BIN + k, (unsigned long long)cnt[k]);
        __syncthreads();
        const unsigned long long v = threadIdx.x < BS_N ? S.sum[threadIdx.x] : 0ull;
        if (!v) return;
        switch (threadIdx.x) {
        case BS_PROD: atomicAdd(&ctl->products, v); break;
        case BS_WB: atomicAdd(&ctl->win_bound, v); break;
        case BS_CB: atomicAdd(&ctl->cur_bound, v); break;
        case BS_CBD: atomicAdd(&ctl->cur_bound_ds, v); break;
        case BS_WDP: atomicAdd(&ctl->wide_ds_prod, v); break;
        case BS_SPAN: atomicAdd(reinterpret_cast<unsigned long long *>(&ctl->span_tiles), v); break;
        default: atomicAdd(&ctl->bin_count[threadIdx.x - BS_BIN], (int)v);
        }
    }
};

// long_list: rows of more than SUM_LONG entries are listed there (ctl->long_rows of them) for
// k_bounds_long; nullptr: every row is taken here
template <int G>
__global__ void __launch_bounds__(SUM_THREADS) k_bounds(int M, const int *__restrict__ arp,
                                                        const int *__restrict__ acol, const int *__restrict__ brp,
                                                        const int *__restrict__ bcol, int N, RowInfo ri,
                                                        int *__restrict__ long_list, ClassLine line, Ctl *ctl) {
    constexpr int RPB = SUM_THREADS / G;  // rows per block iteration
    __shared__ BoundsSmem s_tot;
    const int sub = threadIdx.x & (G - 1);
    BoundsSums mine;
    for (int rb = blockIdx.x * RPB; rb < M; rb += gridDim.x * RPB) {
        const int i = rb + (int)threadIdx.x / G;
        const int lo = i < M ? arp[i] : 0, hi = i < M ? arp[i + 1] : 0;
        const bool listed = long_list && hi - lo > SUM_LONG;
        RowSums<true> r;
        r.walk(sub, listed ? 0 : hi - lo, G, acol + lo, brp, bcol);
        r.template reduce<G>();
        if (i < M && sub == 0) {
            if (listed) long_list[atomicAdd(&ctl->long_rows, 1)] = i;
            else mine.row(i, hi - lo, r, N, ri, line);
        }
    }
    mine.flush(s_tot, ctl);
}

__global__ void __launch_bounds__(SUM_THREADS) k_bounds_long(const int *__restrict__ arp, const int *__restrict__ acol,
                                                             const int *__restrict__ brp, const int *__restrict__ bcol,
                                                             int N, RowInfo ri, const int *__restrict__ long_list,
                                                             ClassLine line, Ctl *ctl) {
    __shared__ SumSmem s_sum;
    __shared__ BoundsSmem s_tot;
    BoundsSums mine;
    const int n = ctl->long_rows;
    for (int e = blockIdx.x; e < n; e += gridDim.x) {
        const int i = long_list[e];
        const int lo = arp[i], hi = arp[i + 1];
        const RowSums<true> r = block_row_sums<true>(lo, hi, acol, brp, bcol, s_sum);
        if (threadIdx.x == 0) mine.row(i, hi - lo, r, N, ri, line);
    }
    mine.flush(s_tot, ctl);
}

// ---------------------------------------------------------------- block scan
constexpr int SCAN_T = 256;
constexpr int SCAN_IPT = 8;
constexpr int SCAN_ITEMS = SCAN_T * SCAN_IPT;

// exclusive block scan of one long long per thread; returns block total
__device__ __forceinline__ long long block_excl_scan(long long v, long long *s_warp, long long &total) {
    const int lane = lane_id(), w = threadIdx.x >> 5;
    long long incl = warp_incl_scan(v);
    if (lane == 31) s_warp[w] = incl;
    __syncthreads();
    if (w == 0) {
        long long x = lane < (SCAN_T / 32) ? s_warp[lane] : 0;
        long long xi = warp_incl_scan(x);
        if (lane < (SCAN_T / 32)) s_warp[lane] = xi - x;
        if (lane == 31) s_warp[SCAN_T / 32] = xi;
    }
    __syncthreads();
    total = s_warp[SCAN_T / 32];
    long long r = incl - v + s_warp[w];
    __syncthreads();
    return r;
}

// exclusive scan of n ints, `chunks` of SCAN_ITEMS per tile; in and out may be the same array (a
// block reads each of its chunks before it writes it).  int output saturates, and a total beyond
// INT_MAX sets DERR_OVERFLOW.
template <class T>
__global__ void __launch_bounds__(SCAN_T) k_scan_lb(const int *in, T *out, int n, int chunks, int ntiles,
                                                    long long *total64, LookBack lb, Ctl *ctl, bool gated) {
    if (gated && !tiles_read(ctl)) return;  // every block: no ticket is taken
    __shared__ long long s_warp[SCAN_T / 32 + 1];
    __shared__ long long s_prefix;
    __shared__ int s_tile;
    if (threadIdx.x == 0) s_tile = lb_ticket(lb);
    __syncthreads();
    const int tile = s_tile;
    const long long lo = (long long)tile * chunks * SCAN_ITEMS + (long long)threadIdx.x * SCAN_IPT;
    int vals[SCAN_IPT];
    long long v = 0;
    for (int c = 0; c < chunks; c++) {
        const long long base = lo + (long long)c * SCAN_ITEMS;
#pragma unroll
        for (int j = 0; j < SCAN_IPT; j++) {
            vals[j] = base + j < n ? in[base + j] : 0;
            v += vals[j];
        }
    }
    long long sum;
    const long long ex0 = block_excl_scan(v, s_warp, sum);
    if (threadIdx.x < WARP) {
        const unsigned long long p = lb_prefix(lb, 0, tile, (unsigned long long)sum, ctl);
        if (threadIdx.x == 0) {
            s_prefix = (long long)p;
            lb_done(lb, ntiles);
        }
    }
    __syncthreads();
    long long run = s_prefix;
    auto put = [&](long long at, long long x) {
        if (sizeof(T) == 4) out[at] = (T)(x < (long long)INT_MAX ? x : (long long)INT_MAX);
        else out[at] = (T)x;
    };
    if (tile == ntiles - 1 && threadIdx.x == 0) {
        const long long total = run + sum;
        *total64 = total;
        put(n, total);
        if (sizeof(T) == 4 && total > (long long)INT_MAX) set_err(&ctl->err, DERR_OVERFLOW);
    }
    for (int c = 0; c < chunks; c++) {
        const long long base = lo + (long long)c * SCAN_ITEMS;
        long long ex = ex0, tot = sum;
        if (chunks > 1) {
            v = 0;
#pragma unroll
            for (int j = 0; j < SCAN_IPT; j++) {
                vals[j] = base + j < n ? in[base + j] : 0;
                v += vals[j];
            }
            ex = block_excl_scan(v, s_warp, tot);
        }
        ex += run;
#pragma unroll
        for (int j = 0; j < SCAN_IPT; j++) {
            if (base + j < n) put(base + j, ex);
            ex += vals[j];
        }
        run += tot;
    }
}

LookBack next_epoch(ScanState &s, cudaStream_t st) {
    if (++s.epoch >> LB_EPOCH_BITS) {  // the words of the launches before must not match again
        cudaMemsetAsync(s.word, 0, scan_state_bytes(), st);
        s.epoch = 1;
    }
    unsigned long long *w = reinterpret_cast<unsigned long long *>(s.word);
    return LookBack{reinterpret_cast<unsigned *>(w + (size_t)LB_STREAMS * LB_TILES), w, s.epoch,
                    s.polls > 0 ? s.polls : LB_POLLS};
}

size_t scan_state_bytes() { return sizeof(unsigned long long) * ((size_t)LB_STREAMS * LB_TILES + 1); }

void launch_scan(const int *in, int *out, int n, long long *total64, ScanState &scan, Ctl *ctl, cudaStream_t st,
                 bool gated) {
    int chunks;
    const int nt = lb_tiles(n, SCAN_ITEMS, chunks);
    k_scan_lb<int><<<nt, SCAN_T, 0, st>>>(in, out, n, chunks, nt, total64, next_epoch(scan, st), ctl, gated);
}

void launch_scan64(const int *in, long long *out, int n, long long *total64, ScanState &scan, Ctl *ctl,
                   cudaStream_t st) {
    int chunks;
    const int nt = lb_tiles(n, SCAN_ITEMS, chunks);
    k_scan_lb<long long><<<nt, SCAN_T, 0, st>>>(in, out, n, chunks, nt, total64, next_epoch(scan, st), ctl, false);
}

// Stable binning in one pass: every row at its place in its class's bin, rows in ascending order
// (row panels are slices of the bins).
__global__ void __launch_bounds__(BIN_T) k_bins(int M, const signed char *__restrict__ cls, int rows, int ntiles,
                                                int *__restrict__ bins, LookBack lb, Ctl *ctl) {
    __shared__ BinSmem<NBIN> S;
    const int tile = lb_tile(lb, &S.tile);
    bin_tile<NBIN>(cls, tile, rows, M, ntiles, lb, ctl, S,
                   [&](int b, int at, int i) { bins[(size_t)b * M + at] = i; });
}

static void launch_bins(int M, const RowInfo &ri, ScanState &scan, Ctl *ctl, cudaStream_t st) {
    if (M <= 0) return;
    int chunks;
    const int nt = lb_tiles(M, BIN_ROWS, chunks);
    k_bins<<<nt, BIN_T, 0, st>>>(M, ri.cls, chunks * BIN_ROWS, nt, ri.bins, next_epoch(scan, st), ctl);
}

void launch_bounds(const DevCSR &A, const DevCSR &B, RowInfo ri, Ctl *ctl, int grid, ScanState &scan, cudaStream_t st,
                   bool counts_only) {
    // an average warp's share of the products, by the averages of A's and B's rows: 24 warps per SM in the
    // fused row kernel, 48 in the count pass
    const float share = B.M ? (float)((double)A.nnz * (double)B.nnz / B.M / (grid * (counts_only ? 6.0 : 3.0))) : 0.f;
    const ClassLine line{fmaxf((float)DS_TILES, share), counts_only ? LLONG_MAX : max(DS_PROD, (long long)share)};
    const double avg = A.M ? (double)A.nnz / A.M : 0.0;
    // the bins are written after this pass: until then their space holds the long rows
    int *list = long_rows_apart(A) ? ri.bins : nullptr;
    const int lanes = avg <= 6 ? 4 : avg <= 12 ? 8 : avg <= 24 ? 16 : 32;
    auto k = avg <= 6 ? k_bounds<4> : avg <= 12 ? k_bounds<8> : avg <= 24 ? k_bounds<16> : k_bounds<32>;
    k<<<grid_for(grid, A.M, SUM_THREADS / lanes), SUM_THREADS, 0, st>>>(A.M, A.rp, A.col, B.rp, B.col, B.N, ri, list,
                                                                        line, ctl);
    if (list) k_bounds_long<<<grid / 2, SUM_THREADS, 0, st>>>(A.rp, A.col, B.rp, B.col, B.N, ri, list, line, ctl);
    launch_bins(A.M, ri, scan, ctl, st);
}

// products of every PROD_CHUNK consecutive rows: one warp per chunk (the host
// orders its row panels by them)
__global__ void __launch_bounds__(256) k_chunk_prod(int M, const long long *__restrict__ prod,
                                                    long long *__restrict__ out) {
    static_assert(PROD_CHUNK == 2 * WARP, "two rows per lane");
    const int nch = (M + PROD_CHUNK - 1) / PROD_CHUNK;
    const int lane = lane_id();
    for (int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < nch; c += (gridDim.x * blockDim.x) >> 5) {
        const int r0 = c * PROD_CHUNK + lane, r1 = r0 + WARP;
        long long v = (r0 < M ? prod[r0] : 0ll) + (r1 < M ? prod[r1] : 0ll);
        v = warp_sum(v);
        if (lane == 0) out[c] = v;
    }
}

// row pointers of rows r0..r1-1 as a panel of its own: crp[r0] = 0
__global__ void __launch_bounds__(256) k_panel_ptr(const long long *__restrict__ rp, int r0, int r1,
                                                   int *__restrict__ crp) {
    const long long first = rp[r0];
    for (long long i = r0 + blockIdx.x * (long long)blockDim.x + threadIdx.x; i <= r1;
         i += (long long)gridDim.x * blockDim.x)
        crp[i] = (int)(rp[i] - first);
}

void launch_panel_ptr(const long long *rp, int r0, int r1, int *crp, int grid, cudaStream_t st) {
    k_panel_ptr<<<grid_for(grid, (long long)r1 - r0 + 1, 256), 256, 0, st>>>(rp, r0, r1, crp);
}

void launch_chunk_prod(int M, const long long *prod, long long *out, int grid, cudaStream_t st) {
    if (M > 0) k_chunk_prod<<<grid, 256, 0, st>>>(M, prod, out);
}

// ---------------------------------------------------------------- scan in three launches
// for callers without a handle (the allocation-free tile conversion, the AMG generators)
__global__ void __launch_bounds__(SCAN_T) k_scan_sums(const int *__restrict__ in, int n, long long *bsum) {
    __shared__ long long s_warp[SCAN_T / 32 + 1];
    const long long base = (long long)blockIdx.x * SCAN_ITEMS + threadIdx.x * SCAN_IPT;
    long long v = 0;
#pragma unroll
    for (int j = 0; j < SCAN_IPT; j++)
        if (base + j < n) v += in[base + j];
    long long tot;
    block_excl_scan(v, s_warp, tot);
    if (threadIdx.x == 0) bsum[blockIdx.x] = tot;
}

__global__ void __launch_bounds__(SCAN_T) k_scan_top(long long *bsum, int nb, long long *total64) {
    __shared__ long long s_warp[SCAN_T / 32 + 1];
    long long carry = 0;
    for (int b0 = 0; b0 < nb; b0 += SCAN_T) {
        const int b = b0 + threadIdx.x;
        long long v = b < nb ? bsum[b] : 0;
        long long tot;
        long long ex = block_excl_scan(v, s_warp, tot);
        if (b < nb) bsum[b] = ex + carry;
        carry += tot;
    }
    if (threadIdx.x == 0) *total64 = carry;
}

// in and out may be the same array (in-place scan; the allocation-free tile conversion and the
// AMG generators rely on it), so neither is __restrict__: every thread loads its SCAN_IPT items
// into registers before the block scan's barriers and afterwards stores only those same items,
// blocks cover disjoint ranges, and out[n] lies past every item read.
__global__ void __launch_bounds__(SCAN_T) k_scan_out(const int *in, int *out, int n,
                                                     const long long *__restrict__ boff, const long long *total64,
                                                     Ctl *ctl) {
    __shared__ long long s_warp[SCAN_T / 32 + 1];
    const long long base = (long long)blockIdx.x * SCAN_ITEMS + threadIdx.x * SCAN_IPT;
    int vals[SCAN_IPT];
    long long v = 0;
#pragma unroll
    for (int j = 0; j < SCAN_IPT; j++) {
        vals[j] = base + j < n ? in[base + j] : 0;
        v += vals[j];
    }
    long long tot;
    long long ex = block_excl_scan(v, s_warp, tot) + boff[blockIdx.x];
    const bool ovf = *total64 > (long long)INT_MAX;
#pragma unroll
    for (int j = 0; j < SCAN_IPT; j++) {
        if (base + j < n) out[base + j] = ovf ? 0 : (int)ex;
        ex += vals[j];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        out[n] = ovf ? 0 : (int)*total64;
        if (ovf) set_err(&ctl->err, DERR_OVERFLOW);
    }
}

size_t scan_tmp_ints(int n) {
    const int nb = (n + SCAN_ITEMS - 1) / SCAN_ITEMS;
    return (size_t)(nb > 0 ? nb : 1) * 2 + 2;
}

void launch_scan3(const int *in, int *out, int n, long long *total64, int *tmp, Ctl *ctl, cudaStream_t st) {
    const int nb = n > 0 ? (n + SCAN_ITEMS - 1) / SCAN_ITEMS : 1;
    long long *bsum = reinterpret_cast<long long *>(tmp);
    k_scan_sums<<<nb, SCAN_T, 0, st>>>(in, n, bsum);
    k_scan_top<<<1, SCAN_T, 0, st>>>(bsum, nb, total64);
    k_scan_out<<<nb, SCAN_T, 0, st>>>(in, out, n, bsum, total64, ctl);
}

}  // namespace hsmu
