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
// rows are binned on the device by a stable compaction (count per 32-row
// chunk, scan, emit), so every bin lists its rows in ascending order and the
// rows of a row panel are one contiguous slice of each bin.
//
// Scan: three launches (block sums, scan of block sums, block scans), 64-bit
// running totals, int32 output; replaces cub::DeviceScan::ExclusiveSum plus
// the full-array D2H copies of the reference
// (src/compressed/compressed_tileOR.cuh:620-622).
#include <climits>

#include "hsmu_common.cuh"
#include "hsmu_kernels.h"
#include "hsmu_rowops.cuh"
#include "hsmu_rowsums.cuh"

namespace hsmu {

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
    __device__ __forceinline__ void row(int i, int len, const RowSums &sums, int N, const RowInfo &ri) {
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
            bin = prod <= TINY_MAX ? BIN_TINY : span <= SPAN_T && prod <= DS_PROD ? BIN_DS : scattered ? BIN_H : BIN_L;
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
                                                        int *__restrict__ long_list, Ctl *ctl) {
    constexpr int RPB = SUM_THREADS / G;  // rows per block iteration
    __shared__ BoundsSmem s_tot;
    const int sub = threadIdx.x & (G - 1);
    BoundsSums mine;
    for (int rb = blockIdx.x * RPB; rb < M; rb += gridDim.x * RPB) {
        const int i = rb + (int)threadIdx.x / G;
        const int lo = i < M ? arp[i] : 0, hi = i < M ? arp[i + 1] : 0;
        const bool listed = long_list && hi - lo > SUM_LONG;
        RowSums r;
        r.walk(lo + sub, listed ? lo : hi, G, acol, brp, bcol);
        r.reduce<G>();
        if (i < M && sub == 0) {
            if (listed) long_list[atomicAdd(&ctl->long_rows, 1)] = i;
            else mine.row(i, hi - lo, r, N, ri);
        }
    }
    mine.flush(s_tot, ctl);
}

__global__ void __launch_bounds__(SUM_THREADS) k_bounds_long(const int *__restrict__ arp, const int *__restrict__ acol,
                                                             const int *__restrict__ brp, const int *__restrict__ bcol,
                                                             int N, RowInfo ri, const int *__restrict__ long_list,
                                                             Ctl *ctl) {
    __shared__ SumSmem s_sum;
    __shared__ BoundsSmem s_tot;
    BoundsSums mine;
    const int n = ctl->long_rows;
    for (int e = blockIdx.x; e < n; e += gridDim.x) {
        const int i = long_list[e];
        const int lo = arp[i], hi = arp[i + 1];
        const RowSums r = block_row_sums(lo, hi, acol, brp, bcol, s_sum);
        if (threadIdx.x == 0) mine.row(i, hi - lo, r, N, ri);
    }
    mine.flush(s_tot, ctl);
}

// stable binning: rows of each class per 32-row chunk (warp per chunk) ...
__global__ void __launch_bounds__(256) k_bin_count(int M, const signed char *__restrict__ cls, int *__restrict__ cnt) {
    const int nch = (M + WARP - 1) / WARP;
    const int lane = lane_id();
    for (int c = (blockIdx.x * blockDim.x + threadIdx.x) / WARP; c < nch; c += gridDim.x * blockDim.x / WARP) {
        const int i = c * WARP + lane;
        const int b = i < M ? cls[i] : -1;
#pragma unroll
        for (int k = 0; k < NBIN; k++) {
            const int n = __popc(__ballot_sync(FULL, b == k));
            if (lane == k) cnt[k * nch + c] = n;
        }
    }
}

// ... then, after the scan of those counts, every row at its place in its bin
__global__ void __launch_bounds__(256) k_bin_emit(int M, const signed char *__restrict__ cls,
                                                  const int *__restrict__ off, int *__restrict__ bins) {
    const int nch = (M + WARP - 1) / WARP;
    const int lane = lane_id();
    for (int c = (blockIdx.x * blockDim.x + threadIdx.x) / WARP; c < nch; c += gridDim.x * blockDim.x / WARP) {
        const int i = c * WARP + lane;
        const int b = i < M ? cls[i] : -1;
#pragma unroll
        for (int k = 0; k < NBIN; k++) {
            const unsigned m = __ballot_sync(FULL, b == k);
            if (b == k) bins[(size_t)k * M + (off[k * nch + c] - off[k * nch]) + __popc(m & lanemask_lt())] = i;
        }
    }
}

size_t bin_scratch_ints(int M) { return (size_t)NBIN * ((M + WARP - 1) / WARP) * 2 + 2; }

void launch_bounds(const DevCSR &A, const DevCSR &B, RowInfo ri, Ctl *ctl, int grid, int *scan_tmp, cudaStream_t st) {
    const double avg = A.M ? (double)A.nnz / A.M : 0.0;
    // the bins are written after this pass: until then their space holds the long rows
    int *list = long_rows_apart(A) ? ri.bins : nullptr;
    auto k = avg <= 6 ? k_bounds<4> : avg <= 12 ? k_bounds<8> : avg <= 24 ? k_bounds<16> : k_bounds<32>;
    k<<<grid, SUM_THREADS, 0, st>>>(A.M, A.rp, A.col, B.rp, B.col, B.N, ri, list, ctl);
    if (list) k_bounds_long<<<grid / 2, SUM_THREADS, 0, st>>>(A.rp, A.col, B.rp, B.col, B.N, ri, list, ctl);
    const int nch = (A.M + WARP - 1) / WARP;
    int *cnt = ri.bin_cnt, *off = ri.bin_cnt + (size_t)NBIN * nch + 1;
    k_bin_count<<<grid, 256, 0, st>>>(A.M, ri.cls, cnt);
    launch_scan(cnt, off, NBIN * nch, &ctl->binned, scan_tmp, ctl, st);
    k_bin_emit<<<grid, 256, 0, st>>>(A.M, ri.cls, off, ri.bins);
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

void launch_chunk_prod(int M, const long long *prod, long long *out, int grid, cudaStream_t st) {
    if (M > 0) k_chunk_prod<<<grid, 256, 0, st>>>(M, prod, out);
}

// ---------------------------------------------------------------- scan
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

__global__ void __launch_bounds__(SCAN_T) k_scan_out64(const int *__restrict__ in, long long *__restrict__ out, int n,
                                                       const long long *__restrict__ boff,
                                                       const long long *total64) {
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
#pragma unroll
    for (int j = 0; j < SCAN_IPT; j++) {
        if (base + j < n) out[base + j] = ex;
        ex += vals[j];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) out[n] = *total64;
}

void launch_scan64(const int *in, long long *out, int n, long long *total64, int *tmp, cudaStream_t st) {
    const int nb = n > 0 ? (n + SCAN_ITEMS - 1) / SCAN_ITEMS : 1;
    long long *bsum = reinterpret_cast<long long *>(tmp);
    k_scan_sums<<<nb, SCAN_T, 0, st>>>(in, n, bsum);
    k_scan_top<<<1, SCAN_T, 0, st>>>(bsum, nb, total64);
    k_scan_out64<<<nb, SCAN_T, 0, st>>>(in, out, n, bsum, total64);
}

size_t scan_tmp_ints(int n) {
    const int nb = (n + SCAN_ITEMS - 1) / SCAN_ITEMS;
    return (size_t)(nb > 0 ? nb : 1) * 2 + 2;
}

void launch_scan(const int *in, int *out, int n, long long *total64, int *tmp, Ctl *ctl, cudaStream_t st) {
    const int nb = n > 0 ? (n + SCAN_ITEMS - 1) / SCAN_ITEMS : 1;
    long long *bsum = reinterpret_cast<long long *>(tmp);
    k_scan_sums<<<nb, SCAN_T, 0, st>>>(in, n, bsum);
    k_scan_top<<<1, SCAN_T, 0, st>>>(bsum, nb, total64);
    k_scan_out<<<nb, SCAN_T, 0, st>>>(in, out, n, bsum, total64, ctl);
}

}  // namespace hsmu
