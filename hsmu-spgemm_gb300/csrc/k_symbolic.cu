// Stage 3: exact symbolic count, nnz(C(i,:)) for every row.
//
// GB300 counterpart of the reference's two symbolic passes
// (k_tilePtr_symbolic_* in src/compressed/compressed_tilePtr_symbolic.cuh:174-496,
// which count C tiles with a shared-memory hash, and k_tileOR_* in
// src/compressed/compressed_tileOR.cuh:19-337, which OR the u64 B tile masks
// into those tiles and sum their popcounts).  Both are folded into one pass:
// the row's C tiles are ORed into a dense per-tile table indexed by
// (tile id - first tile of the row), which needs no hashing or probing
// because the bounds kernel already knows the row's exact tile span.
//   BIN_DS rows (span <= SPAN_T, without the rows that stand out): one warp per row,
//                4 KB table per warp.
//   BIN_L  rows: one CTA per row, the span processed in chunks of DCH_COUNT
//                tiles (32 KB); B tile ranges restricted per chunk by binary
//                search when the span needs more than one chunk.
// Every B tile access is a coalesced 4+8 byte load of the flat (A entry,
// B tile) sequence, 32 lanes busy regardless of row lengths.
// Tiny rows are counted here too, without tiles (hsmu_rowops.cuh); scattered
// rows have their own kernels (k_scatter.cu).
// With a tile store, the large-row pass also writes every row's non-empty C
// tiles (id + mask, ascending) to the store, compacted chunk by chunk with one
// block scan, so that the structure pass can stream them (the reference
// likewise keeps C's tiles between its symbolic passes, C->d_tile_col /
// C->d_mask_num, src/compressed/compressed_tileOR.cuh:389-623).
#include "hsmu_block.cuh"
#include "hsmu_kernels.h"
#include "hsmu_rowops.cuh"
#include "hsmu_tilelist.cuh"

namespace hsmu {

constexpr int DS_WARPS = 8;

// Runs of repeated rows of A (rep_a, k_row_repeat) share one C structure: up to RUN_MAX of them are
// counted by the warp of their first row.  place: the row's place in its run (32: in a run too long to
// tell) -- it is the first of a group when run_leads(place).
constexpr int RUN_MAX = 4;
__device__ __forceinline__ int run_place(const unsigned char *__restrict__ rep_a, int i) {
    const int x = i - lane_id();
    const unsigned m = __ballot_sync(FULL, x > 0 && rep_a[x]);
    return m == FULL ? 32 : __ffs(~m) - 1;
}
__device__ __forceinline__ bool run_leads(int place) { return place >= 32 || place % RUN_MAX == 0; }
// rows of the group that row i leads (of M)
__device__ __forceinline__ int run_rows(const unsigned char *__restrict__ rep_a, int i, int place, int M) {
    const int l = lane_id();
    const bool in = l > 0 && l < RUN_MAX && i + l < M && place + l < 32 && rep_a[i + l];
    return __ffs(~(__ballot_sync(FULL, in) | 1u)) - 1;
}

// Rows of the warp class.  A group of repeated rows is counted once: 27-point stencil, 40^3 grid x 3
// dofs 303 -> 114 us.  (The fused row kernel taking such a group with one table gained 1 %: it is
// bound by the FP64 pipe.)

__global__ void __launch_bounds__(DS_WARPS * 32) k_count_ds(int M, const int *__restrict__ arp,
                                                            const int *__restrict__ acol,
                                                            const int *__restrict__ tptr,
                                                            const int *__restrict__ tcol,
                                                            const unsigned long long *__restrict__ tmask,
                                                            RowInfo ri, Ctl *ctl) {
    __shared__ unsigned long long s_mask[DS_WARPS][SPAN_T];
    const int lane = lane_id(), w = threadIdx.x >> 5;
    unsigned long long *msk = s_mask[w];
    const int n = unless_failed(ctl, ctl->bin_count[BIN_DS]);
    const int *rows = ri.bins + (size_t)BIN_DS * M;
    const int nwarps = gridDim.x * DS_WARPS, gw = blockIdx.x * DS_WARPS + w;
    for (int turn = 0; (long long)turn * nwarps < n; turn++) {
        // where repeated rows are counted with the first of them the warps move on by one per turn: a
        // stride that the length of the runs divides would give every first row to the same warps
        const long long r = (long long)turn * nwarps + (ri.rep_a ? (gw + turn) % nwarps : gw);
        if (r >= n) continue;
        const int i = rows[r];
        int nrun = 1;
        if (ri.rep_a) {
            const int place = run_place(ri.rep_a, i);
            if (!run_leads(place)) continue;
            nrun = run_rows(ri.rep_a, i, place, M);
        }
        const int t0 = ri.tmin[i];
        const int span = ri.tmax[i] - t0 + 1;
        for (int t = lane; t < span; t += WARP) msk[t] = 0ull;
        __syncwarp();
        bool bad = false;
        warp_or_tiles<false>(arp[i], arp[i + 1], 0, WARP, acol, tptr, tcol, tmask, t0, span, msk, bad, ri.rep);
        if (bad) set_err(&ctl->err, DERR_INTERNAL);
        __syncwarp();
        int cnt = 0;
        for (int t = lane; t < span; t += WARP) cnt += popc64(msk[t]);
        cnt = warp_sum(cnt);
        if (lane < nrun) {
            ri.cnnz[i + lane] = cnt;
            if (cnt > FUSE_CAP) {  // goes through numeric windows: count them for the cursor array
                atomicAdd(&ctl->wide_rows, 1);
                const unsigned long long wb = cnt / WIN_CUT + (span - 1) / WIN_TCAP + 1;
                atomicAdd(&ctl->cur_bound, wb * (unsigned long long)(arp[i + 1] - arp[i]));
            }
        }
        __syncwarp();
    }
}

// threads of a block, and of an SM's blocks together.  Where no row spans more than SPAN_T tiles the
// large class holds only rows of many products, the heaviest of which is the pass's tail: 16 warps each
// (A*A^T of 30,011 vertices: 257 us with 8, 187 with 16).  Wider rows are mostly lighter, and the
// barriers between their phases cost more in larger blocks (R-MAT scale 18: 5.35 ms with 8, 6.17 with 16).
constexpr int L_WIDE = 256, L_NARROW = 512;
constexpr int L_BLOCK_THREADS = 1536;

// Large rows, one CTA per row: the OR of B's tile masks per chunk of the row's
// tile span, then
//   LM_COUNT  the row's nnz;
//   LM_STORE  also the row's tile list in the arena (the plain path: the
//             structure pass streams it once C is allocated);
//   LM_SPEC   the same in the learned path's speculative pass: the row is
//             flagged ROW_OVERFLOW so that the pass after the exact scan
//             writes it, from its list, straight to its place in C.  (Writing
//             the columns into the predicted slot in this pass, so that the
//             list needs no second pass, was measured slower: R-MAT 18 47.3 ms
//             against 44.1 for the plain path -- the emission lengthens this
//             barrier-bound kernel, and the slot still has to be copied to C.)
// A row that finds the arena full keeps no list (ts.cnt = -1) and is left to
// the OR-walk structure kernel.
enum LMode { LM_COUNT = 0, LM_STORE = 1, LM_SPEC = 2 };

template <int MODE, int L_THREADS>
__global__ void __launch_bounds__(L_THREADS, L_BLOCK_THREADS / L_THREADS) k_count_l(int M, const int *__restrict__ arp,
                                                       const int *__restrict__ acol,
                                                       const int *__restrict__ tptr,
                                                       const int *__restrict__ tcol,
                                                       const unsigned long long *__restrict__ tmask,
                                                       RowInfo ri, TileStore ts, RowOut out, Ctl *ctl) {
    constexpr bool STORE = MODE != LM_COUNT;
    if (scan_failed(ctl)) return;
    constexpr bool SPEC = MODE == LM_SPEC;
    extern __shared__ unsigned long long s_dyn[];
    unsigned long long *msk = s_dyn;  // DCH_COUNT entries
    __shared__ int s_red[L_THREADS / 32];
    __shared__ long long s_tsum[L_THREADS / 32];
    __shared__ ListSmem<L_THREADS / 32> s_ls;
    __shared__ long long s_off;
    __shared__ int s_next;
    const int lane = lane_id(), w = threadIdx.x >> 5;
    constexpr int NWARP = L_THREADS / 32;
    const int n = ctl->bin_count[BIN_L];
    const int *rows = ri.bins + (size_t)BIN_L * M;
    // one row at a time from a counter (RowCounter)
    for (int r = blockIdx.x; r < n;) {
        int next = 0;
        if (threadIdx.x == 0) next = draw_row(&ctl->rows[ROWS_COUNT_L], 0);
        const int i = rows[r];
        const int tmin = ri.tmin[i], tmax = ri.tmax[i];
        const int a_lo = arp[i], a_hi = arp[i + 1];
        const bool one_chunk = (tmax - tmin + 1) <= DCH_COUNT;
        int total = 0;
        ListRun run{0, 0, 0, -1ll};
        long long sbase = -1;
        int scap = 0;
        if (ri.store) {
            // the row's list has at most one C tile per tile of its span and per B tile it
            // reads; the sizes add up to the arena the next call wants
            long long ts_sum = 0;
            for (int p = a_lo + (int)threadIdx.x; p < a_hi; p += L_THREADS) {
                const int k = __ldg(acol + p);
                ts_sum += __ldg(tptr + k + 1) - __ldg(tptr + k);
            }
            ts_sum = warp_sum(ts_sum);
            if (lane == 0) s_tsum[w] = ts_sum;
            __syncthreads();
            long long tsum = 0;
            for (int j = 0; j < NWARP; j++) tsum += s_tsum[j];
            scap = (int)min(tsum, (long long)(tmax - tmin + 1));
            if (threadIdx.x == 0) atomicAdd(reinterpret_cast<unsigned long long *>(&ctl->store_tiles), (unsigned long long)scap);
        }
        if (STORE) {
            // reserve the row's list in the arena (none when it is full)
            if (threadIdx.x == 0) {
                long long o = atomicAdd(reinterpret_cast<unsigned long long *>(&ctl->store_used),
                                        (unsigned long long)scap);
                if (o + scap > ts.cap) o = -1;
                s_off = o;
                ts.off[i] = o;
            }
            __syncthreads();
            sbase = s_off;
        }
        for (int c0 = tmin; c0 <= tmax; c0 += DCH_COUNT) {
            const int c1 = min(c0 + DCH_COUNT, tmax + 1);
            for (int t = threadIdx.x; t < c1 - c0; t += L_THREADS) msk[t] = 0ull;
            __syncthreads();
            bool bad = false;
            if (one_chunk)
                warp_or_tiles<false, true, L_THREADS == L_WIDE>(a_lo, a_hi, w * WARP, NWARP * WARP, acol, tptr, tcol, tmask, c0, c1 - c0, msk, bad);
            else
                warp_or_tiles<true, true, L_THREADS == L_WIDE>(a_lo, a_hi, w * WARP, NWARP * WARP, acol, tptr, tcol, tmask, c0, c1 - c0, msk, bad);
            if (bad) set_err(&ctl->err, DERR_INTERNAL);
            __syncthreads();
            if (STORE && sbase >= 0) {
                // the chunk's non-empty tiles appended to the row's list, with their slots
                // and window starts (hsmu_tilelist.cuh)
                if (!chunk_to_list<NWARP>(msk, c1 - c0, c0, tmin, run, s_ls, sbase, scap, ts.tcol, ts.tent) &&
                    threadIdx.x == 0)
                    set_err(&ctl->err, DERR_INTERNAL);
                total = run.slots;
            } else {
                int cnt = 0;
                for (int t = threadIdx.x; t < c1 - c0; t += L_THREADS) cnt += popc64(msk[t]);
                cnt = warp_sum(cnt);
                if (lane == 0) s_red[w] = cnt;
                __syncthreads();
                if (threadIdx.x == 0) {
                    int s = 0;
                    for (int j = 0; j < NWARP; j++) s += s_red[j];
                    total += s;
                }
            }
            __syncthreads();
        }
        const bool listed = STORE && sbase >= 0 && run.tiles <= scap;
        if (threadIdx.x == 0) {
            ri.cnnz[i] = total;
            if (STORE) {
                ts.cnt[i] = listed ? run.tiles : -1;  // over the capacity: reported above
                ts.nwin[i] = listed ? run.wins : 0;   // scanned in row order into the rows' first windows
            }
            if (SPEC) out.flag[i] = listed ? ROW_OVERFLOW : ROW_NONE;  // unlisted: the OR-walk kernel
            s_next = next;
        }
        __syncthreads();
        r = s_next;
        __syncthreads();
    }
    if (threadIdx.x == 0) rows_done(&ctl->rows[ROWS_COUNT_L]);
}

constexpr int TINY_THREADS = 256;

// tiny rows: one thread per row, a warp's rows by one network (hsmu_rowops.cuh)
__global__ void __launch_bounds__(TINY_THREADS) k_count_tiny(int M, const int *__restrict__ arp,
                                                             const int *__restrict__ acol,
                                                             const int *__restrict__ brp,
                                                             const int *__restrict__ bcol, RowInfo ri, Ctl *ctl) {
    __shared__ int s_q[TINY_THREADS / WARP][TINY_MAX][WARP];
    int (*qs)[WARP] = s_q[threadIdx.x >> 5];
    const int n = unless_failed(ctl, ctl->bin_count[BIN_TINY]);
    const int *rows = ri.bins + (size_t)BIN_TINY * M;
    bool bad = false;
    for (int r0 = blockIdx.x * TINY_THREADS + (threadIdx.x & ~31); r0 < n; r0 += gridDim.x * TINY_THREADS) {
        const int r = r0 + lane_id();
        const int i = r < n ? rows[r] : -1;
        const int a_lo = i >= 0 ? arp[i] : 0, a_hi = i >= 0 ? arp[i + 1] : 0;
        if (__all_sync(FULL, a_hi - a_lo <= 1)) {  // one entry of A each: its B row
            if (i < 0) continue;
            const int k = a_lo < a_hi ? __ldg(acol + a_lo) : -1;
            ri.cnnz[i] = k >= 0 ? __ldg(brp + k + 1) - __ldg(brp + k) : 0;
            continue;
        }
        const int np = tiny_list<false>(a_lo, a_hi, acol, nullptr, brp, qs, nullptr);
        const int most = __reduce_max_sync(FULL, np);
        int c;
        if (most > TINY_MAX) {  // a row of another class
            bad = true;
            c = 0;
        } else if (most <= 8) {
            c = tiny_list_count<8>(np, bcol, qs);
        } else if (most <= 16) {
            c = tiny_list_count<16>(np, bcol, qs);
        } else {
            c = tiny_list_count<32>(np, bcol, qs);
        }
        if (i >= 0) ri.cnnz[i] = c;
    }
    if (bad) set_err(&ctl->err, DERR_INTERNAL);
}

void launch_count_light(const DevCSR &A, const DevCSR &B, RowInfo ri, Ctl *ctl, int nsm, cudaStream_t st) {
    k_count_tiny<<<grid_for(nsm * 4, A.M, TINY_THREADS), TINY_THREADS, 0, st>>>(A.M, A.rp, A.col, B.rp, B.col, ri, ctl);
    if (B.N > SPAN_T * 64) launch_count_scattered(A, B, ri, ctl, nsm, st);  // else no row's span is that wide
}

void launch_count_warp(const DevCSR &A, const DevTiles &Bt, RowInfo ri, Ctl *ctl, int nsm, cudaStream_t st) {
    k_count_ds<<<grid_for(nsm * 6, A.M, DS_WARPS), DS_WARPS * 32, 0, st>>>(A.M, A.rp, A.col, Bt.ptr, Bt.col, Bt.mask, ri, ctl);
}

template <int MODE, int NT>
static void count_large(const DevCSR &A, const DevTiles &Bt, const RowInfo &ri, const TileStore &ts, const RowOut &out,
                        Ctl *ctl, int nsm, cudaStream_t st) {
    const size_t smem = DCH_COUNT * sizeof(unsigned long long);
    k_count_l<MODE, NT><<<grid_for(nsm * (L_BLOCK_THREADS / NT), A.M, 1), NT, smem, st>>>(A.M, A.rp, A.col, Bt.ptr, Bt.col,
                                                                                     Bt.mask, ri, ts, out, ctl);
}

void launch_count_large(const DevCSR &A, const DevTiles &Bt, int N, RowInfo ri, const TileStore *ts, Ctl *ctl, int nsm,
                        cudaStream_t st) {
    const bool store = ts && ts->tcol && ts->tent && ts->cap > 0 && ri.store, narrow = N <= SPAN_T * 64;
    if (store && narrow) count_large<LM_STORE, L_NARROW>(A, Bt, ri, *ts, RowOut{}, ctl, nsm, st);
    else if (store) count_large<LM_STORE, L_WIDE>(A, Bt, ri, *ts, RowOut{}, ctl, nsm, st);
    else if (narrow) count_large<LM_COUNT, L_NARROW>(A, Bt, ri, TileStore{}, RowOut{}, ctl, nsm, st);
    else count_large<LM_COUNT, L_WIDE>(A, Bt, ri, TileStore{}, RowOut{}, ctl, nsm, st);
}

void launch_spec_large(const DevCSR &A, const DevTiles &Bt, int N, RowInfo ri, const TileStore &ts, RowOut out, Ctl *ctl,
                       int nsm, cudaStream_t st) {
    if (N <= SPAN_T * 64) count_large<LM_SPEC, L_NARROW>(A, Bt, ri, ts, out, ctl, nsm, st);
    else count_large<LM_SPEC, L_WIDE>(A, Bt, ri, ts, out, ctl, nsm, st);
}

void launch_count(const DevCSR &A, const DevCSR &B, const DevTiles &Bt, RowInfo ri, Ctl *ctl, int nsm,
                  cudaStream_t st) {
    launch_count_light(A, B, ri, ctl, nsm, st);
    launch_count_warp(A, Bt, ri, ctl, nsm, st);
    launch_count_large(A, Bt, B.N, ri, nullptr, ctl, nsm, st);
}

int configure_count() {
    for (auto k : {k_count_l<LM_COUNT, L_WIDE>, k_count_l<LM_STORE, L_WIDE>, k_count_l<LM_SPEC, L_WIDE>,
                   k_count_l<LM_COUNT, L_NARROW>, k_count_l<LM_STORE, L_NARROW>, k_count_l<LM_SPEC, L_NARROW>}) {
        const int e = (int)cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                DCH_COUNT * (int)sizeof(unsigned long long));
        if (e) return e;
    }
    return 0;
}

}  // namespace hsmu
