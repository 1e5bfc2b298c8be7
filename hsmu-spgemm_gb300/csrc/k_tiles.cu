// Stage 1: B (CSR, sorted rows) -> 64-column bit tiles.
//
// GB300 counterpart of the reference's Initialize_compressed_mask64_matrix
// (src/compressed/compressed_mask64.cuh:343-424: compute_tile64_nums :61-152,
// k_compute_flop, the CUB scan, compute_tile64_col :153-246 and
// compute_tile64_mask_num :248-342).  The reference builds shared-memory
// bitmaps per row partition, copies tile_ptr to the host and partitions on
// the host; here one warp walks each sorted B row 32 entries at a time: a
// tile starts where (col >> 6) changes (ballot + popc), and the tile's u64
// mask is a segmented OR over the lanes of the tile (5 shuffle steps).  Two
// launches (count, fill) around a device scan; no host round trip; tile
// columns come out sorted, and each tile also records the CSR offset of its
// first entry (tile_off) so the numeric phase can jump straight to it.
#include "hsmu_common.cuh"
#include "hsmu_kernels.h"
#include "hsmu_products.cuh"
#include "hsmu_steps.cuh"

namespace hsmu {

// Steps of 32 entries whose loads are in flight.  A hub row of a power-law graph is a chain of hundreds of
// steps, and with one step's load in flight it was the pass's tail: R-MAT scale 18 count 207 -> 120 us, fill
// 385 -> 310 us, scale 15 30 -> 16 and 71 -> 56 us with four.  Rows of one step are taken apart, whole tiles
// straight to their places (count / fill, against the four-step loop for all rows: 150,001 rows of 12 entries
// 16.5 / 33.5 -> 10.4 / 24.5 us, 27-point rows of a 64^3 grid 27.5 / 57.4 -> 19 / 40.2; against a loop of one
// step, by the average of the rows: R-MAT scale 17 of 7.6 entries 57.8 / 130 -> 30 / 85.4, a 5-point Laplacian
// of 4.2 million rows 340 / 880 -> 327 / 791).
constexpr int TILE_U = 4;

// the 32 lanes' column bits, ORed over each run of lanes from a lane to seg_end
__device__ __forceinline__ unsigned long long tile_or(unsigned long long v, int seg_end) {
#pragma unroll
    for (int d = 1; d < WARP; d <<= 1) {
        const unsigned long long o = __shfl_down_sync(FULL, v, d);
        if (lane_id() + d <= seg_end) v |= o;
    }
    return v;
}
// the last lane of the tile that a lane's column lies in, of nvalid lanes
__device__ __forceinline__ int tile_end(unsigned heads, int nvalid) {
    const int lane = lane_id();
    const unsigned above = lane == 31 ? 0u : heads & ~((2u << lane) - 1u);
    return above ? __ffs(above) - 2 : nvalid - 1;
}

template <bool FILL>
__global__ void __launch_bounds__(256) k_tiles(int K, const int *__restrict__ brp, const int *__restrict__ bcol,
                                               int N, int *__restrict__ tcnt_or_ptr, int *__restrict__ tcol,
                                               unsigned long long *__restrict__ tmask, int *__restrict__ toff,
                                               int validate, Ctl *ctl, bool gated) {
    if (gated && !tiles_read(ctl)) return;
    const int lane = lane_id();
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    for (int k = gw; k < K; k += nw) {
        const int s = brp[k], e = brp[k + 1];
        int run = FILL ? tcnt_or_ptr[k] : 0;  // output position (FILL) / count
        if (e - s <= WARP) {  // one step, every tile whole
            const bool valid = lane < e - s;
            const int c = valid ? __ldg(bcol + s + lane) : 0;
            const int cp = __shfl_up_sync(FULL, c, 1);
            const bool head = valid && (lane == 0 || c >> 6 != cp >> 6);
            const unsigned heads = __ballot_sync(FULL, head);
            if (FILL) {
                const unsigned long long v = tile_or(valid ? 1ull << (c & 63) : 0ull, tile_end(heads, e - s));
                if (head) {
                    const int pos = run + __popc(heads & lanemask_lt());
                    tcol[pos] = c >> 6;
                    tmask[pos] = v;
                    toff[pos] = s + lane;
                }
            } else if (lane == 0) {
                tcnt_or_ptr[k] = __popc(heads);
            }
            if (validate && __any_sync(FULL, valid && (c < 0 || c >= N || (lane > 0 && c <= cp))) && lane == 0)
                set_err(&ctl->err, DERR_UNSORTED);
            continue;
        }
        bool have_pend = false;
        int pend_t = -1, pend_off = 0;
        unsigned long long pend_m = 0;
        int prev_col = -1;
        bool bad = false;
        for (StepPos base0 = s; step_in(base0, 0, e); base0 += WARP * TILE_U) {
            int cu[TILE_U];
#pragma unroll
            for (int u = 0; u < TILE_U; u++) {
                cu[u] = step_in(base0, u * WARP + lane, e) ? __ldg(bcol + base0 + u * WARP + lane) : 0;
            }
#pragma unroll
            for (int u = 0; u < TILE_U; u++) {
                if (!step_in(base0, u * WARP, e)) break;
                const int base = (int)base0 + u * WARP;
                const bool valid = step_in(base, lane, e);
                const int c = cu[u];
                if (validate) {
                    int cp = __shfl_up_sync(FULL, c, 1);
                    if (lane == 0) cp = prev_col;
                    if (valid && (c <= cp || c < 0 || c >= N)) bad = true;
                    prev_col = __shfl_sync(FULL, c, WARP - 1);
                }
                const int t = c >> 6;
                int tp = __shfl_up_sync(FULL, t, 1);
                if (lane == 0) tp = have_pend ? pend_t : -1;
                const bool head = valid && (t != tp);
                const unsigned heads = __ballot_sync(FULL, head);
                const int nvalid = min(WARP, e - base);
                if (!FILL) {
                    run += __popc(heads);
                    pend_t = __shfl_sync(FULL, t, nvalid - 1);  // tile open at the end of this chunk
                    have_pend = true;
                    continue;
                }
                const unsigned long long v = tile_or(valid ? 1ull << (c & 63) : 0ull, tile_end(heads, nvalid));
                const unsigned long long lane0_or = __shfl_sync(FULL, v, 0);
                if (have_pend) {
                    if (!(heads & 1u)) pend_m |= lane0_or;  // lane 0 continues the pending tile
                    if (heads) {
                        if (lane == 0) {
                            tcol[run] = pend_t;
                            tmask[run] = pend_m;
                            toff[run] = pend_off;
                        }
                        run++;
                        have_pend = false;
                    }
                }
                if (heads) {
                    const int last = 31 - __clz(heads);
                    if (head && lane != last) {
                        const int pos = run + __popc(heads & lanemask_lt());
                        tcol[pos] = t;
                        tmask[pos] = v;
                        toff[pos] = base + lane;
                    }
                    run += __popc(heads) - 1;
                    pend_t = __shfl_sync(FULL, t, last);
                    pend_m = __shfl_sync(FULL, v, last);
                    pend_off = base + last;
                    have_pend = true;
                }
            }
        }
        if (FILL) {
            if (have_pend && lane == 0) {
                tcol[run] = pend_t;
                tmask[run] = pend_m;
                toff[run] = pend_off;
            }
        } else {
            if (lane == 0) tcnt_or_ptr[k] = run;
        }
        if (validate && __any_sync(FULL, bad) && lane == 0) set_err(&ctl->err, DERR_UNSORTED);
    }
}

void launch_tiles_count(const DevCSR &B, int *tcnt, int validate, Ctl *ctl, int grid, cudaStream_t st, bool gated) {
    k_tiles<false><<<grid_for(grid, B.M, 256 / WARP), 256, 0, st>>>(B.M, B.rp, B.col, B.N, tcnt, nullptr, nullptr,
                                                                    nullptr, validate, ctl, gated);
}

void launch_tiles_fill(const DevCSR &B, const int *tptr, int *tcol, unsigned long long *tmask, int *toff, Ctl *ctl,
                       int grid, cudaStream_t st, bool gated) {
    // five blocks fit an SM: a grid of eight leaves a second wave of three (4.2 million rows 935 us, 791 so); but
    // a gated launch may have nothing to do, and four thousand empty blocks take 4 us
    k_tiles<true><<<grid_for(gated ? grid : 4 * grid, B.M, 256 / WARP), 256, 0, st>>>(B.M, B.rp, B.col, B.N, const_cast<int *>(tptr), tcol,
                                                                   tmask, toff, 0, ctl, gated);
}

// rep[k] = 1 when row k of B holds the same columns as row k - 1 (the rows of one finite-element
// node; the fused row kernel chains their products).  One warp per row, stopped at the first
// difference; a block takes 32 rows, as many as the row kernel looks at together, and counts
// the chains that they form.
__global__ void __launch_bounds__(256) k_row_repeat(int K, const int *__restrict__ brp, const int *__restrict__ bcol,
                                                    unsigned char *__restrict__ rep, int *chains) {
    __shared__ unsigned s_join;  // rows of the 32 that repeat the one before them
    const int lane = lane_id(), w = threadIdx.x >> 5;
    int found = 0;
    for (int k0 = blockIdx.x * WARP; k0 < K; k0 += gridDim.x * WARP) {
        if (threadIdx.x == 0) s_join = 0;
        __syncthreads();
        for (int k = k0 + w; k < min(k0 + WARP, K); k += 256 / WARP) {
            const int s = brp[k], n = brp[k + 1] - s;
            bool same = k > 0 && n > 0 && s - brp[k - 1] == n;
            for (int base = 0; same && base < n; base += WARP) {
                const int i = base + lane;
                same = !__any_sync(FULL, i < n && __ldg(bcol + s + i) != __ldg(bcol + s - n + i));
            }
            if (lane == 0) {
                rep[k] = same;
                if (same) atomicOr(&s_join, 1u << (k - k0));
            }
        }
        __syncthreads();
        if (w == 0) {
            const int pos = lane - (31 - __clz(~(s_join & ~1u) & lanemask_le()));  // place in its run
            found += __popc(__ballot_sync(FULL, k0 + lane < K && pos % REP_MAX == 0));
        }
        __syncthreads();
    }
    if (threadIdx.x == 0 && chains && found) atomicAdd(chains, found);
}

void launch_row_repeat(const DevCSR &B, unsigned char *rep, int *chains, int grid, cudaStream_t st) {
    k_row_repeat<<<grid_for(grid, B.M, WARP), 256, 0, st>>>(B.M, B.rp, B.col, rep, chains);
}

// Validation of A: sorted, unique, in-range columns (one warp per row).
__global__ void __launch_bounds__(256) k_validate(int M, const int *__restrict__ rp, const int *__restrict__ col,
                                                  int N, long long nnz, Ctl *ctl) {
    const int lane = lane_id();
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    bool bad = false;
    for (int i = gw; i < M; i += nw) {
        const int s = rp[i], e = rp[i + 1];
        if (s > e || s < 0 || e > nnz) { bad = true; continue; }
        int prev = -1;
        for (int base = s; base < e; base += WARP) {
            const int idx = base + lane;
            const bool valid = idx < e;
            const int c = valid ? col[idx] : 0;
            int cp = __shfl_up_sync(FULL, c, 1);
            if (lane == 0) cp = prev;
            if (valid && (c <= cp || c < 0 || c >= N)) bad = true;
            prev = __shfl_sync(FULL, c, WARP - 1);
        }
    }
    if (bad) set_err(&ctl->err, DERR_UNSORTED);
}

void launch_validate(const DevCSR &A, Ctl *ctl, int grid, cudaStream_t st) {
    k_validate<<<grid_for(grid, A.M, 256 / WARP), 256, 0, st>>>(A.M, A.rp, A.col, A.N, A.nnz, ctl);
}

}  // namespace hsmu
