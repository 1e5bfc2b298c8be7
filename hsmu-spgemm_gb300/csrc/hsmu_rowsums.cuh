// Sums over the B rows that a row of A references: products, tiles (bounds
// pass), longest row, first and last column -- what the bounds pass (k_rows.cu)
// and the learned scheduler's features (learned.cu) are made of.
//
// Bound by L2 latency: three dependent gathers per entry.  A group of G lanes
// takes a row, SUM_U entries per lane in flight; rows of more than SUM_LONG
// entries are listed and taken by a block each in a second launch (in one launch
// a hub row of a power-law graph, thousands of entries on G lanes, or the blocks
// that hold several hubs, ran long after the rest).  R-MAT scale 15: bounds
// 101 -> 17 + 8 us, features 65 -> 12 + 7 us; scale 18: bounds 477 -> 68 + 47 us.
#pragma once
#include "hsmu_common.cuh"
#include "hsmu_steps.cuh"

namespace hsmu {

constexpr int SUM_THREADS = 256;
constexpr int SUM_LONG = 256;
constexpr int SUM_U = 4;

template <bool TILES>
struct RowSums {
    long long prod;  // sum of the B rows' lengths
    float tiles;     // TILES: of the smaller of length and tiles from first to last column (for a dividing
                     // line: single precision will do)
    int longest;     // the longest of them
    int cmin, cmax;  // first and last column (INT_MAX, -1: none)

    // entries first, first + stride, ... of the len from acol on
    __device__ __forceinline__ void walk(int first, int len, int stride, const int *__restrict__ acol,
                                         const int *__restrict__ brp, const int *__restrict__ bcol) {
        prod = 0;
        tiles = 0.f;
        longest = 0;
        cmin = INT_MAX;
        cmax = -1;
        for (StepPos p = first; step_in(p, 0, len); p += stride * SUM_U) {
            int s[SUM_U], e[SUM_U];
#pragma unroll
            for (int u = 0; u < SUM_U; u++) {
                s[u] = e[u] = 0;
                if (step_in(p, u * stride, len)) {
                    const int k = __ldg(acol + p + u * stride);
                    s[u] = __ldg(brp + k);
                    e[u] = __ldg(brp + k + 1);
                }
            }
#pragma unroll
            for (int u = 0; u < SUM_U; u++) {
                prod += e[u] - s[u];
                longest = max(longest, e[u] - s[u]);
                if (e[u] > s[u]) {
                    const int c0 = __ldg(bcol + s[u]), c1 = __ldg(bcol + e[u] - 1);
                    cmin = min(cmin, c0);
                    cmax = max(cmax, c1);
                    if (TILES) tiles += (float)min(e[u] - s[u], (c1 >> 6) - (c0 >> 6) + 1);
                }
            }
        }
    }

    // over the W lanes of a group
    template <int W>
    __device__ __forceinline__ void reduce() {
#pragma unroll
        for (int d = W / 2; d > 0; d >>= 1) {
            prod += __shfl_xor_sync(FULL, prod, d, W);
            if (TILES) tiles += __shfl_xor_sync(FULL, tiles, d, W);
            longest = max(longest, __shfl_xor_sync(FULL, longest, d, W));
            cmin = min(cmin, __shfl_xor_sync(FULL, cmin, d, W));
            cmax = max(cmax, __shfl_xor_sync(FULL, cmax, d, W));
        }
    }
};

struct SumSmem {
    unsigned long long prod;
    float tiles;
    int longest, cmin, cmax;
};

// one long row by the whole block (SUM_THREADS threads, all of them call it); valid on every thread
template <bool TILES>
__device__ __forceinline__ RowSums<TILES> block_row_sums(int lo, int hi, const int *__restrict__ acol,
                                                  const int *__restrict__ brp, const int *__restrict__ bcol,
                                                  SumSmem &S) {
    __syncthreads();  // the previous row's sums have been read
    if (threadIdx.x == 0) {
        S.prod = 0;
        S.tiles = 0.f;
        S.longest = 0;
        S.cmin = INT_MAX;
        S.cmax = -1;
    }
    __syncthreads();
    RowSums<TILES> r;
    r.walk((int)threadIdx.x, hi - lo, SUM_THREADS, acol + lo, brp, bcol);
    r.template reduce<WARP>();
    if (lane_id() == 0) {
        atomicAdd(&S.prod, (unsigned long long)r.prod);
        if (TILES) atomicAdd(&S.tiles, r.tiles);
        atomicMax(&S.longest, r.longest);
        atomicMin(&S.cmin, r.cmin);
        atomicMax(&S.cmax, r.cmax);
    }
    __syncthreads();
    r.prod = (long long)S.prod;
    r.tiles = S.tiles;
    r.longest = S.longest;
    r.cmin = S.cmin;
    r.cmax = S.cmax;
    return r;
}

}  // namespace hsmu
