// Single-pass scans: a look-back over the earlier tiles' sums, and stable
// binning by it (k_rows.cu, k_numeric.cu).
//
// The method is the single-pass prefix scan with decoupled look-back (D. Merrill and
// M. Garland, 2016), with a word layout and bounded waits of this file's own.
//
// One launch instead of three: a block takes the next tile of the input (a
// ticket, so every earlier tile has been started), publishes the tile's sum,
// and looks back over its predecessors' words until one holds a prefix.  A word
// is flag | epoch | value, so one 64-bit store publishes it; words of earlier
// launches carry another epoch and need no clearing.  The ticket counter resets
// itself when the last block is done.  The look-back's polls are bounded: a
// block that gives up sets DERR_TIMEOUT and goes on with what it has, a prefix
// no larger than the right one, so what it writes stays in bounds; the kernels
// that index by the result take no row then (unless_failed, scan_failed).
//
// Small calls are launch-bound: with three launches per scan and two more for the
// binning a Laplacian product had 18, now 10 (64^2 grid 163 -> 130 us, 256^2 210 ->
// 177 us).  Two million items take 36 us (three launches: 32), 65,536 take 4.7 (9).
#pragma once
#include "hsmu_common.cuh"
#include "hsmu_kernels.h"

namespace hsmu {

constexpr int LB_EPOCH_BITS = 18;
constexpr int LB_VALUE_BITS = 44;  // sums saturate there (1.7e13 entries are beyond any memory)
constexpr unsigned long long LB_MAX = (1ull << LB_VALUE_BITS) - 1;
constexpr unsigned long long LB_SUM = 1ull << 62, LB_PREFIX = 2ull << 62;
constexpr int LB_POLLS = 1 << 20;

__device__ __forceinline__ unsigned long long lb_word(unsigned long long flag, unsigned epoch, unsigned long long v) {
    return flag | ((unsigned long long)epoch << LB_VALUE_BITS) | (v < LB_MAX ? v : LB_MAX);
}

// thread 0 of the block: the tile to take
__device__ __forceinline__ int lb_ticket(LookBack lb) { return (int)atomicAdd(&lb.ctr[0], 1u); }
// thread 0, once per block after its ticket and before it ends
__device__ __forceinline__ void lb_done(LookBack lb, int ntiles) {
    if (atomicAdd(&lb.ctr[1], 1u) == (unsigned)ntiles - 1u) {
        lb.ctr[0] = 0;
        lb.ctr[1] = 0;
    }
}

// one whole warp: the sum of `stream`'s tiles before `tile`, whose own sum is `mine`
__device__ __forceinline__ unsigned long long lb_prefix(LookBack lb, int stream, int tile, unsigned long long mine,
                                                        Ctl *ctl) {
    const int lane = lane_id();
    volatile unsigned long long *w = lb.word + (size_t)stream * LB_TILES;
    if (tile == 0) {
        if (lane == 0) w[0] = lb_word(LB_PREFIX, lb.epoch, mine);
        return 0;
    }
    if (lane == 0) w[tile] = lb_word(LB_SUM, lb.epoch, mine);
    unsigned long long sum = 0;
    for (int at = tile - 1; at >= 0; at -= WARP) {  // 32 predecessors, the nearest on lane 0
        const int t = at - lane;
        unsigned long long x = 0;
        bool ready = false;
        for (int poll = 0; poll < lb.polls; poll++) {
            if (t >= 0 && !ready) {
                x = w[t];
                ready = (x >> 62) != 0 && (unsigned)((x >> LB_VALUE_BITS) & ((1u << LB_EPOCH_BITS) - 1u)) == lb.epoch;
            }
            if (__all_sync(FULL, t < 0 || ready)) break;
        }
        const bool gave_up = !__all_sync(FULL, t < 0 || ready);
        if (gave_up) {
            if (lane == 0) set_err(&ctl->err, DERR_TIMEOUT);
            if (!ready) x = 0;
        }
        // lanes up to the nearest prefix count
        const unsigned pre = __ballot_sync(FULL, ready && (x >> 62) == 2);
        const int last = pre ? __ffs(pre) - 1 : WARP - 1;
        sum += warp_sum(t >= 0 && lane <= last ? x & LB_MAX : 0ull);
        if (pre || gave_up) break;
    }
    if (lane == 0) w[tile] = lb_word(LB_PREFIX, lb.epoch, sum + mine);
    return sum;
}

// tiles of a single-pass launch over n items: at most LB_TILES, of `chunks` pieces each
inline int lb_tiles(long long n, int piece, int &chunks) {
    const long long pieces = n > 0 ? (n + piece - 1) / piece : 1;
    chunks = (int)((pieces + LB_TILES - 1) / LB_TILES);
    return (int)((pieces + chunks - 1) / chunks);
}

// the whole block: the tile to take
__device__ __forceinline__ int lb_tile(LookBack lb, int *s_tile) {
    if (threadIdx.x == 0) *s_tile = lb_ticket(lb);
    __syncthreads();
    return *s_tile;
}

// Items of a tile at their places in their classes' lists, in ascending order: a tile counts its items
// of each class, one warp per class looks back, and the items are then placed 256 at a time.
constexpr int BIN_T = 256;
constexpr int BIN_ROWS = 4 * BIN_T;  // items of a piece

template <int NB>
struct BinSmem {
    int cnt[NB], warp[NB][BIN_T / WARP];
    int tile;
};

// The whole block (BIN_T threads), once: tile `tile` of `rows` items each of n; cls[i]: an item's class, -1 for
// none; put(class, place, item).  Returns with cnt holding the classes' counts up to the tile's end.
template <int NB, class Put>
__device__ __forceinline__ void bin_tile(const signed char *cls, int tile, int rows, int n, int ntiles, LookBack lb,
                                         Ctl *ctl, BinSmem<NB> &S, Put put) {
    static_assert(NB <= LB_STREAMS && NB <= BIN_T / WARP, "a look-back stream and a warp per class");
    constexpr int NW = BIN_T / WARP;
    const int lane = lane_id(), w = threadIdx.x >> 5;
    if (threadIdx.x < NB) S.cnt[threadIdx.x] = 0;
    __syncthreads();
    const long long lo = (long long)tile * rows;
    const int r0 = (int)lo, r1 = (int)min(lo + rows, (long long)n);
    int cnt[NB] = {};
    for (int i = r0 + (int)threadIdx.x; i < r1; i += BIN_T) {
        const int b = cls[i];
#pragma unroll
        for (int k = 0; k < NB; k++) cnt[k] += b == k;
    }
#pragma unroll
    for (int k = 0; k < NB; k++) {
        const int c = warp_sum(cnt[k]);
        if (lane == 0 && c) atomicAdd(&S.cnt[k], c);
    }
    __syncthreads();
    if (w < NB) {
        const unsigned long long p = lb_prefix(lb, w, tile, (unsigned long long)S.cnt[w], ctl);
        __syncwarp();
        if (lane == 0) S.cnt[w] = (int)p;  // from here: where the tile's next item of the class goes
    }
    __syncthreads();
    if (threadIdx.x == 0) lb_done(lb, ntiles);
    for (int c0 = r0; c0 < r1; c0 += BIN_T) {
        const int i = c0 + (int)threadIdx.x;
        const int b = i < r1 ? cls[i] : -1;
        unsigned mine = 0;
#pragma unroll
        for (int k = 0; k < NB; k++) {
            const unsigned m = __ballot_sync(FULL, b == k);
            if (b == k) mine = m;
            if (lane == k) S.warp[k][w] = __popc(m);
        }
        __syncthreads();
        if (b >= 0) {
            int at = S.cnt[b] + __popc(mine & lanemask_lt());
            for (int j = 0; j < w; j++) at += S.warp[b][j];
            put(b, at, i);
        }
        __syncthreads();
        if (threadIdx.x < NB)
            for (int j = 0; j < NW; j++) S.cnt[threadIdx.x] += S.warp[threadIdx.x][j];
        __syncthreads();
    }
}

}  // namespace hsmu
