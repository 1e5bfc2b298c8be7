// Scattered rows (class BIN_H): at most H_ROW entries of A and H_MAX
// intermediate products spread over more than SPAN_T tiles, as in uniformly
// random matrices and the lighter rows of power-law graphs.  One warp per row.
//
// The CTA-per-row passes (k_count_l, k_struct_ls, k_numeric) clear and scan a
// dense table of the row's whole tile span and hand the row on through a tile
// list, windows and cursors; for a row of a few hundred products that is nearly
// all of its time.  Here the row's products are read once into registers (lane
// l of step s holds product 32 s + l of the flat (A entry, B entry) order) and
// put in order by ranks: an occupancy bitmap over the tiles of the span, set by
// every product and prefix-counted, numbers the row's tiles in ascending order;
// every product then sets its column's bit in its tile's mask, and a prefix
// count of the masks gives each tile's first slot.  Linear in the products: no
// sort, no search, one bit of shared memory per tile of the span.
//
// Values: when the row has as many entries as products (no column twice, the
// usual case) every product is its entry; otherwise the products are added to
// an accumulator step by step, lanes that share a slot in lane order -- the
// oracle's order, 0.0 + p_1 + p_2 + ..., either way.
//
// Bound by instruction issue (1,600 warp instructions a row, 47 % of the issue slots) and latency.
// Measured on 150,001 rows of 12 uniform columns (144 products per row): count 155 us, fill 414 us
// (166 and 432 before a row's range and A columns were read during the row ahead of it; a form that read
// the products again and looked every slot up: 191 and 646; the CTA-per-row passes: count 1,889,
// structure 379, cursors 55, values 362 us).
#include "hsmu_block.cuh"
#include "hsmu_kernels.h"
#include "hsmu_products.cuh"
#include "hsmu_rowops.cuh"
#include "hsmu_tilelist.cuh"

namespace hsmu {

constexpr int H_OCCW = H_SPAN / 64;
constexpr int H_STEPS = H_MAX / WARP;
static_assert(H_ROW == WARP, "one lane per A entry");

struct HSmem {
    unsigned long long tmask[H_MAX];  // a tile's columns, by rank; then the accumulator
    unsigned long long occ[H_OCCW];
    unsigned short opre[H_OCCW];      // tiles before each word of occ; then the conflict stamps
    unsigned short tbase[H_MAX];
    unsigned short tid[H_MAX];        // tile id less the row's first tile, by rank
};
static_assert(sizeof(unsigned short) * H_OCCW >= H_MAX, "a stamp per slot");

// One row's products, a lane holding one per step: column (-1: none) and, for VALS, the term and
// A value of add_term.
template <int AR, bool VALS>
struct HProducts {
    int n;  // products of the row, -1: more than the class holds
    int c[H_STEPS];
    double p[VALS ? H_STEPS : 1];
    double av[VALS && AR == AR_FMA ? H_STEPS : 1];

    // k: the lane's A entry's column (HRows)
    __device__ __forceinline__ void load(int a_lo, int a_hi, int k, const double *__restrict__ aval,
                                         const int *__restrict__ brp, const int *__restrict__ bcol,
                                         const double *__restrict__ bval) {
        const int lane = lane_id();
        int lo = 0, len = 0;
        double a = 0.0;
        if (a_lo + lane < a_hi) {
            if (VALS) a = __ldg(aval + a_lo + lane);
            lo = __ldg(brp + k);
            len = __ldg(brp + k + 1) - lo;
        }
        const int incl = warp_incl_scan(len);
        n = __shfl_sync(FULL, incl, WARP - 1);
        if (n <= 0 || n > H_MAX || a_hi - a_lo > H_ROW) {
            n = -1;
            return;
        }
        // the non-empty B rows packed into the first lanes: flat start, entry shift, A value
        const unsigned ne = __ballot_sync(FULL, len > 0);
        const int nseg = __popc(ne);
        const int src = nth_set_bit(ne, min(lane, nseg - 1));
        const int st = __shfl_sync(FULL, incl - len, src);
        const int d = __shfl_sync(FULL, lo - (incl - len), src);
        if (VALS) a = __shfl_sync(FULL, a, src);
        const int start = lane < nseg ? st : INT_MAX;
        int before = 0;
#pragma unroll
        for (int s = 0; s < H_STEPS; s++) {
            c[s] = -1;
            if (s * WARP < n) {
                const unsigned rel = (unsigned)(start - s * WARP);
                const unsigned sm = __reduce_or_sync(FULL, rel < 32u ? 1u << rel : 0u);
                const int sg = before + __popc(sm & lanemask_le()) - 1;
                before += __popc(sm);
                const int g = s * WARP + lane;
                const int e = g + __shfl_sync(FULL, d, sg);
                const bool v = g < n;
                if (v) c[s] = __ldg(bcol + e);
                if (VALS) {
                    const double as = __shfl_sync(FULL, a, sg);
                    p[s] = term<AR>(as, v ? __ldg(bval + e) : 0.0);
                    if (AR == AR_FMA) av[s] = as;
                }
            }
        }
    }
};

// A warp's rows of a class list, the next one's A range and A columns read while the current one is
// computed: two of a row's four dependent round trips to memory.
struct HRows {
    const int *rows, *arp, *acol;
    int end, stride, r;
    int i, a_lo, a_hi, k;  // the current row (i < 0: none), its A range, the lane's A column

    __device__ __forceinline__ void range() {
        a_lo = i >= 0 ? __ldg(arp + i) : 0;
        a_hi = i >= 0 ? __ldg(arp + i + 1) : 0;
    }
    __device__ __forceinline__ void column() { k = a_lo + lane_id() < a_hi ? __ldg(acol + a_lo + lane_id()) : 0; }
    __device__ __forceinline__ void row() { i = r < end ? rows[r] : -1; }
    __device__ __forceinline__ HRows(const int *rows, const int *arp, const int *acol, int begin, int end, int stride)
        : rows(rows), arp(arp), acol(acol), end(end), stride(stride), r(begin) {
        row();
        range();
        column();
    }
    // the next row's first step; range() and column() follow
    __device__ __forceinline__ void next() {
        r += stride;
        row();
    }
};

// Ranks the tiles of a row's products (first tile t0, `span` tiles): tmask by rank, and for FILL
// each tile's id in tid and rank << 6 | column bit in every product's c.  Returns the number of
// tiles, -1 (nothing usable) for a column outside.
// `midway` runs once, between the passes.
template <bool FILL, class P, class F>
__device__ __forceinline__ int h_order(P &R, int t0, int span, HSmem &S, F midway) {
    const int lane = lane_id();
    const int nw = (span + 63) >> 6;
    if (R.n < 0 || span <= 0 || nw > H_OCCW) {
        midway();
        return -1;
    }
    for (int q = lane; q < nw; q += WARP) S.occ[q] = 0ull;
    __syncwarp();
    bool bad = false;
#pragma unroll
    for (int s = 0; s < H_STEPS; s++) {
        if (s * WARP >= R.n) break;
        const int t = (R.c[s] >> 6) - t0;
        if (R.c[s] >= 0) {
            if ((unsigned)t < (unsigned)span) smem_setbit64(&S.occ[t >> 6], t & 63);
            else bad = true;
        }
    }
    midway();
    if (__any_sync(FULL, bad)) return -1;  // the vote orders the warp's shared accesses as well
    __syncwarp();
    const int per = (nw + WARP - 1) / WARP;
    const int q0 = min(nw, lane * per), q1 = min(nw, q0 + per);
    int sum = 0;
    for (int q = q0; q < q1; q++) sum += popc64(S.occ[q]);
    const int incl = warp_incl_scan(sum);
    const int ntiles = __shfl_sync(FULL, incl, WARP - 1);  // at most n
    int run = incl - sum;
    for (int q = q0; q < q1; q++) {
        S.opre[q] = (unsigned short)run;
        run += popc64(S.occ[q]);
    }
    for (int q = lane; q < ntiles; q += WARP) S.tmask[q] = 0ull;
    __syncwarp();
#pragma unroll
    for (int s = 0; s < H_STEPS; s++) {
        if (s * WARP >= R.n) break;
        if (R.c[s] >= 0) {
            const int t = (R.c[s] >> 6) - t0;
            const int r = S.opre[t >> 6] + rank64(S.occ[t >> 6], t & 63);
            smem_setbit64(&S.tmask[r], R.c[s] & 63);
            if (FILL) {
                S.tid[r] = (unsigned short)t;
                R.c[s] = (r << 6) | (R.c[s] & 63);
            }
        }
    }
    __syncwarp();
    return ntiles;
}

constexpr int HC_WARPS = 4;
constexpr int HC_CTAS_PER_SM = 6;

__global__ void __launch_bounds__(HC_WARPS * 32, HC_CTAS_PER_SM)
    k_count_h(int M, const int *__restrict__ arp, const int *__restrict__ acol, const int *__restrict__ brp,
              const int *__restrict__ bcol, RowInfo ri, Ctl *ctl) {
    extern __shared__ unsigned long long s_dyn[];
    const int lane = lane_id(), w = threadIdx.x >> 5;
    HSmem &S = reinterpret_cast<HSmem *>(s_dyn)[w];
    const int n = unless_failed(ctl, ctl->bin_count[BIN_H]);
    const int *rows = ri.bins + (size_t)BIN_H * M;
    HRows H(rows, arp, acol, blockIdx.x * HC_WARPS + w, n, gridDim.x * HC_WARPS);
    while (H.i >= 0) {
        const int i = H.i;
        const int t0 = ri.tmin[i], t1 = ri.tmax[i];
        HProducts<AR_RN, false> R;
        R.load(H.a_lo, H.a_hi, H.k, nullptr, brp, bcol, nullptr);
        H.next();
        const int nt = h_order<false>(R, t0, t1 - t0 + 1, S, [&] { H.range(); });
        H.column();
        int cnt = 0;
        for (int q = lane; q < nt; q += WARP) cnt += popc64(S.tmask[q]);
        cnt = warp_sum(cnt);
        if (lane == 0) {
            ri.cnnz[i] = cnt;
            if (nt < 0) set_err(&ctl->err, DERR_INTERNAL);
        }
        __syncwarp();
    }
}

constexpr int HF_WARPS = 4;
// 24 warps per SM at 80 registers; the fused multiply-add keeps every product's A value too, and the
// integer product spills at 80
template <int AR>
constexpr int hf_ctas() {
    return AR == AR_FMA ? 4 : AR == AR_IMUL ? 5 : 6;
}
static_assert(hf_ctas<AR_RN>() * (HF_WARPS * sizeof(HSmem) + 1024) <= 228 * 1024, "CTAs per SM");

// columns and values of every scattered row of the panel
template <int AR>
__global__ void __launch_bounds__(HF_WARPS * 32, hf_ctas<AR>())
    k_fill_h(int M, const int *__restrict__ arp, const int *__restrict__ acol, const double *__restrict__ aval,
             const int *__restrict__ brp, const int *__restrict__ bcol, const double *__restrict__ bval, RowInfo ri,
             RowOut out, Ctl *ctl) {
    extern __shared__ unsigned long long s_dyn[];
    const int lane = lane_id(), w = threadIdx.x >> 5;
    HSmem &S = reinterpret_cast<HSmem *>(s_dyn)[w];
    const int *rows = ri.bins + (size_t)BIN_H * M;
    int b0, b1;
    bin_slice(rows, unless_failed(ctl, ctl->bin_count[BIN_H]), out, M, b0, b1);
    HRows H(rows, arp, acol, b0 + blockIdx.x * HF_WARPS + w, b1, gridDim.x * HF_WARPS);
    while (H.i >= 0) {
        const int i = H.i;
        if (skip_row(out, i)) {
            H.next();
            H.range();
            H.column();
            continue;
        }
        const int t0 = ri.tmin[i], t1 = ri.tmax[i];
        const long long rowbase = out_base(out, i);
        const int limit = out_limit(out, i);
        HProducts<AR, true> R;
        R.load(H.a_lo, H.a_hi, H.k, aval, brp, bcol, bval);
        H.next();
        const int nt = h_order<true>(R, t0, t1 - t0 + 1, S, [&] { H.range(); });
        H.column();
        int nnz = 0;  // first slot of every tile
        for (int q0 = 0; q0 < nt; q0 += WARP) {
            const int q = q0 + lane;
            const int pc = q < nt ? popc64(S.tmask[q]) : 0;
            const int incl = warp_incl_scan(pc);
            if (q < nt) S.tbase[q] = (unsigned short)(nnz + incl - pc);
            nnz += __shfl_sync(FULL, incl, WARP - 1);
        }
        __syncwarp();
        const bool fits = nt >= 0 && nnz <= limit;
        if (lane == 0) {
            if (nt < 0 || (out.mode != OUT_SPEC && nnz != limit)) set_err(&ctl->err, DERR_INTERNAL);
            if (out.mode == OUT_SPEC) {
                out.cnnz[i] = nnz;
                out.flag[i] = fits ? ROW_VALUES : ROW_OVERFLOW;
                if (!fits) atomicAdd(&ctl->fallback, 1);
            }
        }
        if (!fits || (out.mode != OUT_SPEC && nnz != limit)) {
            __syncwarp();
            continue;
        }
        // columns: every lane its own tiles' (mostly one or two entries each)
        int *__restrict__ ocol = out.ccol + rowbase;
        for (int q = lane; q < nt; q += WARP) {
            unsigned long long m = S.tmask[q];
            int at = S.tbase[q];
            const int cb = (t0 + S.tid[q]) << 6;
            while (m) {
                ocol[at++] = cb + __ffsll((long long)m) - 1;
                m &= m - 1ull;
            }
        }
        // every product's slot takes its rank's place
#pragma unroll
        for (int s = 0; s < H_STEPS; s++) {
            if (s * WARP >= R.n) break;
            if (R.c[s] >= 0) {
                const int rk = R.c[s] >> 6;
                R.c[s] = S.tbase[rk] + rank64(S.tmask[rk], R.c[s] & 63);
            }
        }
        __syncwarp();
        double *acc = reinterpret_cast<double *>(S.tmask);
        if (nnz == R.n) {
#pragma unroll
            for (int s = 0; s < H_STEPS; s++) {
                if (s * WARP >= R.n) break;
                if (R.c[s] >= 0) acc[R.c[s]] = add_term<AR>(0.0, AR == AR_FMA ? R.av[s] : 0.0, R.p[s]);
            }
        } else {
            unsigned char *tag = reinterpret_cast<unsigned char *>(S.opre);
            for (int q = lane; q < nnz; q += WARP) acc[q] = 0.0;
            __syncwarp();
            // one step per iteration, the register arrays moved down by one after each: a loop
            // body instead of H_STEPS copies of it (cold instruction fetches were a third of the
            // kernel's time on a power-law graph's few thousand rows)
#pragma unroll 1
            for (int left = R.n; left > 0; left -= WARP) {
                // lanes that share a slot are found by stamps (hsmu_products.cuh) and add in lane order
                const int slot = R.c[0];
                const bool act = slot >= 0;
                const double a = AR == AR_FMA ? R.av[0] : 0.0;
                if (act) tag[slot] = (unsigned char)lane;
                __syncwarp();
                const int seen = act ? (int)tag[slot] : lane;
                const unsigned lm = __ballot_sync(FULL, seen != lane);
                int rank = 0, maxr = 0;
                if (lm) {
                    const unsigned cm = lm | __reduce_or_sync(FULL, seen != lane ? 1u << seen : 0u);
                    if ((cm >> lane) & 1u) rank = __popc(__match_any_sync(cm, slot) & lanemask_lt());
                    maxr = (int)__reduce_max_sync(FULL, (unsigned)rank);
                }
                for (int rr = 0; rr <= maxr; rr++) {
                    if (act && rank == rr) acc[slot] = add_term<AR>(acc[slot], a, R.p[0]);
                    __syncwarp();
                }
#pragma unroll
                for (int s = 0; s + 1 < H_STEPS; s++) {
                    R.c[s] = R.c[s + 1];
                    R.p[s] = R.p[s + 1];
                    if (AR == AR_FMA) R.av[s] = R.av[s + 1];
                }
            }
        }
        __syncwarp();
        for (int q = lane; q < nnz; q += WARP) out.cval[rowbase + q] = acc[q];
        __syncwarp();
    }
}

void launch_count_scattered(const DevCSR &A, const DevCSR &B, RowInfo ri, Ctl *ctl, int nsm, cudaStream_t st) {
    k_count_h<<<grid_for(nsm * HC_CTAS_PER_SM, A.M, HC_WARPS), HC_WARPS * 32, HC_WARPS * sizeof(HSmem), st>>>(A.M, A.rp, A.col, B.rp, B.col, ri,
                                                                                     ctl);
}

template <int AR>
static void fill_scattered(const DevCSR &A, const DevCSR &B, RowInfo ri, RowOut out, Ctl *ctl, int nsm,
                           cudaStream_t st) {
    k_fill_h<AR><<<grid_for(nsm * hf_ctas<AR>(), A.M, HF_WARPS), HF_WARPS * 32, HF_WARPS * sizeof(HSmem), st>>>(A.M, A.rp, A.col, A.val, B.rp,
                                                                                       B.col, B.val, ri, out, ctl);
}

void launch_fill_scattered(const DevCSR &A, const DevCSR &B, RowInfo ri, RowOut out, Ctl *ctl, int arith, int nsm,
                           cudaStream_t st) {
    if (arith == AR_IMUL) fill_scattered<AR_IMUL>(A, B, ri, out, ctl, nsm, st);
    else if (arith == AR_FMA) fill_scattered<AR_FMA>(A, B, ri, out, ctl, nsm, st);
    else fill_scattered<AR_RN>(A, B, ri, out, ctl, nsm, st);
}

int configure_scattered() {
    int e = (int)cudaFuncSetAttribute(k_count_h, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      HC_WARPS * (int)sizeof(HSmem));
    for (auto k : {k_fill_h<AR_RN>, k_fill_h<AR_FMA>, k_fill_h<AR_IMUL>})
        if (!e) e = (int)cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              HF_WARPS * (int)sizeof(HSmem));
    return e;
}

}  // namespace hsmu
