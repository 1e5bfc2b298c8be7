// The product loop shared by the fused row kernel (k_struct_ds) and the
// window kernel (k_numeric): accumulate a_ik * b_kj into a shared-memory
// accumulator for one C row (or one window of it), in the oracle's order.
//
// Order: for each C entry the products are added as 0.0 + p_1 + p_2 + ...
// in A(i,:)'s storage order, exactly like the host Gustavson oracle, so
// results are bit-identical to it in each arithmetic mode (AR_RN: every
// p = a*b rounded before the add, as the reference does; AR_FMA: each step
// one fused multiply-add).
//
// The A entries are taken 32 at a time (one per lane); seg(p) gives the B
// entry range [elo, ehi) that A entry p contributes to this accumulator.
//   * repeated rows (rep given): consecutive A entries whose B rows are
//     consecutive and hold the same columns -- the rows of one finite-element
//     node -- form chains of up to REP_MAX rows.  A lane takes one column of a
//     chain: one look-up and one accumulator round trip for all its rows'
//     products, added in row order.  The columns of successive chains are laid
//     end to end over the lanes, which leaves none idle: the FP64 pipe, which
//     binds these rows, takes as long for a step of 17 lanes as for one of 32.
//     Two chains that share a step share no slot when the younger one's last
//     column lies before the older one's first (stencil rows: always);
//     otherwise they add one after the other.  27-point stencil, 40^3 grid x 3
//     dofs: fused row kernel 5.68 -> 5.16 ms (FP64 pipe 78 % busy, no lane
//     idle); holding the sums in registers over repeated rows without laying
//     chains end to end left 16 % of the lanes idle and took 5.79 ms.
//   * segments that fill steps of 32 well (callers may turn this path off): the
//     segments one after another, 32 entries per step, the B loads of the next
//     LU steps issued before the current ones are used.  Entries of one B row
//     have distinct columns, so a step has no slot conflict and only a change
//     of segment needs a warp sync.  Scalar 27-point rows (33^3 grid, fused
//     multiply-add): 215 us on the flat path with its match per step, 169 us.
//   * otherwise: the flat sequence of (A entry, B entry) items, 32 per step.
//     The non-empty segments are packed into lanes; one OR-reduction per step
//     marks the segment starts inside it, so every lane gets its segment from
//     a popcount.  A step inside one segment has distinct slots; lanes of a
//     step spanning several segments that hit the same slot add in lane order
//     = A-entry order (found by __match_any_sync, or with TAG by stamping lane
//     ids into a byte per slot and matching only the lanes that collide).
#pragma once
#include "hsmu_block.cuh"
#include "hsmu_dmul.cuh"

namespace hsmu {

// Arithmetic of one accumulation step c <- c + a*b (hsmu_opts.arith):
//   AR_RN   (0) product rounded, then added: RN(c + RN(a*b));
//   AR_FMA  (1) fused, one rounding per product: RN(c + a*b) -- one FP64
//               pipe operation per product instead of two;
//   AR_IMUL (2) as AR_RN, with the product formed exactly on the integer pipe.
// term() is what can be computed before the accumulator slot is known;
// add_term() folds it into the accumulator.
enum Arith { AR_RN = 0, AR_FMA = 1, AR_IMUL = 2 };

template <int AR>
__device__ __forceinline__ double term(double a, double b) {
    if (AR == AR_FMA) return b;
    if (AR == AR_IMUL) return dmul_int(a, b);
    return __dmul_rn(a, b);
}

template <int AR>
__device__ __forceinline__ double add_term(double c, double a, double t) {
    if (AR == AR_FMA) return __fma_rn(a, t, c);
    return __dadd_rn(c, t);
}

// steps of 32 B entries in flight on the segment path
constexpr int LU = 3;
// groups of A entries take the segment path where one segment at a time keeps this share of
// the lanes busy (27-point rows: 84 %); below it the flat path wins
constexpr int WALK_LANES_PCT = 70;
// most rows of a chain (4: the wider step's registers spill, 5.16 -> 5.99 ms), and the columns its leaders must average: shorter chains laid end to
// end would often meet the same columns twice in a step
constexpr int REP_MAX = 3;
constexpr int CROSS_SEG_MIN = 36;

// SegFn:    void(int p, int k, int &elo, int &ehi)  -- called for valid lanes
// LookupFn: int(int j) -> slot in acc, or -1 if j is not in the accumulator
// PG: load the next group of 32 A entries before processing the current one
// (for rows with many A entries; costs registers in the short-row kernels)
// REP: rep[k] is nonzero when B row k holds the same columns as row k - 1
// (k_row_repeat); seg() must then give whole B rows.
// TAG: `tag` is a byte per accumulator slot (any contents), used to find the
// lanes of a step that share a slot; without it every multi-entry step runs
// a full-warp match.
// LONG: groups may take the segment path (else every group
// runs flat, where a step inside one segment needs no conflict test either).
template <int AR, bool NC = true, bool PG = false, bool TAG = false, bool LONG = true, bool REP = false,
          class SegFn,
          class LookupFn>
__device__ __forceinline__ void warp_accumulate(int a_lo, int a_hi, const int *__restrict__ acol,
                                                const double *__restrict__ aval, const int *__restrict__ brp,
                                                const int *__restrict__ bcol, const double *__restrict__ bval,
                                                SegFn seg, LookupFn lookup, double *acc, bool &bad,
                                                unsigned char *tag = nullptr, const unsigned char *rep = nullptr) {
    const int lane = lane_id();
    // A entries 32 at a time (PG: the next group's entries and segments are
    // loaded before the current group is processed)
    int n_elo = 0, n_ehi = 0;
    double n_a = 0.0;
    if (PG && a_lo + lane < a_hi) {
        n_a = ldx<NC>(aval + a_lo + lane);
        seg(a_lo + lane, ldx<NC>(acol + a_lo + lane), n_elo, n_ehi);
    }
    for (int pb = a_lo; pb < a_hi; pb += WARP) {
        int elo = 0, ehi = 0, k = -1;
        double a = 0.0;
        bool join = false;  // this entry's B row repeats the previous entry's
        static_assert(!(PG && REP), "repeated rows are found in the group being processed");
        if (PG) {
            elo = n_elo;
            ehi = n_ehi;
            a = n_a;
            n_elo = n_ehi = 0;
            n_a = 0.0;
            if (pb + WARP + lane < a_hi) {
                const int pn = pb + WARP + lane;
                n_a = ldx<NC>(aval + pn);
                seg(pn, ldx<NC>(acol + pn), n_elo, n_ehi);
            }
        } else if (pb + lane < a_hi) {
            a = ldx<NC>(aval + pb + lane);
            k = ldx<NC>(acol + pb + lane);
            seg(pb + lane, k, elo, ehi);
        }
        if (REP) {
            const int k_up = __shfl_up_sync(FULL, k, 1);
            join = lane > 0 && k >= 0 && k == k_up + 1 && rep[k];
        }
        const int len = ehi - elo;
        const int incl = warp_incl_scan(len);
        const int total = __shfl_sync(FULL, incl, WARP - 1);
        if (total == 0) continue;
        const unsigned ne = __ballot_sync(FULL, len > 0);
        const int nseg = __popc(ne);
        if (REP) {
            // ---- repeated rows: the chains of each leader's columns, 32 per step
            const unsigned jm = __ballot_sync(FULL, join);
            const int pos = lane - (31 - __clz(~jm & lanemask_le()));  // place in the run of repeated rows
            const unsigned behind = lane == 31 ? 0u : jm >> (lane + 1);
            const int grp = min(REP_MAX, __ffs(~behind));            // rows of the chain a leader starts
            unsigned todo = __ballot_sync(FULL, len > 0 && pos % REP_MAX == 0);
            const int nlead = __popc(todo);
            const int lead_len = ((todo >> lane) & 1u) ? len : 0;
            const int items = (int)__reduce_add_sync(FULL, (unsigned)lead_len);
            if (4 * nlead <= 3 * nseg && items >= CROSS_SEG_MIN * nlead) {
                int es = 0, ls = 0, g = 0, l0 = 0, off = 0;  // current chain rows: first entry, length, rows, lane
                auto next_seg = [&]() {
                    l0 = __ffs(todo) - 1;
                    todo &= todo - 1;
                    es = __shfl_sync(FULL, elo, l0);
                    ls = __shfl_sync(FULL, len, l0);
                    g = __shfl_sync(FULL, grp, l0);
                };
                // one step: nv valid lanes, the first rm of them of the older leader (rm = 32: one
                // leader); every lane's rows (gl), first lane (sl) and B entries (j, b)
                auto fetch = [&](int &j, double *b, int &gl, int &sl, int &rm, int &nv) {
                    nv = 0;
                    if (off >= ls) {
                        if (!todo) return;
                        next_seg();
                        off = 0;
                    }
                    int e = es + off + lane, l = ls;
                    gl = g;
                    sl = l0;
                    rm = WARP;
                    nv = min(WARP, ls - off);
                    off += nv;
                    if (nv < WARP && todo) {
                        rm = nv;
                        next_seg();
                        off = min(WARP - rm, ls);
                        nv = rm + off;
                        if (lane >= rm) {
                            e = es + lane - rm;
                            l = ls;
                            gl = g;
                            sl = l0;
                        }
                    }
                    j = 0;
                    if (lane < nv) j = ldx<NC>(bcol + e);
                    else gl = 0;
#pragma unroll
                    for (int m = 0; m < REP_MAX; m++) {
                        b[m] = 0.0;
                        if (m < gl) b[m] = ldx<NC>(bval + e + m * l);
                    }
                };
                int jc = 0, gc = 0, lc = 0, rc = WARP, nc;
                double bc[REP_MAX];
                fetch(jc, bc, gc, lc, rc, nc);
                while (nc > 0) {
                    int jn = 0, gn = 0, ln = 0, rn = WARP, nn;
                    double bn[REP_MAX];
                    fetch(jn, bn, gn, ln, rn, nn);
                    const int q = lookup(jc);
                    const bool act = lane < nc && q >= 0;
                    bad |= lane < nc && q < 0;
                    double av[REP_MAX], pr[REP_MAX];
                    const int gm = (int)__reduce_max_sync(FULL, (unsigned)gc);
#pragma unroll
                    for (int m = 0; m < REP_MAX; m++) {
                        if (m < gm) {
                            av[m] = __shfl_sync(FULL, a, lc + m);
                            pr[m] = term<AR>(av[m], bc[m]);
                        }
                    }
                    auto chain = [&]() {
                        double v = acc[q];
#pragma unroll
                        for (int m = 0; m < REP_MAX; m++)
                            if (m < gc) v = add_term<AR>(v, av[m], pr[m]);
                        acc[q] = v;
                    };
                    // two leaders: their columns ascend, so when the younger one's last column
                    // lies before the older one's first, no two lanes share a slot
                    if (rc == WARP || __shfl_sync(FULL, jc, nc - 1) < __shfl_sync(FULL, jc, 0)) {
                        if (act) chain();
                    } else {
                        if (act && lane < rc) chain();
                        __syncwarp();
                        if (act && lane >= rc) chain();
                    }
                    __syncwarp();
                    jc = jn;
                    gc = gn;
                    lc = ln;
                    rc = rn;
                    nc = nn;
#pragma unroll
                    for (int m = 0; m < REP_MAX; m++) bc[m] = bn[m];
                }
                continue;
            }
        }
        if (LONG && 32 * WALK_LANES_PCT * (int)__reduce_add_sync(FULL, (unsigned)(len + 31) >> 5) <= 100 * total) {
            // ---- one segment after another, 32 entries per step
            unsigned todo = ne;
            int es = 0, ls = 0, off = 0;  // current segment: first entry, length, entries taken
            double as = 0.0;
            // one step: nv valid lanes (0: no step left), sy: the first of its segment
            auto fetch = [&](int &j, double &b, double &av, int &nv, bool &sy) {
                nv = 0;
                sy = false;
                if (off >= ls) {
                    if (!todo) return;
                    const int sgi = __ffs(todo) - 1;
                    todo &= todo - 1;
                    es = __shfl_sync(FULL, elo, sgi);
                    ls = __shfl_sync(FULL, len, sgi);
                    as = __shfl_sync(FULL, a, sgi);
                    off = 0;
                    sy = true;
                }
                nv = min(WARP, ls - off);
                av = as;
                if (lane < nv) {
                    j = ldx<NC>(bcol + es + off + lane);
                    b = ldx<NC>(bval + es + off + lane);
                }
                off += nv;
            };
            int jc[LU], nc[LU];
            double bc[LU], ac[LU];
            bool sc[LU];
#pragma unroll
            for (int u = 0; u < LU; u++) {
                jc[u] = 0;
                bc[u] = ac[u] = 0.0;
                fetch(jc[u], bc[u], ac[u], nc[u], sc[u]);
            }
            while (nc[0] > 0) {
                int jn[LU], nn[LU];
                double bn[LU], an[LU];
                bool sn[LU];
#pragma unroll
                for (int u = 0; u < LU; u++) {
                    jn[u] = 0;
                    bn[u] = an[u] = 0.0;
                    fetch(jn[u], bn[u], an[u], nn[u], sn[u]);
                }
#pragma unroll
                for (int u = 0; u < LU; u++) {
                    if (nc[u] == 0) break;
                    if (sc[u]) __syncwarp();
                    // every lane multiplies and looks up (invalid lanes: b = 0, result unused)
                    const double pr = term<AR>(ac[u], bc[u]);
                    const int q = lookup(jc[u]);
                    const bool v = lane < nc[u];
                    bad |= v && q < 0;
                    if (v && q >= 0) acc[q] = add_term<AR>(acc[q], ac[u], pr);
                }
#pragma unroll
                for (int u = 0; u < LU; u++) {
                    jc[u] = jn[u];
                    bc[u] = bn[u];
                    ac[u] = an[u];
                    nc[u] = nn[u];
                    sc[u] = sn[u];
                }
            }
            __syncwarp();
            continue;
        }
        // ---- short segments: flat (A entry, B entry) order, 32 items per step.
        // The non-empty segments are packed into lanes 0..nseg-1 (flat start
        // st, B-entry shift d = elo - st, a).  Each step ORs the starts that
        // fall inside it into one 32-bit mask; the segment of a lane's item is
        // then the number of starts up to it (one popc), and a step with no
        // start after its first item holds one A entry (no slot conflicts).
        const int excl = incl - len;
        const int src = nth_set_bit(ne, min(lane, nseg - 1));
        const int st_src = __shfl_sync(FULL, excl, src);
        const int c_d = __shfl_sync(FULL, elo - excl, src);
        const double c_a = __shfl_sync(FULL, a, src);
        const int c_st = lane < nseg ? st_src : INT_MAX;
        const unsigned le = lanemask_le();
        auto starts = [&](int f) -> unsigned {
            const unsigned rel = (unsigned)(c_st - f);
            return __reduce_or_sync(FULL, rel < 32u ? 1u << rel : 0u);
        };
        unsigned sm = starts(0);
        int cb = 0;  // packed segments that start before the current step
        int j = 0;
        double b = 0.0, as;
        {
            const int sg = __popc(sm & le) - 1;
            const int e = lane + __shfl_sync(FULL, c_d, sg);
            as = __shfl_sync(FULL, c_a, sg);
            if (lane < total) {
                j = ldx<NC>(bcol + e);
                b = ldx<NC>(bval + e);
            }
        }
        for (int f = 0; f < total; f += WARP) {
            const bool gv = f + lane < total;
            const bool multi = (sm >> 1) != 0u;  // a segment starts after the step's first item
            cb += __popc(sm);
            int j_n = 0;
            double b_n = 0.0, as_n = 0.0;
            if (f + WARP < total) {
                sm = starts(f + WARP);
                const int sg_n = cb + __popc(sm & le) - 1;
                const int gn = f + WARP + lane;
                const int e = gn + __shfl_sync(FULL, c_d, sg_n);
                as_n = __shfl_sync(FULL, c_a, sg_n);
                if (gn < total) {
                    j_n = ldx<NC>(bcol + e);
                    b_n = ldx<NC>(bval + e);
                }
            }
            // every lane multiplies and looks up (invalid lanes: b = 0, result unused)
            const double pr = term<AR>(as, b);
            const int q = lookup(j);
            bad |= gv && q < 0;
            const bool act = gv && q >= 0;
            const int slot = act ? q : -1 - lane;
            if (!multi) {
                // one A entry in this step: all slots distinct
                if (act) acc[slot] = add_term<AR>(acc[slot], as, pr);
            } else if (TAG) {
                // each lane stamps its id on its slot; a lane that reads back another
                // id shares the slot with that lane.  Only such lanes are matched.
                if (act) tag[slot] = (unsigned char)lane;
                __syncwarp();
                const int seen = act ? (int)tag[slot] : lane;
                const bool lost = seen != lane;
                const unsigned lm = __ballot_sync(FULL, lost);
                if (lm == 0u) {
                    if (act) acc[slot] = add_term<AR>(acc[slot], as, pr);
                } else {
                    const unsigned cm = lm | __reduce_or_sync(FULL, lost ? 1u << seen : 0u);
                    const bool inc = (cm >> lane) & 1u;
                    int rank = 0;
                    if (inc) rank = __popc(__match_any_sync(cm, slot) & lanemask_lt());
                    const int maxr = (int)__reduce_max_sync(FULL, (unsigned)rank);
                    // round 0: the lanes that share no slot together with the first lane
                    // of each shared slot (all their slots are distinct), then one round
                    // per further lane of a shared slot
                    if (act && rank == 0) acc[slot] = add_term<AR>(acc[slot], as, pr);
                    __syncwarp();
                    for (int rr = 1; rr <= maxr; rr++) {
                        if (inc && rank == rr) acc[slot] = add_term<AR>(acc[slot], as, pr);
                        __syncwarp();
                    }
                }
            } else {
                const unsigned grp = __match_any_sync(FULL, slot);
                const int rank = __popc(grp & lanemask_lt());
                const int maxr = (int)__reduce_max_sync(FULL, act ? (unsigned)rank : 0u);
                for (int rr = 0; rr < maxr; rr++) {
                    if (act && rank == rr) acc[slot] = add_term<AR>(acc[slot], as, pr);
                    __syncwarp();
                }
                if (act && rank == maxr) acc[slot] = add_term<AR>(acc[slot], as, pr);
            }
            __syncwarp();
            j = j_n;
            b = b_n;
            as = as_n;
        }
    }
}

}  // namespace hsmu
