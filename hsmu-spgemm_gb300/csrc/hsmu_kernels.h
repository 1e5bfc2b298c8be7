// Host-side launch wrappers of the engine's kernels (one translation unit
// per stage; the orchestration in engine.cu only sees these declarations).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace hsmu {

struct Ctl;
struct Window;

struct DevCSR {
    int M, N;
    long long nnz;
    const int *rp;
    const int *col;
    const double *val;
};

struct DevTiles {
    const int *ptr;                  // [K+1]
    const int *col;                  // [T]
    const unsigned long long *mask;  // [T]
    const int *off;                  // [T]
};

// where the structure pass puts each row (see k_structure.cu)
enum OutMode : int { OUT_PLAIN = 0, OUT_SPEC = 1, OUT_REDO = 2 };
enum RowFlag : unsigned char { ROW_NONE = 0, ROW_VALUES = 1, ROW_COLUMNS = 2, ROW_OVERFLOW = 3 };
struct RowOut {
    int mode;
    const int *crp;         // PLAIN / REDO: final row pointers
    const long long *soff;  // SPEC: speculative slot offsets [M+1]
    int *ccol;              // destination columns
    double *cval;           // destination values
    int *cnnz;              // SPEC: exact nnz found per row
    unsigned char *flag;    // SPEC: written; REDO: rows flagged ROW_OVERFLOW are redone
    int lo, hi;             // only rows lo <= i < hi are written (a row panel; 0, M: all rows)
};

// per-row data of A produced by the bounds kernel
struct RowInfo {
    long long *prod;   // intermediate products of the row
    int *tmin;         // first C tile id (INT_MAX for an empty row)
    int *tmax;         // last C tile id (-1 for an empty row)
    int *bins;         // NBIN slabs of M row ids, each in ascending row order
    int *cnnz;         // exact nnz per row (count pass)
    signed char *cls;  // row class (RowBin) of every row, -1 for an empty row
    const unsigned char *rep;  // B rows that repeat the row before them (nullable; launch_row_repeat)
    const unsigned char *rep_a;  // the same of A (nullable): such a row's C row has the structure of the one before
    int store;         // 1: the tile store is in use -- the count pass sizes each large row's
                       // list, min(tile span, sum of its B rows' tile counts), and adds the
                       // sizes up in Ctl::store_tiles (the arena the next call wants)
};

// C tiles of the large-class rows, kept by the count pass (which builds them
// anyway) so that the structure pass streams each row's tile list instead of
// repeating the OR walk over B's tiles.  Each large row reserves min(tile span,
// sum of its B rows' tile counts) entries of the arena (tcol/tent, `cap`
// entries, owned by the handle) with one atomic; a row that finds the arena full keeps nothing (cnt[i] = -1) and
// the structure pass walks B for it as before.  Row i's list:
// tcol/tent[off[i] .. off[i] + cnt[i]), tile ids ascending.
//
// A tile's column mask and its slot word are written and read together, so
// they share one 16-byte entry: one 128-bit store in the count pass, one
// 128-bit load in the structure pass.
struct alignas(16) TileEnt {
    unsigned long long mask;    // column mask
    long long info;             // first slot | (window ordinal + 1) << 32 (hsmu_tilelist.cuh)
};

struct TileStore {
    long long *off;             // [M] written by the count pass
    int *cnt;                   // [M] tiles stored per row, -1: none
    int *nwin;                  // [M] numeric windows of the row (0 for rows without a list)
    int *wbase;                 // [M+1] index of the row's first window: exclusive scan of nwin in row
                                // order (nullable: the structure pass reserves them itself)
    int *tcol;                  // arena: tile ids
    TileEnt *tent;              // arena: column mask and slot word of each tile
    long long cap;              // arena entries
    int all_stored;             // host: every large row got a list (no OR-walk rows left)
};

// Look-back state of the single-pass scans (k_rows.cu): one per stream that scans, its words zeroed
// once (scan_state_bytes())
constexpr int LB_TILES = 4096;  // most tiles of a launch
constexpr int LB_STREAMS = 4;   // sums looked back over at once
struct ScanState {
    void *word;
    unsigned epoch;
    int polls;  // polls of an earlier tile's sum before a look-back gives up (0: the default limit)
};
struct LookBack {
    unsigned *ctr;             // tickets handed out, blocks done
    unsigned long long *word;  // [LB_STREAMS][LB_TILES]
    unsigned epoch;
    int polls;
};
size_t scan_state_bytes();
// the state for one launch that looks back
LookBack next_epoch(ScanState &s, cudaStream_t st);

// blocks of a grid-stride launch: `most`, or fewer when `per_block` items each are enough (a small
// call's launches otherwise spend their time on a thousand empty blocks)
inline int grid_for(int most, long long items, int per_block) {
    const long long need = (items + per_block - 1) / per_block;
    return need < 1 ? 1 : (need < most ? (int)need : most);
}

// k_tiles.cu
// gated: nothing is done when no row of A reads B's tiles (Ctl::bin_count, after the bounds pass)
void launch_tiles_count(const DevCSR &B, int *tcnt, int validate, Ctl *ctl, int grid, cudaStream_t st,
                        bool gated = false);
void launch_tiles_fill(const DevCSR &B, const int *tptr, int *tcol, unsigned long long *tmask, int *toff, Ctl *ctl,
                       int grid, cudaStream_t st, bool gated = false);
// rep[k]: row k of B has the columns of row k - 1 (B.M bytes); *chains (nullable) is raised by the
// number of chains that the rows form
void launch_row_repeat(const DevCSR &B, unsigned char *rep, int *chains, int grid, cudaStream_t st);
void launch_validate(const DevCSR &A, Ctl *ctl, int grid, cudaStream_t st);

// k_rows.cu
// counts_only: the call ends with the count pass (lines for its warps, none by products)
void launch_bounds(const DevCSR &A, const DevCSR &B, RowInfo ri, Ctl *ctl, int grid, ScanState &scan, cudaStream_t st,
                   bool counts_only = false);
// whether rows of many entries are taken in a launch of their own (hsmu_rowsums.cuh): it costs about
// 3 us where there are none (a 5-point Laplacian of 65,536 rows: 9 + 3 us) and takes 30 us off a
// power-law graph of 430,000 entries, so small or short-rowed matrices go without
inline bool long_rows_apart(const DevCSR &A) {
    return A.nnz >= (1 << 20) || (A.nnz >= (1 << 16) && A.nnz > 6ll * A.M);
}
// out[c] = products of rows c*PROD_CHUNK .. (c+1)*PROD_CHUNK-1 (ceil(M / PROD_CHUNK) entries)
constexpr int PROD_CHUNK = 64;
// crp[r0..r1] = rp[r0..r1] - rp[r0]
void launch_panel_ptr(const long long *rp, int r0, int r1, int *crp, int grid, cudaStream_t st);
void launch_chunk_prod(int M, const long long *prod, long long *out, int grid, cudaStream_t st);
// exclusive scan of int counts (n entries) into out[0..n]; total (int64) into *total64;
// sets DERR_OVERFLOW if the total exceeds INT32_MAX.
// in == out (an in-place scan) is allowed.
// gated: as launch_tiles_count (out and *total64 are then left alone)
void launch_scan(const int *in, int *out, int n, long long *total64, ScanState &scan, Ctl *ctl, cudaStream_t st,
                 bool gated = false);
// same with int64 output (no overflow limit)
void launch_scan64(const int *in, long long *out, int n, long long *total64, ScanState &scan, Ctl *ctl,
                   cudaStream_t st);
// the int scan without a state: three launches, tmp holds scan_tmp_ints(n) ints
size_t scan_tmp_ints(int n);
void launch_scan3(const int *in, int *out, int n, long long *total64, int *tmp, Ctl *ctl, cudaStream_t st);

// learned.cu
// long_list (nullable): scratch of M + 1 ints
void launch_features(const DevCSR &A, const DevCSR &B, float4 *feat, long long *prod_out, int nsm, cudaStream_t st,
                     int *long_list = nullptr);
// wide_prod (nullable): incremented by the products of every warp-class row predicted clearly
// above FUSE_CAP entries; large_no_slot: rows of the large class get no slot (the caller keeps
// their tile lists)
void launch_capacity(const float *params, const float4 *feat, const long long *prod, const signed char *cls, int M,
                     int N, float margin, int *cap, int nsm, cudaStream_t st, unsigned long long *wide_prod,
                     bool large_no_slot);
void launch_compact(int M, const long long *soff, const int *crp, const unsigned char *flag, const int *scol,
                    const double *sval, int *ccol, double *cval, int nsm, cudaStream_t st);

// k_symbolic.cu
void launch_count(const DevCSR &A, const DevCSR &B, const DevTiles &Bt, RowInfo ri, Ctl *ctl, int nsm,
                  cudaStream_t st);
// the same by class: rows that need no tiles (tiny, scattered), warp rows, the large class
// (ts: nullable; when given, the large rows' C tiles are stored while the arena lasts)
void launch_count_light(const DevCSR &A, const DevCSR &B, RowInfo ri, Ctl *ctl, int nsm, cudaStream_t st);
void launch_count_warp(const DevCSR &A, const DevTiles &Bt, RowInfo ri, Ctl *ctl, int nsm, cudaStream_t st);
// N: columns of B
void launch_count_large(const DevCSR &A, const DevTiles &Bt, int N, RowInfo ri, const TileStore *ts, Ctl *ctl, int nsm,
                        cudaStream_t st);
// learned path, large rows: exact count and tile list in its speculative pass;
// every listed row is flagged ROW_OVERFLOW (out.flag) so that the pass after the
// exact scan writes it at its place in C (k_symbolic.cu)
void launch_spec_large(const DevCSR &A, const DevTiles &Bt, int N, RowInfo ri, const TileStore &ts, RowOut out, Ctl *ctl,
                       int nsm, cudaStream_t st);

// k_scatter.cu: rows of the scattered class (exact count; columns and values)
void launch_count_scattered(const DevCSR &A, const DevCSR &B, RowInfo ri, Ctl *ctl, int nsm, cudaStream_t st);
void launch_fill_scattered(const DevCSR &A, const DevCSR &B, RowInfo ri, RowOut out, Ctl *ctl, int arith, int nsm,
                           cudaStream_t st);

// k_structure.cu
// writes C's columns and numeric windows; rows that fit one warp also get their values
// class_rows: rows per class (BIN_*) when known on the host; kernels of empty classes are skipped
// ts (nullable, PLAIN mode): large rows are built from their stored tile lists
void launch_structure(const DevCSR &A, const DevCSR &B, const DevTiles &Bt, RowInfo ri, RowOut out, Window *win,
                      long long win_cap, Ctl *ctl, int arith, int nsm, cudaStream_t st,
                      const int *class_rows = nullptr, const TileStore *ts = nullptr);
// the classes that need no tiles, alone (launch_structure launches them too unless class_rows says
// that there are none)
void launch_structure_light(const DevCSR &A, const DevCSR &B, RowInfo ri, RowOut out, Ctl *ctl, int arith, int nsm,
                            cudaStream_t st, const int *class_rows);

// k_numeric.cu
// flag (nullable): speculative-pass windows of rows flagged ROW_OVERFLOW are skipped;
// scol/soff (nullable): speculative slots holding the columns of speculative-pass
// windows, which the kernel copies to ccol
// per-window cursors into the B rows (k_win_cursors): off/item_off sized
// for win_cap windows + 1, cur for cap entries (Ctl::cur_bound)
struct WinCursors {
    long long *off;
    int *item_off;  // the cursor pass's work items per window, scanned
    int *cur;
    int *heavy;     // windows of rows with many A entries (win_cap entries)
    long long cap;
};
void launch_numeric(const DevCSR &A, const DevCSR &B, const DevTiles &Bt, const int *crp, int *ccol, double *cval,
                    const Window *win, long long win_cap, const unsigned char *flag, const int *scol,
                    const long long *soff, const WinCursors &wc, Ctl *ctl, int arith, int nsm, cudaStream_t st,
                    ScanState &scan, int wait_polls = 0, const TileStore *ts = nullptr);

int run_dmul_selftest(unsigned long long n, unsigned long long seed, unsigned long long *out, cudaStream_t st);
// FP64 lane operations per second of a full-grid chain probe
int run_fp64_rate(int iters, int nsm, double *lane_ops_per_s, cudaStream_t st);

// hsmu_status of the device error bits collected in Ctl::err (0 -> HSMU_OK)
int status_from_dev_err(int err);

// smem sizes are set once per device (cudaFuncSetAttribute)
int configure_kernels();

// k_transpose.cu: B = A^T (rows of B in ascending column order), scratch sized by the helpers
int launch_transpose(const DevCSR &A, int *trp, int *tcol, double *tval, int *scratch_i, double *scratch_d,
                     int *hist, ScanState &scan, long long *total64, Ctl *ctl, int nsm, cudaStream_t st);
size_t transpose_scratch_ints(long long nnz);
size_t transpose_scratch_doubles(long long nnz);
size_t transpose_hist_ints(long long nnz);

}  // namespace hsmu
