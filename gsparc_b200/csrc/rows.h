// rows.h -- the planning kernels of a group (rows.cu): Y's run and column
// tables, X's rows, the row classes and the unit lists.
#pragma once

#include "kernels.cuh"
#include "scan.cuh"

namespace gs {

// Per-job constants of the planning kernels.
struct BPrep {
    int x_ncbits;
    int y_nfbits;
    uint64_t light_max;  // rows with more products go to the windowed accumulator
    uint64_t col_word0;  // first word of the job's Y free indices in the presence bits
    uint64_t con_word0;  // first word of the job's contract keys in the run lookup table
};

// Device counters of a group.
enum {
    kCntCols = 0,     // distinct Y free indices
    kCntRuns = 1,     // runs of Y
    kCntRows = 2,
    kCntHeavy = 3,
    kCntLight = 4,    // light rows
    kCntUnits = 5,    // light units
    kCntStream = 7,
    kCntLightProd = 8,  // products of the light rows
    kCntRange = 9,    // 9..11 shard row range and products
    kCntBmAll = 12,   // words of every kept bitmap
    kCntBmDense = 13, // words of the dense rows' kept bitmaps
    kCntNarrow = 14,     // narrow rows among the heavy ones
    kCntNarrowCols = 15, // most columns of a job with narrow rows
    kCntProducts = 16,
    kCntErr = 17,        // error bits of the planning kernels and the radix sort (low word)
    kCntLightRuns = 18,  // runs of the light rows
    kCntLong = 19,       // light rows of more than kOrderScan runs
    kCnts = 20
};

constexpr uint8_t kRowNone = 0, kRowLight = 1, kRowStream = 2, kRowHeavy = 3, kRowNarrow = 4;  // narrow: heavy, over few columns

// Sorted Y keys -> run table (run_key, run_start with the closing entry, count
// in cnts), ydup per job; marks every entry's free index in the presence bits
// (bits null: writes the prefixed free index to yfk instead).  With ctab (zero
// at entry), also the run lookup table: for every 32 contract keys of a job
// the keys that have a run (word 0) and the first of these runs (word 1).
void launch_y_runs(const uint64_t *ykeys, uint64_t ny, int kby, const BPrep *jobs, uint64_t *run_key,
                   uint32_t *run_start, uint64_t *cnts, unsigned int *ydup, uint32_t *bits, uint64_t *yfk,
                   uint2 *ctab, const ScanState &st, cudaStream_t s);
// Presence bits -> distinct free indices of every job (cols, ascending) and
// the number of distinct ones before every word (wpre).
void launch_col_table(const uint32_t *bits, uint64_t nwords, const BPrep *jobs, int g, uint32_t *wpre, uint64_t *cols,
                      uint64_t *cnts, const ScanState &st, cudaStream_t s);
// Column rank of every Y entry inside its job, and the jobs' column ranges.
void launch_y_ranks(const uint64_t *ykeys, uint64_t ny, int kby, const BPrep *jobs, int g, const uint32_t *bits,
                    const uint32_t *wpre, const uint64_t *cnts, uint32_t *rank, BatchJob *acc,
                    const unsigned int *ydup, const unsigned int *err, cudaStream_t s);

constexpr uint32_t kOrderScan = 64;

struct RowArrays {
    uint64_t *xprefix;   // [nx + 1] matched products before every X nonzero
    uint32_t *mpre;      // [nx + 1] matched X nonzeros before every one
    uint32_t *mrun;      // [matched] the matched X nonzeros
    uint32_t *mrow;      // [matched] their rows
    uint32_t *row_start; // [nrows + 1]
    uint32_t *row_k0;    // [nrows + 1] first matched X nonzero (index into mrun)
    uint64_t *row_xf;    // [nrows]
    uint16_t *row_job;   // [nrows]
    uint64_t *row_prod;  // [nrows]
    uint8_t *row_class;  // [nrows]
    uint32_t *row_nnz;   // [nrows] stream rows: their products; 0 otherwise
    uint32_t *row_xi;    // [nrows] stream rows: their matched X nonzero; narrow and light rows: their number
    uint32_t *H, *SR, *L;  // heavy, stream and light rows, in row order
    uint64_t *sprefix;   // [stream + 1] products before every stream row
    uint64_t *lpre;      // [light + 1] products of the light rows before each one
    uint32_t *lk0;       // [light + 1] runs (matched X nonzeros) of the light rows before each one
    uint32_t *ustart;    // [light units + 1] first light row (index into L) of every unit
    uint32_t *lrun;      // [light runs] their X nonzeros, light row after light row
    uint32_t *lrow;      // [light runs] their light rows (indices into L)
    uint64_t *loff;      // [light runs] products of the light rows' runs before each one
    // X sorted by its free bits alone (null: by all bits): [nx / kOrderScan + 1]
    // the light rows (indices into L) of more than kOrderScan runs, in any order
    uint32_t *longs;
    uint32_t *row_rb, *row_mx;  // heavy rows: all ones and 0 (null: not wanted)
};
// Match of every X nonzero -> prefix sums, matched list and rows.
void launch_x_rows(const uint64_t *xkeys, uint64_t nx, int kbx, const BPrep *jobs, const uint32_t *cnt,
                   const uint8_t *row_flag, const RowArrays &r, uint64_t *cnts, const ScanState &st, cudaStream_t s);
// A relabeled job (wide.cu) whose output keys fit 64 bits: rank -> original free
// part of X and Y, original Y free bits.  xf null: not one.
struct WideTab {
    const uint64_t *xf, *yf;
    int nfbits_y, pad;
};
// Maps row_xf, cols and the Y free bits of those jobs (n: the larger of nx, ny).
void launch_wide_tables(const WideTab *tab, int g, uint64_t n, const uint16_t *row_job, uint64_t *row_xf,
                        uint64_t *cols, BatchJob *acc, const uint64_t *cnts, const unsigned int *err,
                        cudaStream_t s);
// y_f of every Y entry (all jobs' Y free bits fit 32; after launch_wide_tables).
void launch_y_cols32(const uint64_t *ykeys, uint64_t ny, int kby, const BatchJob *acc, const uint64_t *cols,
                     const uint32_t *rank, uint32_t *out, const unsigned int *err, cudaStream_t s);
// Row classes, their lists and product prefixes (rows outside `range` get no class).
void launch_row_classes(uint64_t nx, const BPrep *jobs, const BatchJob *acc, const uint64_t *range,
                        const RowArrays &r, uint64_t *cnts, const ScanState &st, cudaStream_t s);
// Light units: consecutive light rows of fewer than bin + light_max products.
void launch_light_units(uint64_t nx, uint64_t bin, const RowArrays &r, uint64_t *cnts, const ScanState &st,
                        cudaStream_t s);
// The light rows' runs (lrun, lrow, loff; with `longs`, those of rows of up to
// kOrderScan runs in the order of their contract keys) and, with row_rb and
// row_mx, the rank span of every heavy row.
void launch_matched_runs(uint64_t nx, const uint32_t *pos, const uint32_t *cnt, const uint32_t *yrank,
                         const RowArrays &r, const uint64_t *cnts, const unsigned int *err, cudaStream_t s);
// The runs (lrun, loff) of the rows in `longs` in the order of their contract keys.
void launch_light_order(uint64_t nx, const uint32_t *pos, const uint32_t *cnt, const RowArrays &r,
                        const uint64_t *cnts, const unsigned int *err, int sm_count, cudaStream_t s);
// Kept bitmaps: of every heavy row the words with all / only dense
// rows kept (w_*, by row), their word offsets (off_*, by row) and totals.
void launch_heavy_bitmaps(uint64_t nx, const RowArrays &r, uint32_t *w_all, uint32_t *w_dense,
                          uint64_t *off_all, uint64_t *off_dense, uint64_t *cnts, const ScanState &st, cudaStream_t s);

// row_off[r] = outputs before row r (nrows + 1 entries).
void launch_row_offsets(const uint32_t *row_nnz, uint64_t nrows, uint64_t *row_off, const ScanState &st,
                        cudaStream_t s);
// unit_off[0..n] and part_off[0..n) of a heavy list (narrow.cu), units of about
// `slice` products.
void launch_narrow_units(const uint32_t *list, uint32_t n, const uint8_t *row_class, const uint64_t *row_prod,
                         uint64_t slice, uint32_t *unit_off, uint32_t *part_off, const ScanState &st, cudaStream_t s);

}  // namespace gs
