// rows.cu -- planning kernels of a group of contractions: from the sorted
// operands to Y's run and column tables, X's rows, the row classes and the
// unit lists the accumulation kernels take.
//
// Every step is one kernel: the per-item values, their prefix sums (scan.cuh)
// and the lists that follow are made in one pass.  As separate flag, scan and
// select kernels the same steps took 56 launches for a contraction of 2,000
// nonzeros (now 19; stage events 0.53 -> 0.35 ms) and 74 for one of 2e7 (now
// 31).  Small inputs are bound by the chain of dependent loads of one tile
// (5 to 12 us a kernel), large ones by memory.
//
// Columns: the rank of a Y free index among its job's distinct ones comes from
// a presence bitmap over the job's free index space and a prefix of its words
// (mark, scan, look up) where the space is small against Y or absolutely; the
// caller sorts the free indices where it is not.
#include "rows.h"

#include "blockops.cuh"
#include "runtab.h"

namespace gs {

namespace {
using namespace dev;

constexpr int kThreads = 256;

inline int grid_for(uint64_t n) {
    uint64_t g = (n + kThreads - 1) / kThreads;
    if (g < 1) g = 1;
    if (g > 148ull * 32) g = 148ull * 32;
    return (int)g;
}

__device__ __forceinline__ uint64_t shr(uint64_t v, int s) { return s >= 64 ? 0ull : (v >> s); }
__device__ __forceinline__ uint64_t low_mask(int b) { return b >= 64 ? ~0ull : ((1ull << b) - 1); }

// A thread's 8 consecutive items move as 16-byte words where all are there
// (arrays are 256-byte aligned, so items 8 t of 4 and 8 bytes are aligned).
__device__ __forceinline__ void load8(const uint32_t *p, uint32_t (&v)[kScanItems]) {
    const uint4 a = *reinterpret_cast<const uint4 *>(p), b = *reinterpret_cast<const uint4 *>(p + 4);
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
}

__device__ __forceinline__ void load8(const uint64_t *p, uint64_t (&v)[kScanItems]) {
#pragma unroll
    for (int q = 0; q < kScanItems; q += 2) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2 *>(p + q);
        v[q] = a.x;
        v[q + 1] = a.y;
    }
}

// Y: runs of (job, contract key).  A job whose Y repeats a coordinate gets
// ydup[job] set: its runs may hold a free index twice, so none of its rows is
// streamed.
__global__ void __launch_bounds__(kScanThreads)
    k_y_runs(const uint64_t *__restrict__ ykeys, uint64_t ny, int kby, const BPrep *__restrict__ jobs,
             uint64_t *__restrict__ run_key, uint32_t *__restrict__ run_start, uint64_t *__restrict__ cnts,
             unsigned int *__restrict__ ydup, uint32_t *__restrict__ bits, uint64_t *__restrict__ yfk,
             uint2 *__restrict__ ctab, ScanState st) {
    __shared__ ScanShared<1> sh;
    const uint32_t tile = next_tile(st, sh);
    const uint64_t i0 = (uint64_t)tile * kScanTile + (uint64_t)threadIdx.x * kScanItems;
    const uint64_t km = low_mask(kby);
    uint64_t rk[kScanItems];
    uint32_t flags = 0, first = 0;  // bit q: a run starts there; it is the first of its table word
    uint64_t pk = i0 > 0 && i0 < ny ? ykeys[i0 - 1] : 0;
    uint64_t pj = ~0ull, prk = 0;
    if (i0 > 0 && i0 < ny) {
        pj = shr(pk, kby);
        prk = shr(pk & km, jobs[pj].y_nfbits);
    }
    uint64_t last_word = ~0ull;
    uint32_t word = 0;
    uint64_t kk[kScanItems];
    const bool whole = i0 + kScanItems <= ny;
    if (whole) load8(ykeys + i0, kk);
#pragma unroll
    for (int q = 0; q < kScanItems; ++q) {
        const uint64_t i = i0 + q;
        rk[q] = 0;
        if (i < ny) {
            const uint64_t key = whole ? kk[q] : ykeys[i];
            const uint64_t j = shr(key, kby);
            const BPrep b = jobs[j];
            const uint64_t loc = key & km;
            rk[q] = shr(loc, b.y_nfbits);
            if (j != pj || rk[q] != prk) {
                flags |= 1u << q;
                if (j != pj || (rk[q] >> 5) != (prk >> 5)) first |= 1u << q;
            }
            if (i > 0 && pk == key) atomicOr(&ydup[j], 1u);
            pk = key;
            pj = j;
            prk = rk[q];
            rk[q] |= kby >= 64 ? 0ull : j << kby;
            const uint64_t f = loc & low_mask(b.y_nfbits);
            if (bits) {
                const uint64_t w = b.col_word0 + (f >> 5);
                if (w != last_word) {
                    // most indices are marked already: look before the atomic
                    if (word && (word & ~__ldcg(bits + last_word))) atomicOr(&bits[last_word], word);
                    last_word = w;
                    word = 0;
                }
                word |= 1u << (f & 31);
            } else {
                yfk[i] = (kby >= 64 ? 0ull : j << kby) | f;
            }
        }
    }
    if (bits && word && (word & ~__ldcg(bits + last_word))) atomicOr(&bits[last_word], word);
    uint64_t x[1] = {(uint64_t)__popc(flags)};
    if (!tile_scan<1>(st, sh, tile, x)) return;
#pragma unroll
    for (int q = 0; q < kScanItems; ++q)
        if (flags >> q & 1u) {
            run_key[x[0]] = rk[q];
            run_start[x[0]] = (uint32_t)(i0 + q);
            if (ctab) {
                const BPrep b = jobs[shr(rk[q], kby)];
                const uint64_t c = rk[q] & km;
                if (run_in_table(c, b.x_ncbits)) {
                    uint2 *t = ctab + b.con_word0 + (c >> 5);
                    atomicOr(&t->x, 1u << (c & 31));
                    if (first >> q & 1u) t->y = (uint32_t)x[0];
                }
            }
            ++x[0];
        }
    if ((uint64_t)(tile + 1) * kScanTile >= ny && threadIdx.x == 0) {
        cnts[kCntRuns] = sh.through[0];
        run_start[sh.through[0]] = (uint32_t)ny;
    }
}

__device__ __forceinline__ int job_of_word(const BPrep *jobs, int g, uint64_t w) {
    int lo = 0, hi = g;  // last job with col_word0 <= w
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (jobs[mid].col_word0 <= w)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

__global__ void __launch_bounds__(kScanThreads)
    k_col_table(const uint32_t *__restrict__ bits, uint64_t nwords, const BPrep *__restrict__ jobs, int g,
                uint32_t *__restrict__ wpre, uint64_t *__restrict__ cols, uint64_t *__restrict__ cnts, ScanState st) {
    __shared__ ScanShared<1> sh;
    const uint32_t tile = next_tile(st, sh);
    const uint64_t w0 = (uint64_t)tile * kScanTile + (uint64_t)threadIdx.x * kScanItems;
    uint32_t b[kScanItems];
    uint32_t n = 0;
#pragma unroll
    for (int q = 0; q < kScanItems; ++q) {
        b[q] = w0 + q < nwords ? bits[w0 + q] : 0u;
        n += __popc(b[q]);
    }
    uint64_t x[1] = {n};
    if (!tile_scan<1>(st, sh, tile, x)) return;
    uint32_t c = (uint32_t)x[0];
    if (n) {
        int j = job_of_word(jobs, g, w0);
        for (int q = 0; q < kScanItems; ++q) {
            if (w0 + q >= nwords) break;
            while (j + 1 < g && jobs[j + 1].col_word0 <= w0 + q) ++j;
            wpre[w0 + q] = c;
            const uint64_t f0 = (w0 + q - jobs[j].col_word0) << 5;
            for (uint32_t v = b[q]; v; v &= v - 1) cols[c++] = f0 + (uint32_t)(__ffs(v) - 1);
        }
    } else {
#pragma unroll
        for (int q = 0; q < kScanItems; ++q)
            if (w0 + q < nwords) wpre[w0 + q] = c;
    }
    if ((uint64_t)(tile + 1) * kScanTile >= nwords && threadIdx.x == 0) cnts[kCntCols] = sh.through[0];
}

__global__ void k_y_ranks(const uint64_t *__restrict__ ykeys, uint64_t ny, int kby, const BPrep *__restrict__ jobs,
                          int g, const uint32_t *__restrict__ bits, const uint32_t *__restrict__ wpre,
                          const uint64_t *__restrict__ cnts, uint32_t *__restrict__ rank, BatchJob *__restrict__ acc,
                          const unsigned int *__restrict__ ydup, const unsigned int *__restrict__ err) {
    if (*err & kScanErr) return;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t t0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t km = low_mask(kby);
    for (uint64_t i = t0; i < ny; i += stride) {
        const uint64_t key = ykeys[i];
        const BPrep b = jobs[shr(key, kby)];
        const uint64_t f = key & km & low_mask(b.y_nfbits);
        const uint64_t w = b.col_word0 + (f >> 5);
        rank[i] = wpre[w] - wpre[b.col_word0] + __popc(bits[w] & ((1u << (f & 31)) - 1u));
    }
    for (uint64_t j = t0; j < (uint64_t)g; j += stride) {
        BatchJob b;
        b.y_nfbits = jobs[j].y_nfbits;
        b.ydup = ydup[j];
        b.wide = 0;
        b.cols_off = wpre[jobs[j].col_word0];
        b.ncols = (uint32_t)((j + 1 < (uint64_t)g ? wpre[jobs[j + 1].col_word0] : cnts[kCntCols]) - b.cols_off);
        acc[j] = b;
    }
}

__global__ void __launch_bounds__(kScanThreads)
    k_x_rows(const uint64_t *__restrict__ xkeys, uint64_t nx, int kbx, const BPrep *__restrict__ jobs,
             const uint32_t *__restrict__ cnt, const uint8_t *__restrict__ row_flag, RowArrays r,
             uint64_t *__restrict__ cnts, ScanState st) {
    __shared__ ScanShared<2> sh;
    const uint32_t tile = next_tile(st, sh);
    const uint64_t i0 = (uint64_t)tile * kScanTile + (uint64_t)threadIdx.x * kScanItems;
    uint32_t c[kScanItems];
    uint32_t flags = 0;
    uint64_t x[2] = {0, 0};  // products; matched nonzeros and (above 32 bits) rows
    const bool whole = i0 + kScanItems <= nx;
    uint64_t fl = 0;  // 8 flag bytes
    if (whole) {
        load8(cnt + i0, c);
        fl = *reinterpret_cast<const uint64_t *>(row_flag + i0);
    }
#pragma unroll
    for (int q = 0; q < kScanItems; ++q) {
        const uint64_t i = i0 + q;
        if (!whole) c[q] = i < nx ? cnt[i] : 0u;
        if (whole ? (fl >> (8 * q) & 0xffu) != 0 : i < nx && row_flag[i]) flags |= 1u << q;
        x[0] += c[q];
        x[1] += (c[q] != 0) + ((uint64_t)(flags >> q & 1u) << 32);
    }
    if (!tile_scan<2>(st, sh, tile, x)) return;
    uint32_t m = (uint32_t)x[1], row = (uint32_t)(x[1] >> 32);  // rows that start before this nonzero
    uint64_t p = x[0];
    const uint64_t km = low_mask(kbx);
    if (whole) {
        uint64_t pp[kScanItems];
        uint32_t mm[kScanItems];
#pragma unroll
        for (int q = 0; q < kScanItems; ++q) {
            pp[q] = q ? pp[q - 1] + c[q - 1] : p;
            mm[q] = q ? mm[q - 1] + (c[q - 1] != 0) : m;
        }
#pragma unroll
        for (int q = 0; q < kScanItems; q += 2)
            *reinterpret_cast<ulonglong2 *>(r.xprefix + i0 + q) = make_ulonglong2(pp[q], pp[q + 1]);
#pragma unroll
        for (int q = 0; q < kScanItems; q += 4)
            *reinterpret_cast<uint4 *>(r.mpre + i0 + q) = make_uint4(mm[q], mm[q + 1], mm[q + 2], mm[q + 3]);
    }
#pragma unroll
    for (int q = 0; q < kScanItems; ++q) {
        const uint64_t i = i0 + q;
        if (i >= nx) break;
        if (flags >> q & 1u) {
            const uint64_t key = xkeys[i];
            const uint64_t j = shr(key, kbx);
            r.row_start[row] = (uint32_t)i;
            r.row_k0[row] = m;
            r.row_xf[row] = shr(key & km, jobs[j].x_ncbits);
            r.row_job[row] = (uint16_t)j;
            ++row;
        }
        if (!whole) {
            r.xprefix[i] = p;
            r.mpre[i] = m;
        }
        if (c[q]) {
            r.mrun[m] = (uint32_t)i;
            r.mrow[m] = row - 1;
            ++m;
            p += c[q];
        }
    }
    if ((uint64_t)(tile + 1) * kScanTile >= nx && threadIdx.x == 0) {
        const uint32_t nm = (uint32_t)sh.through[1], nr = (uint32_t)(sh.through[1] >> 32);
        r.xprefix[nx] = sh.through[0];
        r.mpre[nx] = nm;
        r.row_start[nr] = (uint32_t)nx;
        r.row_k0[nr] = nm;
        cnts[kCntRows] = nr;
        cnts[kCntProducts] = sh.through[0];
    }
}

// Relabeled jobs whose output keys fit 64 bits: the tables that output keys are
// made from (row_xf, cols, the job's Y free bits) get the original values, so
// every kernel writes final keys.  As a pass over the finished output the same
// map took 199 us for 6.2e7 outputs of 4e5 x 2.5e5 nonzeros.
__global__ void k_wide_tables(const WideTab *__restrict__ tab, int g, const uint16_t *__restrict__ row_job,
                              uint64_t *__restrict__ row_xf, uint64_t *__restrict__ cols,
                              BatchJob *__restrict__ acc, const uint64_t *__restrict__ cnts,
                              const unsigned int *__restrict__ err) {
    if (*err & kScanErr) return;
    const uint64_t nr = cnts[kCntRows], nc = cnts[kCntCols];
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t t0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (uint64_t r = t0; r < nr; r += stride) {
        const WideTab t = tab[row_job[r]];
        if (t.xf) row_xf[r] = t.xf[row_xf[r]];
    }
    for (uint64_t c = t0; c < nc; c += stride) {
        int lo = 0, hi = g;  // last job whose columns start at or before c
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (acc[mid].cols_off <= c)
                lo = mid;
            else
                hi = mid;
        }
        const WideTab t = tab[lo];
        if (t.xf) cols[c] = t.yf[cols[c]];
    }
    for (uint64_t j = t0; j < (uint64_t)g; j += stride)
        if (tab[j].xf) {
            acc[j].y_nfbits = tab[j].nfbits_y;
            acc[j].wide = 1;
        }
}

// y_f of every Y entry in 32 bits (all jobs' Y free bits fit).
__global__ void k_y_cols32(const uint64_t *__restrict__ ykeys, uint64_t ny, int kby, const BatchJob *__restrict__ acc,
                           const uint64_t *__restrict__ cols, const uint32_t *__restrict__ rank,
                           uint32_t *__restrict__ out, const unsigned int *__restrict__ err) {
    if (*err & kScanErr) return;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < ny; i += stride)
        out[i] = (uint32_t)cols[acc[shr(ykeys[i], kby)].cols_off + rank[i]];
}

// Row classes: single-run rows of jobs without repeated Y coordinates stream
// (their output count is their product count), other rows with more than the
// job's light limit of products are heavy (narrow where the job has few
// columns and the row many products for them), the rest with products are light.
__global__ void __launch_bounds__(kScanThreads)
    k_row_classes(const BPrep *__restrict__ jobs, const BatchJob *__restrict__ acc,
                  const uint64_t *__restrict__ range, RowArrays r, uint64_t *__restrict__ cnts, ScanState st) {
    __shared__ ScanShared<5> sh;
    if (ld_acquire(st.err) & kScanErr) return;
    const uint64_t nr = cnts[kCntRows];
    const uint32_t tile = next_tile(st, sh);
    if ((uint64_t)tile * kScanTile >= nr) return;
    const uint64_t r0 = range ? range[0] : 0, r1 = range ? range[1] : nr;
    const uint64_t i0 = (uint64_t)tile * kScanTile + (uint64_t)threadIdx.x * kScanItems;
    uint8_t cl[kScanItems];
    uint64_t pr[kScanItems];
    uint32_t rn[kScanItems];
    // heavy and (above 32 bits) stream rows; light and narrow rows; light, stream products; light runs
    uint64_t x[5] = {0, 0, 0, 0, 0};
#pragma unroll
    for (int q = 0; q < kScanItems; ++q) {
        const uint64_t i = i0 + q;
        cl[q] = kRowNone;
        pr[q] = 0;
        rn[q] = 0;
        if (i < nr) {
            pr[q] = r.xprefix[r.row_start[i + 1]] - r.xprefix[r.row_start[i]];
            const uint32_t k0 = r.row_k0[i], runs = r.row_k0[i + 1] - k0;
            rn[q] = runs;
            if (i >= r0 && i < r1 && runs) {
                const uint16_t j = r.row_job[i];
                if (runs == 1 && !acc[j].ydup) {
                    cl[q] = kRowStream;
                    r.row_xi[i] = r.mrun[k0];
                } else {
                    cl[q] = pr[q] > jobs[j].light_max ? kRowHeavy : kRowLight;
                    const uint32_t nc = acc[j].ncols;
                    if (cl[q] == kRowHeavy && nc <= (uint32_t)kNarrowCols && pr[q] >= kNarrowProducts * nc) {
                        cl[q] = kRowNarrow;
                        if (cnts[kCntNarrowCols] < nc)
                            atomicMax((unsigned long long *)&cnts[kCntNarrowCols], (unsigned long long)nc);
                    }
                }
            }
            r.row_prod[i] = pr[q];
            r.row_class[i] = cl[q];
            if (cl[q] == kRowHeavy && r.row_rb) {
                r.row_rb[i] = 0xffffffffu;
                r.row_mx[i] = 0u;
            }
            r.row_nnz[i] = cl[q] == kRowStream ? (uint32_t)pr[q] : 0u;
            x[0] += (cl[q] >= kRowHeavy) + ((uint64_t)(cl[q] == kRowStream) << 32);
            x[1] += (cl[q] == kRowLight) + ((uint64_t)(cl[q] == kRowNarrow) << 32);
            x[2] += cl[q] == kRowLight ? pr[q] : 0;
            x[3] += cl[q] == kRowStream ? pr[q] : 0;
            x[4] += cl[q] == kRowLight ? rn[q] : 0;
        }
    }
    if (!tile_scan<5>(st, sh, tile, x)) return;
#pragma unroll
    for (int q = 0; q < kScanItems; ++q) {
        const uint32_t row = (uint32_t)(i0 + q);
        if (cl[q] >= kRowHeavy) {
            r.H[(uint32_t)x[0]] = row;
            x[0] += 1;
            if (cl[q] == kRowNarrow) {
                r.row_xi[row] = (uint32_t)(x[1] >> 32);
                x[1] += 1ull << 32;
            }
        } else if (cl[q] == kRowStream) {
            r.SR[x[0] >> 32] = row;
            r.sprefix[x[0] >> 32] = x[3];
            x[0] += 1ull << 32;
            x[3] += pr[q];
        } else if (cl[q] == kRowLight) {
            const uint32_t l = (uint32_t)x[1];
            r.L[l] = row;
            r.row_xi[row] = l;
            r.lpre[l] = x[2];
            r.lk0[l] = (uint32_t)x[4];
            if (r.longs && rn[q] > kOrderScan)
                r.longs[atomicAdd((unsigned long long *)&cnts[kCntLong], 1ull)] = l;
            x[1] += 1;
            x[2] += pr[q];
            x[4] += rn[q];
        }
    }
    if ((uint64_t)(tile + 1) * kScanTile >= nr && threadIdx.x == 0) {
        cnts[kCntHeavy] = (uint32_t)sh.through[0];
        cnts[kCntStream] = sh.through[0] >> 32;
        cnts[kCntLight] = (uint32_t)sh.through[1];
        cnts[kCntNarrow] = sh.through[1] >> 32;
        cnts[kCntLightProd] = sh.through[2];
        cnts[kCntLightRuns] = (uint32_t)sh.through[4];
        r.lpre[(uint32_t)sh.through[1]] = sh.through[2];
        r.lk0[(uint32_t)sh.through[1]] = (uint32_t)sh.through[4];
        r.sprefix[sh.through[0] >> 32] = sh.through[3];
    }
}

// A light unit is the light rows whose first products fall in the same bin of
// `bin` products (counted over the light rows): its products stay below
// bin + light_max.  Its rows need not be neighbours: rows of other classes
// between them used to end a unit, which left units of one or two rows (157 to
// 556 products) where single-run rows lie between the light ones.
__global__ void __launch_bounds__(kScanThreads)
    k_light_units(uint64_t bin, RowArrays r, uint64_t *__restrict__ cnts, ScanState st) {
    __shared__ ScanShared<1> sh;
    if (ld_acquire(st.err) & kScanErr) return;
    const uint64_t n = cnts[kCntLight];
    const uint32_t tile = next_tile(st, sh);
    if ((uint64_t)tile * kScanTile >= n) return;
    const uint64_t i0 = (uint64_t)tile * kScanTile + (uint64_t)threadIdx.x * kScanItems;
    uint32_t starts = 0;  // bit q: a unit starts at light row i0 + q
    uint64_t pb = i0 > 0 && i0 < n ? r.lpre[i0 - 1] / bin : 0;
#pragma unroll
    for (int q = 0; q < kScanItems; ++q) {
        const uint64_t i = i0 + q;
        if (i < n) {
            const uint64_t b = r.lpre[i] / bin;
            if (i == 0 || b != pb) starts |= 1u << q;
            pb = b;
        }
    }
    uint64_t x[1] = {(uint64_t)__popc(starts)};
    if (!tile_scan<1>(st, sh, tile, x)) return;
#pragma unroll
    for (int q = 0; q < kScanItems; ++q)
        if (starts >> q & 1u) r.ustart[x[0]++] = (uint32_t)(i0 + q);
    if ((uint64_t)(tile + 1) * kScanTile >= n && threadIdx.x == 0) {
        cnts[kCntUnits] = sh.through[0];
        r.ustart[sh.through[0]] = (uint32_t)n;
    }
}

// A thread per matched X nonzero.  Light rows: their runs one after another,
// with the products before each.  Heavy rows: the rank span (runs are sorted by
// rank, so a run's first and last entries bound it); a warp whose nonzeros are
// of one row (long rows) folds them first.  With a warp per row, 200 rows of
// 5e4 runs took 1155 us (200 warps at work); now 146.
//
// Where X is sorted by its free bits alone, a light row's runs are put in the
// order of their contract keys (the order of their first Y entries), equal keys
// in input order, as a sort by all bits leaves them.  So a light row's sums
// depend neither on the order of the input nor on the jobs beside it.  Up to
// kOrderScan runs: a thread counts the runs before its own (loads that its
// row's other threads make too); more: k_light_order.
__global__ void k_matched_runs(const uint32_t *__restrict__ pos, const uint32_t *__restrict__ cnt,
                               const uint32_t *__restrict__ yrank, RowArrays r, const uint64_t *__restrict__ cnts,
                               const unsigned int *__restrict__ err) {
    if (*err & kScanErr) return;
    uint32_t *const row_rb = r.row_rb, *const row_mx = r.row_mx;
    const uint64_t n = r.row_k0[cnts[kCntRows]];  // matched nonzeros
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t t0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (uint64_t k0 = t0 - (threadIdx.x & 31); k0 < n; k0 += stride) {  // whole warps
        const uint64_t k = k0 + (threadIdx.x & 31);
        const uint32_t row = r.mrow[k < n ? k : n - 1];
        const uint8_t cl = k < n ? r.row_class[row] : kRowNone;
        if (cl == kRowLight) {
            const uint32_t i = r.mrun[k], l = r.row_xi[row], k0r = r.row_k0[row], m = r.row_k0[row + 1] - k0r;
            uint32_t at = (uint32_t)k - k0r;
            uint64_t off = r.xprefix[i] - r.xprefix[r.row_start[row]];
            if (r.longs && m <= kOrderScan) {
                const uint32_t p = pos[i];
                uint32_t n = 0;  // a light row has at most 2048 products
                at = 0;
#pragma unroll 4
                for (uint32_t t = 0; t < m; ++t) {
                    const uint32_t j = r.mrun[k0r + t], q = pos[j], c = cnt[j];
                    if (q < p || (q == p && j < i)) {
                        ++at;
                        n += c;
                    }
                }
                off = n;
            }
            at += r.lk0[l];
            r.lrun[at] = i;
            r.lrow[at] = l;
            r.loff[at] = r.lpre[l] + off;
        }
        if (!row_rb) continue;  // the same in every thread
        const bool heavy = cl == kRowHeavy;
        uint32_t lo = 0xffffffffu, hi = 0;
        if (heavy) {
            const uint32_t i = r.mrun[k], p = pos[i];
            lo = yrank[p];
            hi = yrank[p + cnt[i] - 1];
        }
        const uint32_t first = __shfl_sync(0xffffffffu, row, 0);
        if (__all_sync(0xffffffffu, row == first)) {
            lo = __reduce_min_sync(0xffffffffu, lo);
            hi = __reduce_max_sync(0xffffffffu, hi);
            if ((threadIdx.x & 31) == 0 && heavy) {
                if (lo < __ldcg(row_rb + row)) atomicMin(row_rb + row, lo);
                if (hi > __ldcg(row_mx + row)) atomicMax(row_mx + row, hi);
            }
        } else if (heavy) {
            atomicMin(row_rb + row, lo);
            atomicMax(row_mx + row, hi);
        }
    }
}

// The same order for the light rows of more than kOrderScan runs, a CTA a row: a
// bitonic sort on chip (these rows are few; with none, 3 us).
constexpr int kOrderRuns = 2048;  // a light row has no more products
static_assert(kOrderRuns >= kLightCap / 2, "the largest light_row_max");
__global__ void __launch_bounds__(kThreads)
    k_light_order(const uint32_t *__restrict__ pos, const uint32_t *__restrict__ cnt, RowArrays r,
                  const uint64_t *__restrict__ cnts, const unsigned int *__restrict__ err) {
    constexpr int kPer = kOrderRuns / kThreads;
    __shared__ uint64_t key[kOrderRuns];  // first Y entry, X nonzero
    __shared__ uint32_t s_tmp[33];
    if (*err & kScanErr) return;
    const uint32_t n = (uint32_t)cnts[kCntLong], tid = threadIdx.x;
    for (uint32_t w = blockIdx.x; w < n; w += gridDim.x) {
        const uint32_t l = r.longs[w], a = r.lk0[l], m = min(r.lk0[l + 1] - a, (uint32_t)kOrderRuns);
        uint32_t padded = 1;
        while (padded < m) padded <<= 1;
        __syncthreads();  // the row before this one has left `key`
        for (uint32_t t = tid; t < padded; t += kThreads) {
            const uint32_t i = t < m ? r.lrun[a + t] : 0u;
            key[t] = t < m ? (uint64_t)pos[i] << 32 | i : ~0ull;
        }
        __syncthreads();
        for (uint32_t k = 2; k <= padded; k <<= 1)
            for (uint32_t j = k >> 1; j > 0; j >>= 1) {
                for (uint32_t t = tid; t < padded / 2; t += kThreads) {
                    const uint32_t lo = ((t & ~(j - 1)) << 1) | (t & (j - 1)), hi = lo | j;
                    const uint64_t x = key[lo], y = key[hi];
                    if ((x > y) == ((lo & k) == 0)) {
                        key[lo] = y;
                        key[hi] = x;
                    }
                }
                __syncthreads();
            }
        uint32_t c[kPer], sum = 0, all;
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const uint32_t t = tid * kPer + q;
            c[q] = sum;
            if (t < m) sum += cnt[(uint32_t)key[t]];
        }
        const uint32_t before = block_excl_scan_u32<kThreads>(sum, s_tmp, &all);
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const uint32_t t = tid * kPer + q;
            if (t < m) {
                r.lrun[a + t] = (uint32_t)key[t];
                r.loff[a + t] = r.lpre[l] + before + c[q];
            }
        }
    }
}

__global__ void __launch_bounds__(kScanThreads)
    k_heavy_words(RowArrays r, uint32_t *__restrict__ w_all, uint32_t *__restrict__ w_dense, uint64_t *__restrict__ off_all,
                  uint64_t *__restrict__ off_dense, uint64_t *__restrict__ cnts, ScanState st) {
    __shared__ ScanShared<2> sh;
    if (ld_acquire(st.err) & kScanErr) return;
    const uint64_t n = cnts[kCntHeavy];
    const uint32_t tile = next_tile(st, sh);
    if ((uint64_t)tile * kScanTile >= n) return;
    const uint64_t i0 = (uint64_t)tile * kScanTile + (uint64_t)threadIdx.x * kScanItems;
    uint32_t wa[kScanItems], wd[kScanItems];
    uint64_t x[2] = {0, 0};
#pragma unroll
    for (int q = 0; q < kScanItems; ++q) {
        wa[q] = wd[q] = 0;
        if (i0 + q < n) {
            const uint32_t row = r.H[i0 + q];
            const uint64_t span = (uint64_t)r.row_mx[row] - r.row_rb[row] + 1, prod = r.row_prod[row];
            // narrow rows keep no bitmap here
            const uint32_t words = r.row_class[row] == kRowHeavy ? (uint32_t)(((span + 127) >> 7) << 2) : 0u;
            wa[q] = span <= kKeepBitsMax * prod ? words : 0u;
            wd[q] = span <= kKeepBitsPerProduct * prod ? words : 0u;
            x[0] += wa[q];
            x[1] += wd[q];
        }
    }
    if (!tile_scan<2>(st, sh, tile, x)) return;
#pragma unroll
    for (int q = 0; q < kScanItems; ++q)
        if (i0 + q < n) {
            const uint32_t row = r.H[i0 + q];
            w_all[row] = wa[q];
            w_dense[row] = wd[q];
            off_all[row] = x[0];
            off_dense[row] = x[1];
            x[0] += wa[q];
            x[1] += wd[q];
        }
    if ((uint64_t)(tile + 1) * kScanTile >= n && threadIdx.x == 0) {
        cnts[kCntBmAll] = sh.through[0];
        cnts[kCntBmDense] = sh.through[1];
    }
}

__global__ void __launch_bounds__(kScanThreads)
    k_row_offsets(const uint32_t *__restrict__ row_nnz, uint64_t n, uint64_t *__restrict__ row_off, ScanState st) {
    __shared__ ScanShared<1> sh;
    const uint32_t tile = next_tile(st, sh);
    const uint64_t i0 = (uint64_t)tile * kScanTile + (uint64_t)threadIdx.x * kScanItems;
    uint32_t c[kScanItems];
    if (i0 + kScanItems <= n)
        load8(row_nnz + i0, c);
    else
#pragma unroll
        for (int q = 0; q < kScanItems; ++q) c[q] = i0 + q < n ? row_nnz[i0 + q] : 0u;
    uint64_t x[1] = {0};
#pragma unroll
    for (int q = 0; q < kScanItems; ++q) x[0] += c[q];
    if (!tile_scan<1>(st, sh, tile, x)) return;
#pragma unroll
    for (int q = 0; q < kScanItems; ++q)
        if (i0 + q < n) {
            row_off[i0 + q] = x[0];
            x[0] += c[q];
        }
    if ((uint64_t)(tile + 1) * kScanTile >= n && threadIdx.x == 0) row_off[n] = sh.through[0];
}

void launched() {
    count_launch();
    GS_CUDA(cudaGetLastError());
}

}  // namespace

void launch_y_runs(const uint64_t *ykeys, uint64_t ny, int kby, const BPrep *jobs, uint64_t *run_key,
                   uint32_t *run_start, uint64_t *cnts, unsigned int *ydup, uint32_t *bits, uint64_t *yfk,
                   uint2 *ctab, const ScanState &st, cudaStream_t s) {
    if (ny == 0) return;
    k_y_runs<<<(unsigned)scan_tiles(ny), kScanThreads, 0, s>>>(ykeys, ny, kby, jobs, run_key, run_start, cnts, ydup,
                                                               bits, yfk, ctab, st);
    launched();
}

void launch_col_table(const uint32_t *bits, uint64_t nwords, const BPrep *jobs, int g, uint32_t *wpre, uint64_t *cols,
                      uint64_t *cnts, const ScanState &st, cudaStream_t s) {
    if (nwords == 0) return;
    k_col_table<<<(unsigned)scan_tiles(nwords), kScanThreads, 0, s>>>(bits, nwords, jobs, g, wpre, cols, cnts, st);
    launched();
}

void launch_y_ranks(const uint64_t *ykeys, uint64_t ny, int kby, const BPrep *jobs, int g, const uint32_t *bits,
                    const uint32_t *wpre, const uint64_t *cnts, uint32_t *rank, BatchJob *acc,
                    const unsigned int *ydup, const unsigned int *err, cudaStream_t s) {
    k_y_ranks<<<grid_for(std::max<uint64_t>(ny, (uint64_t)g)), kThreads, 0, s>>>(ykeys, ny, kby, jobs, g, bits, wpre,
                                                                                cnts, rank, acc, ydup, err);
    launched();
}

void launch_x_rows(const uint64_t *xkeys, uint64_t nx, int kbx, const BPrep *jobs, const uint32_t *cnt,
                   const uint8_t *row_flag, const RowArrays &r, uint64_t *cnts, const ScanState &st, cudaStream_t s) {
    if (nx == 0) return;
    k_x_rows<<<(unsigned)scan_tiles(nx), kScanThreads, 0, s>>>(xkeys, nx, kbx, jobs, cnt, row_flag, r, cnts, st);
    launched();
}

void launch_y_cols32(const uint64_t *ykeys, uint64_t ny, int kby, const BatchJob *acc, const uint64_t *cols,
                     const uint32_t *rank, uint32_t *out, const unsigned int *err, cudaStream_t s) {
    if (ny == 0) return;
    k_y_cols32<<<grid_for(ny), kThreads, 0, s>>>(ykeys, ny, kby, acc, cols, rank, out, err);
    launched();
}

void launch_wide_tables(const WideTab *tab, int g, uint64_t n, const uint16_t *row_job, uint64_t *row_xf,
                        uint64_t *cols, BatchJob *acc, const uint64_t *cnts, const unsigned int *err,
                        cudaStream_t s) {
    k_wide_tables<<<grid_for(std::max<uint64_t>(n, (uint64_t)g)), kThreads, 0, s>>>(tab, g, row_job, row_xf, cols, acc,
                                                                                    cnts, err);
    launched();
}

void launch_row_classes(uint64_t nx, const BPrep *jobs, const BatchJob *acc, const uint64_t *range,
                        const RowArrays &r, uint64_t *cnts, const ScanState &st, cudaStream_t s) {
    if (nx == 0) return;
    k_row_classes<<<(unsigned)scan_tiles(nx), kScanThreads, 0, s>>>(jobs, acc, range, r, cnts, st);
    launched();
}

void launch_light_units(uint64_t nx, uint64_t bin, const RowArrays &r, uint64_t *cnts, const ScanState &st,
                        cudaStream_t s) {
    if (nx == 0) return;
    k_light_units<<<(unsigned)scan_tiles(nx), kScanThreads, 0, s>>>(bin, r, cnts, st);
    launched();
}

void launch_matched_runs(uint64_t nx, const uint32_t *pos, const uint32_t *cnt, const uint32_t *yrank,
                         const RowArrays &r, const uint64_t *cnts, const unsigned int *err, cudaStream_t s) {
    if (nx == 0) return;
    k_matched_runs<<<grid_for(nx), kThreads, 0, s>>>(pos, cnt, yrank, r, cnts, err);
    launched();
}

void launch_light_order(uint64_t nx, const uint32_t *pos, const uint32_t *cnt, const RowArrays &r,
                        const uint64_t *cnts, const unsigned int *err, int sm_count, cudaStream_t s) {
    if (nx <= kOrderScan) return;
    k_light_order<<<(unsigned)std::min<uint64_t>(nx / kOrderScan + 1, 8ull * sm_count), kThreads, 0, s>>>(pos, cnt, r,
                                                                                                       cnts, err);
    launched();
}

void launch_heavy_bitmaps(uint64_t nx, const RowArrays &r, uint32_t *w_all, uint32_t *w_dense, uint64_t *off_all,
                          uint64_t *off_dense, uint64_t *cnts, const ScanState &st, cudaStream_t s) {
    if (nx == 0) return;
    k_heavy_words<<<(unsigned)scan_tiles(nx), kScanThreads, 0, s>>>(r, w_all, w_dense, off_all, off_dense, cnts, st);
    launched();
}

void launch_row_offsets(const uint32_t *row_nnz, uint64_t nrows, uint64_t *row_off, const ScanState &st,
                        cudaStream_t s) {
    if (nrows == 0) {
        GS_CUDA(cudaMemsetAsync(row_off, 0, 8, s));
        return;
    }
    k_row_offsets<<<(unsigned)scan_tiles(nrows), kScanThreads, 0, s>>>(row_nnz, nrows, row_off, st);
    launched();
}

}  // namespace gs
