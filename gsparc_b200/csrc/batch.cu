// batch.cu -- many independent contractions run as one.
//
// The reference runs one gsparc::SpTC at a time (include/gsparc/sptc.cuh:16-360,
// driven from main.cu:293-376), so a stream of small contractions pays the
// fixed per-call cost (launches, host round trips) once per contraction.  Here
// the jobs of a batch are split into groups; inside a group every operand key
// carries its job id above the widest key of the group:
//
//     X key = job << kbx | (x_f << ncbits | c),   Y key = job << kby | (c << nfbits | y_f)
//
// so ONE linearise launch per side, ONE radix sort per side, ONE run table and
// ONE match serve every job of the group: sorting by the prefixed key sorts
// each job's keys exactly as the plain path does and keeps jobs apart.  Rows
// (distinct x_f) then know their job, and the accumulation kernels look up the
// job's column table and output key width per row (row_job_params), so ONE
// symbolic and ONE numeric persistent launch take the units of all jobs from
// one work counter.  Unit planning (light units, heavy rows) runs on the
// device, so a group needs two host round trips before its numeric launch
// whatever its number of jobs (the planning kernels are in rows.cu).  Each job's output is the contiguous range of
// the group's sorted output that belongs to it, delivered to the job's sink.
#include <cub/cub.cuh>

#include <algorithm>
#include <chrono>
#include <cstring>
#include <numeric>

#include "chunkkey.h"
#include "engine.h"
#include "kernels.cuh"
#include "rows.h"
#include "runtab.h"
#include "verify.h"
#include "wide.h"

namespace gs {

namespace {

constexpr int kThreads = 256;
constexpr int kMaxGroupJobs = 65535;      // row_job is 16 bits
constexpr uint64_t kMaxGroupNnz = (1ull << 31) - 1;
constexpr uint64_t kFreeSortNnz = 1ull << 12;
constexpr char kLookBackGaveUp[] = "a prefix sum's or the radix sort's look-back gave up";

inline int grid_for(uint64_t n) {
    uint64_t g = (n + kThreads - 1) / kThreads;
    if (g < 1) g = 1;
    if (g > 148ull * 32) g = 148ull * 32;
    return (int)g;
}

__device__ __forceinline__ uint64_t shl(uint64_t v, int s) { return s >= 64 ? 0ull : (v << s); }
__device__ __forceinline__ uint64_t shr(uint64_t v, int s) { return s >= 64 ? 0ull : (v >> s); }
__device__ __forceinline__ uint64_t low_mask(int b) { return b >= 64 ? ~0ull : ((1ull << b) - 1); }

template <class T>
__device__ __forceinline__ uint64_t lower_bound_dev(const T *a, uint64_t lo, uint64_t hi, T v) {
    while (lo < hi) {
        uint64_t mid = (lo + hi) >> 1;
        if (a[mid] < v)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

// One operand of one job, for the batched linearise.
struct BLin {
    LinParams p;
    const uint64_t *idx;  // SoA idx[m * nnz + k]
    const float *val;
    uint64_t nnz;
};

// Per-job summary after the symbolic pass (entry g holds the totals, entry
// g + 1 the largest output of one row and the error bits).
struct JobOut {
    uint64_t row0;     // first row of the job
    uint64_t out_off;  // first output nonzero of the job
    uint64_t ir_off;   // matched products before the job
    uint64_t heavy0;   // heavy rows before the job
};

// reference: include/gsparc/tensor_manager.tpp:249-268 (X) and :272-293 (Y),
// once per job, with the job id above the group's widest key.  A key is masked
// to the group width, so an out-of-range index (flagged per job) can only
// damage its own job's keys.
__global__ void k_blin(const BLin *__restrict__ tab, const uint64_t *__restrict__ offs, int g,
                       uint64_t total, int kb, uint64_t *__restrict__ keys, float *__restrict__ vals,
                       unsigned int *__restrict__ jerr, int perm) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t km = low_mask(kb);
    for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < total; k += stride) {
        int lo = 0, hi = g;  // largest j with offs[j] <= k
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (offs[mid] <= k)
                lo = mid;
            else
                hi = mid;
        }
        const BLin &t = tab[lo];
        const uint64_t l = k - offs[lo];
        uint64_t f = 0, c = 0;
        bool bad = false;
        for (int m = 0; m < t.p.order; ++m) {
            const uint64_t v = t.idx[(uint64_t)m * t.nnz + l];
            bad |= v >= t.p.dims[m];
            if (t.p.is_c[m])
                c |= shl(v, t.p.shift[m]);
            else
                f |= shl(v, t.p.shift[m]);
        }
        if (bad) atomicOr(&jerr[lo], 1u);
        const uint64_t key = t.p.role == 0 ? (shl(f, t.p.ncbits) | c) : (shl(c, t.p.nfbits) | f);
        keys[k] = shl((uint64_t)lo, kb) | (key & km);
        // with perm the sort carries each entry's input position instead of its value
        vals[k] = perm ? __uint_as_float((unsigned int)k) : t.val[l];
    }
}

// The current values of sorted entries whose input positions the sort carried
// (k_blin with perm): vals[i] = the value at input position perm[i].
__global__ void k_bvals(const BLin *__restrict__ tab, const uint64_t *__restrict__ offs, int g, uint64_t total,
                        const float *__restrict__ perm, float *__restrict__ vals) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        const uint64_t k = __float_as_uint(perm[i]);
        int lo = 0, hi = g;  // largest j with offs[j] <= k
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (offs[mid] <= k)
                lo = mid;
            else
                hi = mid;
        }
        vals[i] = tab[lo].val[k - offs[lo]];
    }
}

// Distinct prefixed free indices -> plain free indices (the column tables).
__global__ void k_bcols(const uint64_t *__restrict__ uniq, const uint64_t *__restrict__ ncols_dev,
                        int kby, uint64_t *__restrict__ cols) {
    const uint64_t n = *ncols_dev;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t km = low_mask(kby);
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
        cols[i] = uniq[i] & km;
}

// Per-job column table range inside the group's table.
__global__ void k_bjobs(const uint64_t *__restrict__ uniq, const uint64_t *__restrict__ ncols_dev,
                        int kby, int g, const BPrep *__restrict__ jobs, const unsigned int *__restrict__ ydup,
                        BatchJob *__restrict__ acc) {
    const uint64_t n = *ncols_dev;
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < g; j += gridDim.x * blockDim.x) {
        const uint64_t lo = lower_bound_dev<uint64_t>(uniq, 0, n, shl((uint64_t)j, kby));
        const uint64_t hi = (j + 1 == g) ? n : lower_bound_dev<uint64_t>(uniq, 0, n, shl((uint64_t)(j + 1), kby));
        BatchJob b;
        b.y_nfbits = jobs[j].y_nfbits;
        b.ncols = (uint32_t)(hi - lo);
        b.ydup = ydup[j];
        b.wide = 0;
        b.cols_off = lo;
        acc[j] = b;
    }
}

// Column rank of every Y entry inside its job's column table.
__global__ void k_brank(const uint64_t *__restrict__ ykeys, uint64_t ny, int kby,
                        const BPrep *__restrict__ jobs, const uint64_t *__restrict__ uniq,
                        const BatchJob *__restrict__ acc, uint32_t *__restrict__ rank) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t km = low_mask(kby);
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < ny; i += stride) {
        const uint64_t key = ykeys[i];
        const uint64_t j = shr(key, kby);
        const uint64_t f = key & km & low_mask(jobs[j].y_nfbits);
        const BatchJob b = acc[j];
        const uint64_t p = lower_bound_dev<uint64_t>(uniq, b.cols_off, b.cols_off + b.ncols, shl(j, kby) | f);
        rank[i] = (uint32_t)(p - b.cols_off);
    }
}

// reference: include/gsparc/indexMatch.cuh:67-118, over the run table of all
// jobs: the search key is (job, contract key).  With the lookup table (ctab) a
// run is its word's first run plus the keys below it in the word: one table
// load instead of a binary search, whatever the order of the X nonzeros.
__global__ void k_bmatch(const uint64_t *__restrict__ xkeys, uint64_t nx, int kbx, int kby,
                         const BPrep *__restrict__ jobs, const uint64_t *__restrict__ run_key,
                         const uint32_t *__restrict__ run_start, const uint64_t *__restrict__ nruns_dev,
                         const uint2 *__restrict__ ctab, uint32_t *__restrict__ pos, uint32_t *__restrict__ cnt,
                         uint8_t *__restrict__ row_flag) {
    const uint64_t nr = *nruns_dev;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t km = low_mask(kbx);
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nx; i += stride) {
        const uint64_t key = xkeys[i];
        const uint64_t j = shr(key, kbx);
        const BPrep b = jobs[j];
        const int ncb = b.x_ncbits;
        const uint64_t loc = key & km, c = loc & low_mask(ncb);
        uint64_t r = nr;
        if (ctab) {
            const uint2 t = ctab[b.con_word0 + (c >> 5)];
            r = run_of_key(t.x, t.y, c, nr);
        } else {
            const uint64_t target = shl(j, kby) | c;
            r = lower_bound_dev<uint64_t>(run_key, 0, nr, target);
            if (r < nr && run_key[r] != target) r = nr;
        }
        uint32_t p = 0, n = 0;
        if (r < nr) {
            p = run_start[r];
            n = run_start[r + 1] - p;
        }
        pos[i] = p;
        cnt[i] = n;
        uint8_t flag = 1;
        if (i > 0) {
            const uint64_t pk = xkeys[i - 1];
            flag = (shr(pk, kbx) != j) || (shr(pk & km, ncb) != shr(loc, ncb));
        }
        row_flag[i] = flag;
    }
}

// Row range of one shard of a single job: shard s starts at the first row
// whose product midpoint reaches s/n of the job's products, i.e. the first r
// with n * (P[r] + P[r+1]) >= 2 * s * P[nrows] (P = row product prefix: the
// products before the row's first nonzero), the exact-integer form of the host
// planner gs::plan_shards.
// range = {first row, end row, products of the shard}.
__device__ uint64_t shard_bound(const uint64_t *xprefix, const uint32_t *row_start, uint64_t nr, int s, int n) {
    if (s <= 0) return 0;
    if (s >= n) return nr;
    const unsigned __int128 target = (unsigned __int128)2 * (unsigned)s * xprefix[row_start[nr]];
    uint64_t lo = 0, hi = nr;
    while (lo < hi) {
        const uint64_t mid = (lo + hi) >> 1;
        if ((unsigned __int128)(unsigned)n *
                ((unsigned __int128)xprefix[row_start[mid]] + xprefix[row_start[mid + 1]]) >= target)
            hi = mid;
        else
            lo = mid + 1;
    }
    return lo;
}

__global__ void k_shard_range(const uint64_t *__restrict__ xprefix, const uint32_t *__restrict__ row_start,
                              const uint64_t *__restrict__ nrows_dev, int shard, int nshards,
                              uint64_t *__restrict__ range, const unsigned int *__restrict__ err) {
    if (*err & kScanErr) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        const uint64_t nr = *nrows_dev;
        const uint64_t a = shard_bound(xprefix, row_start, nr, shard, nshards);
        const uint64_t b = shard_bound(xprefix, row_start, nr, shard + 1, nshards);
        range[0] = a;
        range[1] = b;
        range[2] = xprefix[row_start[b]] - xprefix[row_start[a]];
    }
}

// Sort key of the heavy rows' order (descending): rows of the windowed kernel
// before narrow rows, largest first by the product count's binary exponent and
// one mantissa bit, in one 8-bit radix pass (the order only balances the work:
// a row within a third of the next is as good).
__global__ void k_heavy_sizes(const uint32_t *__restrict__ H, uint64_t nh, const uint64_t *__restrict__ row_prod,
                              const uint8_t *__restrict__ row_class, uint8_t *__restrict__ hp) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < nh; k += stride) {
        const uint64_t p = row_prod[H[k]] | 2u;
        const int e = 63 - __clzll((long long)p);
        const bool narrow = row_class && row_class[H[k]] == kRowNarrow;
        hp[k] = (uint8_t)((narrow ? 0 : 128) | (e << 1) | ((p >> (e - 1)) & 1u));
    }
}

// The three row lists of a group, all in row order: light, heavy and
// single-run (stream) rows.
struct UnitLists {
    const uint32_t *L;
    uint64_t nl;
    const uint32_t *H;
    uint64_t nh;
    const uint32_t *SR;
    uint64_t ns;
    __device__ uint64_t size() const { return nl + nh + ns; }
    // row k of the concatenation light | heavy | stream
    __device__ uint32_t row(uint64_t k) const {
        return k < nl ? L[k] : (k < nl + nh ? H[k - nl] : SR[k - nl - nh]);
    }
    // rows of all three lists before row r
    __device__ uint64_t before(uint32_t r) const {
        return lower_bound_dev<uint32_t>(L, 0, nl, r) + lower_bound_dev<uint32_t>(H, 0, nh, r) +
               lower_bound_dev<uint32_t>(SR, 0, ns, r);
    }
};

// Per-job summaries and the largest output of one unit.
__global__ void k_after_counts(UnitLists u, const uint64_t *__restrict__ row_off, const uint16_t *__restrict__ row_job,
                               uint64_t nrows, const uint64_t *__restrict__ xprefix,
                               const uint64_t *__restrict__ xoffs, int g, const unsigned int *__restrict__ err,
                               JobOut *__restrict__ jobs) {
    if (blockIdx.x == 0 && threadIdx.x == 0) jobs[g + 1].out_off = *err;
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j <= g; j += gridDim.x * blockDim.x) {
        const uint64_t r0 = (j == g) ? nrows : lower_bound_dev<uint16_t>(row_job, 0, nrows, (uint16_t)j);
        JobOut o;
        o.row0 = r0;
        o.out_off = row_off[r0];
        o.ir_off = xprefix[xoffs[j]];
        o.heavy0 = lower_bound_dev<uint32_t>(u.H, 0, u.nh, (uint32_t)r0);
        jobs[j] = o;
    }
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    uint64_t m = 0;
    for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < u.size(); k += stride) {
        const uint32_t r = u.row(k);
        const uint64_t v = row_off[r + 1] - row_off[r];
        m = v > m ? v : m;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const uint64_t w = __shfl_xor_sync(0xffffffffu, m, o);
        m = w > m ? w : m;
    }
    if ((threadIdx.x & 31) == 0 && m) atomicMax((unsigned long long *)&jobs[g + 1].row0, (unsigned long long)m);
}

// First row and first output of every unit, the three lists merged in row
// order (the lists are row-ordered and their rows are disjoint).
__global__ void k_merge_starts(UnitLists u, const uint64_t *__restrict__ row_off, uint32_t *__restrict__ urow,
                               uint64_t *__restrict__ uoff) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < u.size(); k += stride) {
        const uint32_t r = u.row(k);
        const uint64_t p = u.before(r);
        urow[p] = r;
        uoff[p] = row_off[r];
    }
}

// Chunk k starts at the first unit whose output starts at or after
// target[k] (target[0] = 0, increasing).  info[5k..5k+4] = first row, first
// output, first light row, first heavy row (row-ordered index), first stream
// row of chunk k; entry K closes the last chunk.
constexpr int kChunkInfo = 5;
__global__ void k_chunk_bounds(const uint32_t *__restrict__ urow, const uint64_t *__restrict__ uoff, uint64_t M,
                               const uint64_t *__restrict__ target, uint64_t K, UnitLists u, uint64_t nrows,
                               uint64_t ntot, uint64_t *__restrict__ info) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k <= K; k += stride) {
        const uint64_t b = k == 0 ? 0 : (k == K ? M : lower_bound_dev<uint64_t>(uoff, 0, M, target[k]));
        const uint32_t row = (uint32_t)(b < M ? urow[b] : nrows);
        uint64_t *o = info + kChunkInfo * k;
        o[0] = row;
        o[1] = b < M ? uoff[b] : ntot;
        o[2] = lower_bound_dev<uint32_t>(u.L, 0, u.nl, row);
        o[3] = lower_bound_dev<uint32_t>(u.H, 0, u.nh, row);
        o[4] = lower_bound_dev<uint32_t>(u.SR, 0, u.ns, row);
    }
}

// Sort keys grouping heavy rows by chunk (chunkkey.h).
__global__ void k_heavy_chunk_keys(const uint32_t *__restrict__ Hs, uint64_t nh,
                                   const uint64_t *__restrict__ row_prod, const uint8_t *__restrict__ row_class,
                                   const uint64_t *__restrict__ info, uint64_t K, uint64_t *__restrict__ keys) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < nh; k += stride) {
        const uint32_t r = Hs[k];
        uint64_t lo = 0, hi = K;  // last chunk whose first row <= r
        while (hi - lo > 1) {
            const uint64_t mid = (lo + hi) >> 1;
            if (info[kChunkInfo * mid] <= r)
                lo = mid;
            else
                hi = mid;
        }
        keys[k] = heavy_chunk_key(lo, row_class && row_class[r] == kRowNarrow, row_prod[r]);
    }
}

template <class T>
void h2d(T *d, const T *h, size_t n, cudaStream_t s) {
    if (n) GS_CUDA(cudaMemcpyAsync(d, h, sizeof(T) * n, cudaMemcpyHostToDevice, s));
}
template <class T>
void d2h(T *h, const T *d, size_t n, cudaStream_t s) {
    if (n) GS_CUDA(cudaMemcpyAsync(h, d, sizeof(T) * n, cudaMemcpyDeviceToHost, s));
}

inline int ceil_log2(uint64_t n) {
    int b = 0;
    while ((1ull << b) < n) ++b;
    return b;
}

struct Job {
    gsparc_job *job;
    const gsparc_tensor *tx, *ty;   // the operands the engine runs on (relabeled when wide)
    std::shared_ptr<WideMap> wide;  // set when the operand keys need more than 64 bits
    Layout LX, LY;
    uint64_t light_max;
    int width;          // widest operand key
    int key_words = 1;  // output key words delivered to the sink (2: 128-bit keys)
    bool done = false;  // reported through the completion callback
};

// First product count after which a job boundary closes a chunk when jobs
// complete one by one (about a millisecond of accumulation); each further cut
// waits for twice as many products, so a batch has O(log) extra chunks.
constexpr uint64_t kFirstCutProducts = 1ull << 26;

struct Times {
    double lin = 0, sort = 0, match = 0, plan = 0, contract = 0, out = 0, total = 0, numeric = 0;
};

// Everything the numeric pass of one group needs, kept on the device by a plan
// (gsparc_plan_*): the sorted operands' positions and current values, the run
// table, the match, the rows, the unit lists and the output offsets.
struct GroupPlan {
    int g = 0;
    uint64_t nx = 0, ny = 0, ntot = 0, nu = 0, nh = 0, nsr = 0, nnarrow = 0;
    int sm_count = 148;
    int gl = 1, gh = 1, gs_grid = 1;
    AccArgs aa{};
    std::vector<uint64_t> job_first;  // g + 1 group-local output offsets
    std::vector<Job *> jobs;
    DBuf<uint8_t> tabs;
    const BLin *d_lx = nullptr, *d_ly = nullptr;
    const uint64_t *d_xoffs = nullptr, *d_yoffs = nullptr;
    DBuf<float> xperm, yperm, xvals, yvals;
    DBuf<uint64_t> ykeys;  // sorted Y keys (the single-run-row copy reads y_f from them)
    DBuf<BatchJob> d_acc;
    DBuf<uint32_t> rank, ycol, pos, cnt, mpre, mrun, row_start, L, ustart, lk0, lrun, lrow, H, H2, SR, row_xi, cursor, pend;
    DBuf<uint64_t> cols, xprefix, row_xf, sprefix, row_off, lpre, loff;
    DBuf<uint16_t> row_job;
    DBuf<uint32_t> Hc;         // heavy rows grouped by chunk (several chunks only)
    DBuf<uint32_t> hbm, row_rb, row_bmw;  // heavy rows' kept column bitmaps (may be empty)
    DBuf<uint64_t> row_bmoff;
    DBuf<uint32_t> nbm, unit_off, part_off;  // narrow rows (may be empty)
    DBuf<float2> part;
    DBuf<uint8_t> row_class;
    DBuf<unsigned int> flags;  // error bits, work counter, windows swept, spare
    struct Chunk {
        uint64_t lu0, lu1, h0, h1, s0, s1, first, n;
    };
    std::vector<Chunk> chunks;
    const uint32_t *heavy_list() const { return Hc.get() ? Hc.get() : (H2.get() ? H2.get() : H.get()); }
};

// Delivers [dk, dk + n) of a job's output (first = offset inside the job);
// kw = key words per nonzero (2: 128-bit keys, dk holds 2n words).
void deliver_slice(gsparc_sink &sink, const uint64_t *dk, const float *dv, uint64_t n, uint64_t first,
                   uint64_t job_nnz, cudaStream_t s2, gsparc_stats &st, uint64_t &bytes_d2h, int kw = 1) {
    if (n == 0) return;
    if (sink.kind == GSPARC_SINK_DEVICE) {
        const uint64_t step = sink.max_chunk_nnz ? sink.max_chunk_nnz : n;
        for (uint64_t off = 0; off < n; off += step) {
            const uint64_t m = std::min(step, n - off);
            if (sink.on_chunk(sink.user, dk + kw * off, dv + off, m, first + off, 1))
                fail(GSPARC_ECALLBACK, "output callback stopped the contraction");
        }
        ++st.chunks;
    } else if (sink.kind == GSPARC_SINK_HOST) {
        if (sink.host_capacity >= job_nnz) {
            d2h(sink.host_keys + kw * first, dk, kw * n, s2);
            d2h(sink.host_vals + first, dv, n, s2);
            bytes_d2h += (8 * kw + 4) * n;
            GS_CUDA(cudaStreamSynchronize(s2));
            if (sink.on_chunk &&
                sink.on_chunk(sink.user, sink.host_keys + kw * first, sink.host_vals + first, n, first, 0))
                fail(GSPARC_ECALLBACK, "output callback stopped the contraction");
        } else {
            for (uint64_t off = 0; off < n; off += sink.host_capacity) {
                const uint64_t m = std::min<uint64_t>(sink.host_capacity, n - off);
                d2h(sink.host_keys, dk + kw * off, kw * m, s2);
                d2h(sink.host_vals, dv + off, m, s2);
                bytes_d2h += (8 * kw + 4) * m;
                GS_CUDA(cudaStreamSynchronize(s2));
                if (sink.on_chunk && sink.on_chunk(sink.user, sink.host_keys, sink.host_vals, m, first + off, 0))
                    fail(GSPARC_ECALLBACK, "output callback stopped the contraction");
            }
        }
        ++st.chunks;
    }
}

void run_group(gsparc_ctx *ctx, std::vector<Job *> &G, uint64_t max_chunk_nnz, int shard, int nshards,
               Times &tm, gsparc_stats &bst, cudaStream_t s, const JobDoneFn *done_fn, GroupPlan *keep = nullptr) {
    Arena &A = ctx->arena;
    const int g = (int)G.size();
    const int jb = ceil_log2((uint64_t)g);
    int kbx = 0, kby = 0;
    uint64_t max_light = 0;
    for (Job *j : G) {
        kbx = std::max(kbx, j->LX.nbits());
        kby = std::max(kby, j->LY.nbits());
        max_light = std::max(max_light, j->light_max);
    }
    // light units hold rows whose first product falls in one bin of light_bin
    // products: fewer than light_bin + light_max <= light_cap products
    const uint64_t light_cap = max_light <= kLightRowMax ? kLightCap / 2 : kLightCap;
    const uint64_t light_bin = light_cap - std::min<uint64_t>(max_light, light_cap - 1);
    GS_REQUIRE(kbx + jb <= 64 && kby + jb <= 64, GSPARC_EINTERNAL, "batch group keys wider than 64 bits");

    cudaEvent_t *ev = ctx->ev;
    auto mark = [&](int i) { GS_CUDA(cudaEventRecord(ev[i], s)); };
    auto at = [&](int i) {
        float t = 0.f;
        GS_CUDA(cudaEventElapsedTime(&t, ev[0], ev[i]));
        return (double)t;
    };
    // The stages up to the symbolic pass; returns where they end.  The operands'
    // run side by side: one ends when both operands are through it (events 1, 2:
    // Y, 10, 9: X).
    auto planning_times = [&] {
        const double lin = std::max(at(1), at(10)), sorted = std::max(at(2), at(9)), match = std::max(at(3), sorted);
        const double end = at(4);
        tm.lin += lin;
        tm.sort += sorted - lin;
        tm.match += match - sorted;
        tm.plan += end - match;
        return end;
    };
    mark(0);

    // ---- job tables ----
    std::vector<uint64_t> xoffs(g + 1, 0), yoffs(g + 1, 0);
    std::vector<BLin> lx(g), ly(g);
    std::vector<BPrep> bp(g);
    uint64_t col_words = 0, con_words = 0;
    int min_ncb = 64;
    const auto words_of = [](int bits) { return bits >= 38 ? 1ull << 33 : ((1ull << bits) + 31) >> 5; };
    for (int j = 0; j < g; ++j) {
        const gsparc_job &J = *G[j]->job;
        const gsparc_tensor *tx = G[j]->tx, *ty = G[j]->ty;
        xoffs[j + 1] = xoffs[j] + tx->nnz;
        yoffs[j + 1] = yoffs[j] + ty->nnz;
        lx[j] = {make_lin_params(G[j]->LX, tx->dims, 0), tx->d_idx, tx->d_val, tx->nnz};
        ly[j] = {make_lin_params(G[j]->LY, ty->dims, 1), ty->d_idx, ty->d_val, ty->nnz};
        bp[j] = {G[j]->LX.ncbits, G[j]->LY.nfbits, G[j]->light_max, col_words, con_words};
        col_words += words_of(G[j]->LY.nfbits);
        con_words += words_of(G[j]->LX.ncbits);
        min_ncb = std::min(min_ncb, G[j]->LX.ncbits);
    }
    const uint64_t nx = xoffs[g], ny = yoffs[g];
    // Column ranks through presence bits (and a prefix of their words) where
    // these take at most 64 B per Y nonzero, or 4 MiB, and a quarter of the
    // memory left; by sorting the free indices otherwise.  For 1.55e5 entries
    // over 2^24 free indices the scan and the lookups take 24 us (ncu) where the
    // sort, its unique and the searches took 60; for 1e7 entries over 300, 42
    // against 600.  The scan's time grows with the space (the bound keeps its
    // bytes within a few times those of the sort's passes over Y), and the
    // memory stays below the sort's two buffers except in the 4 MiB allowance.
    // What the planning needs in any case comes first.
    const uint64_t plan_need = 192 * nx + 96 * ny + (8ull << 20);
    const uint64_t table_most = std::min(std::max<uint64_t>(64 * ny, 4ull << 20),
                                         (A.available() - std::min(A.available(), plan_need)) / 4);
    const bool col_bits = col_words * 8 <= table_most;
    // The run lookup table (8 B per 32 contract keys) under the same bounds.
    // 1e7 x 1e7 nonzeros over 2^24 contract keys: match 241 -> 101 us.
    const bool con_tab = con_words * 8 <= table_most;
    // With the table the match does not care for the order of a row's nonzeros, so X
    // is sorted by its free bits alone where that saves a radix pass (at the size
    // above 4 -> 1 passes of 122 us).  Light rows add in the order of their contract
    // keys whatever the input's order and the jobs beside them, so the planning puts
    // their runs in it (k_matched_runs), which costs by the runs of a row: 8e6 X
    // nonzeros in rows of 2 / 8 / 32 / 64 / 1000 runs of one product take 2.39 / 1.51 /
    // 1.42 / 1.55 / 1.61 ms so and 2.57 / 1.57 / 1.37 / 1.36 / 1.39 sorted by all bits.
    // So not where X has from 16 nonzeros for every free index up to twice what a
    // light row may have products (past that few rows are light), nor for small
    // inputs, where a launch more costs what the passes do.
    const auto passes = [](int bits) { return (bits + 7) / 8; };
    bool by_free = con_tab && nx >= kFreeSortNnz && passes(kbx + jb - min_ncb) < passes(kbx + jb);
    bool any_light = false;
    for (Job *q : G) {
        const uint64_t a = q->LX.nfbits < 64 ? q->tx->nnz >> q->LX.nfbits : 0;
        by_free &= a < 16 || a >= 2 * q->light_max;
        any_light |= q->light_max != 0;
    }
    // relabeled jobs with 64-bit output keys
    bool any_wide = false;
    for (Job *q : G) any_wide |= q->wide && q->key_words == 1;
    // the job tables, copied at once
    const size_t o_ly = sizeof(BLin) * g, o_bp = 2 * o_ly, o_xo = o_bp + sizeof(BPrep) * g,
                 o_yo = o_xo + 8 * (size_t)(g + 1), o_wt = o_yo + 8 * (size_t)(g + 1),
                 tab_bytes = o_wt + sizeof(WideTab) * (any_wide ? g : 0);
    static_assert(sizeof(BLin) % 8 == 0 && sizeof(BPrep) % 8 == 0, "8-byte aligned tables");
    DBuf<uint8_t> tabs(A, tab_bytes, s);
    const BLin *const d_lx = reinterpret_cast<const BLin *>(tabs.get()),
               *const d_ly = reinterpret_cast<const BLin *>(tabs.get() + o_ly);
    const BPrep *const d_bp = reinterpret_cast<const BPrep *>(tabs.get() + o_bp);
    const uint64_t *const d_xoffs = reinterpret_cast<const uint64_t *>(tabs.get() + o_xo),
                   *const d_yoffs = reinterpret_cast<const uint64_t *>(tabs.get() + o_yo);
    DBuf<BatchJob> d_acc(A, g, s);
    // what starts at zero, cleared at once: the counters (kCnt*), the run lookup
    // table, the jobs' error and repeated-coordinate words, the scans' flags, the presence bits
    const uint64_t zf_y = scan_flag_words(ny), zf_c = col_bits ? scan_flag_words(col_words) : 0,
                   zf_x = scan_flag_words(nx);
    const uint64_t tab_words = con_tab ? 2 * con_words : 0;
    // counters, jobs' error and repeated-coordinate words (an even number of
    // words), run table, job summaries, flags, the work counters of the symbolic pass and the first chunk, bits
    constexpr uint64_t zw_work = 6;
    const uint64_t zw_jobs = 2 * (uint64_t)g, zw_out = sizeof(JobOut) / 4 * (uint64_t)(g + 2);
    const uint64_t zwords = 2 * kCnts + zw_jobs + tab_words + zw_out + zf_y + zf_c + 7 * zf_x + zw_work + (col_bits ? col_words : 0);
    DBuf<uint32_t> zero(A, zwords, s);
    uint64_t *const cnts = reinterpret_cast<uint64_t *>(zero.get());
    unsigned int *const d_jerr = zero.get() + 2 * kCnts, *const d_ydup = d_jerr + g;
    unsigned int *const plan_err = reinterpret_cast<unsigned int *>(cnts + kCntErr);
    uint2 *const ctab = con_tab ? reinterpret_cast<uint2 *>(zero.get() + 2 * kCnts + zw_jobs) : nullptr;
    JobOut *const d_jo = reinterpret_cast<JobOut *>(zero.get() + 2 * kCnts + zw_jobs + tab_words);
    uint32_t *const flags_y = zero.get() + 2 * kCnts + zw_jobs + tab_words + zw_out, *const flags_c = flags_y + zf_y,
                    *const flags_x = flags_c + zf_c;
    unsigned int *const work = flags_x + 7 * zf_x;
    uint32_t *const ybits = col_bits ? work + zw_work : nullptr;
    // the scans' sums (one buffer: the scans follow one another on the stream)
    DBuf<uint64_t> scan_vals(A, std::max({scan_value_words<1>(ny), col_bits ? scan_value_words<1>(col_words) : 0,
                                          scan_value_words<kMaxScanSums>(nx)}), s);
    auto scan_state = [&](uint32_t *flags) { return ScanState{flags, scan_vals.get(), plan_err}; };
    // The scans after the first readback report to the context's error word,
    // which is read again after the symbolic pass and at the end.
    auto late_scan = [&](uint32_t *flags, int which) {
        if (ctx->inject_scan == which) {
            ctx->inject_scan = 0;
            GS_CUDA(cudaMemsetAsync(ctx->d_flag, (int)kScanErr, 1, s));
        }
        return ScanState{flags, scan_vals.get(), ctx->d_flag};
    };
    std::vector<uint8_t> h_tabs(tab_bytes);
    std::memcpy(h_tabs.data(), lx.data(), o_ly);
    std::memcpy(h_tabs.data() + o_ly, ly.data(), o_ly);
    std::memcpy(h_tabs.data() + o_bp, bp.data(), sizeof(BPrep) * g);
    std::memcpy(h_tabs.data() + o_xo, xoffs.data(), 8 * (size_t)(g + 1));
    std::memcpy(h_tabs.data() + o_yo, yoffs.data(), 8 * (size_t)(g + 1));
    if (any_wide)
        for (int j = 0; j < g; ++j) {
            WideTab t{};
            if (G[j]->wide && G[j]->key_words == 1)
                t = {G[j]->wide->xf.get(), G[j]->wide->yf.get(), G[j]->wide->nfbits_y, 0};
            std::memcpy(h_tabs.data() + o_wt + sizeof(WideTab) * j, &t, sizeof(t));
        }
    h2d(tabs.get(), h_tabs.data(), tab_bytes, s);
    GS_CUDA(cudaMemsetAsync(zero.get(), 0, 4 * zwords, s));
    GS_CUDA(cudaMemsetAsync(ctx->d_flag, 0, 4 * 4, s));
    bst.bytes_h2d += (sizeof(BLin) * 2 + sizeof(BPrep) + 16) * g;

    // ---- linearise and sort ----
    // X's on the other stream: it is needed at the match, while Y's tables are
    // made on this one.  Its buffers are this stream's, so they are given back
    // only after the join; an error before it waits for the other stream.
    DBuf<uint64_t> xk0(A, nx, s), xk1(A, nx, s), yk0(A, ny, s), yk1(A, ny, s);
    DBuf<float> xv0(A, nx, s), xv1(A, nx, s), yv0(A, ny, s), yv1(A, ny, s);
    if (keep) {
        keep->xvals.reset(A, std::max<uint64_t>(nx, 1), s);
        keep->yvals.reset(A, std::max<uint64_t>(ny, 1), s);
    }
    const cudaStream_t sx = ctx->alt_stream ? ctx->alt_stream : s;
    struct Join {
        cudaStream_t sx = nullptr;
        ~Join() {
            if (sx) cudaStreamSynchronize(sx);
        }
    } join;
    GS_CUDA(cudaEventRecord(ev[8], s));
    GS_CUDA(cudaStreamWaitEvent(sx, ev[8], 0));
    join.sx = sx;
    const int xbegin = by_free ? min_ncb : 0;
    int wx = 0, wy = 0;
    if (nx) {
        k_blin<<<grid_for(nx), kThreads, 0, sx>>>(d_lx, d_xoffs, g, nx, kbx, xk0, xv0, d_jerr, keep != nullptr);
        count_launch();
        GS_CUDA(cudaGetLastError());
    }
    GS_CUDA(cudaEventRecord(ev[10], sx));
    // gsparc_ctx_set_sort; a failed look-back sets bit 8 of the error word
    if (ctx->sort_impl)
        own_sort_pairs(A, nx, xk0, xk1, xv0, xv1, kbx + jb, &wx, plan_err, sx, xbegin);
    else
        sort_pairs(A, nx, xk0, xk1, xv0, xv1, kbx + jb, &wx, sx, xbegin);
    if (keep && nx) {
        k_bvals<<<grid_for(nx), kThreads, 0, sx>>>(d_lx, d_xoffs, g, nx, wx ? xv1 : xv0, keep->xvals);
        count_launch();
        GS_CUDA(cudaGetLastError());
    }
    GS_CUDA(cudaEventRecord(ev[9], sx));
    if (ny) {
        k_blin<<<grid_for(ny), kThreads, 0, s>>>(d_ly, d_yoffs, g, ny, kby, yk0, yv0, d_jerr, keep != nullptr);
        count_launch();
        GS_CUDA(cudaGetLastError());
    }
    mark(1);
    if (ctx->sort_impl)
        own_sort_pairs(A, ny, yk0, yk1, yv0, yv1, kby + jb, &wy, plan_err, s);
    else
        sort_pairs(A, ny, yk0, yk1, yv0, yv1, kby + jb, &wy, s);
    const uint64_t *xkeys = wx ? xk1.get() : xk0.get();
    const float *xvals = wx ? xv1.get() : xv0.get();
    const uint64_t *ykeys = wy ? yk1.get() : yk0.get();
    const float *yvals = wy ? yv1.get() : yv0.get();
    if (wy) { yk0.release(); yv0.release(); } else { yk1.release(); yv1.release(); }
    if (keep) {
        // the sorted "values" are input positions: keep them, fetch the values
        keep->ykeys = wy ? std::move(yk1) : std::move(yk0);  // ykeys keeps pointing at it
        keep->yperm = wy ? std::move(yv1) : std::move(yv0);
        if (ny) {
            k_bvals<<<grid_for(ny), kThreads, 0, s>>>(d_ly, d_yoffs, g, ny, keep->yperm, keep->yvals);
            count_launch();
            GS_CUDA(cudaGetLastError());
        }
        xvals = keep->xvals.get();
        yvals = keep->yvals.get();
    }
    mark(2);

    // ---- Y column tables, ranks and run table ----
    const uint64_t nyb = std::max<uint64_t>(ny, 1), nxb = std::max<uint64_t>(nx, 1);
    DBuf<uint32_t> rank(A, nyb, s);
    DBuf<uint64_t> cols(A, nyb, s), run_key(A, nyb, s);
    DBuf<uint32_t> run_start(A, ny + 1, s);
    if (col_bits) {
        launch_y_runs(ykeys, ny, kby, d_bp, run_key, run_start, cnts, d_ydup, ybits, nullptr, ctab, scan_state(flags_y), s);
        DBuf<uint32_t> wpre(A, col_words, s);
        launch_col_table(ybits, col_words, d_bp, g, wpre, cols, cnts, scan_state(flags_c), s);
        launch_y_ranks(ykeys, ny, kby, d_bp, g, ybits, wpre, cnts, rank, d_acc, d_ydup, plan_err, s);
    } else {
        DBuf<uint64_t> yf0(A, nyb, s), yf1(A, nyb, s);
        launch_y_runs(ykeys, ny, kby, d_bp, run_key, run_start, cnts, d_ydup, nullptr, yf0, ctab, scan_state(flags_y), s);
        int which = 0;
        sort_keys(A, ny, yf0, yf1, kby + jb, &which, s);
        uint64_t *sorted = which ? yf1.get() : yf0.get();
        uint64_t *uniq = which ? yf0.get() : yf1.get();
        if (ny) {
            size_t tmp = 0;
            GS_CUDA(cub::DeviceSelect::Unique(nullptr, tmp, sorted, uniq, cnts + kCntCols, (int)ny, s));
            DBuf<uint8_t> t(A, tmp, s);
            GS_CUDA(cub::DeviceSelect::Unique(t.get(), tmp, sorted, uniq, cnts + kCntCols, (int)ny, s));
            k_bcols<<<grid_for(ny), kThreads, 0, s>>>(uniq, cnts + kCntCols, kby, cols);
            count_launch();
        }
        k_bjobs<<<grid_for(g), kThreads, 0, s>>>(uniq, cnts + kCntCols, kby, g, d_bp, d_ydup, d_acc);
        count_launch();
        GS_CUDA(cudaGetLastError());
        if (ny) {
            k_brank<<<grid_for(ny), kThreads, 0, s>>>(ykeys, ny, kby, d_bp, uniq, d_acc, rank);
            count_launch();
            GS_CUDA(cudaGetLastError());
        }
    }

    // ---- X match, row table and unit planning ----
    GS_CUDA(cudaStreamWaitEvent(s, ev[9], 0));
    join.sx = nullptr;
    if (wx) { xk0.release(); xv0.release(); } else { xk1.release(); xv1.release(); }
    if (keep) keep->xperm = wx ? std::move(xv1) : std::move(xv0);
    DBuf<uint32_t> pos(A, nxb, s), cnt(A, nxb, s);
    DBuf<uint64_t> xprefix(A, nx + 1, s);
    DBuf<uint32_t> row_start(A, nx + 1, s);
    DBuf<uint64_t> row_xf(A, nxb, s), row_prod(A, nxb, s);
    DBuf<uint16_t> row_job(A, nxb, s);
    DBuf<uint32_t> H(A, nxb, s), L(A, nxb, s), ustart(A, nx + 1, s), lk0(A, nx + 1, s), lrun(A, nxb, s), lrow(A, nxb, s);
    DBuf<uint64_t> lpre(A, nx + 1, s), loff(A, nxb, s);
    DBuf<uint32_t> mpre(A, nx + 1, s), mrun(A, nxb, s), row_xi(A, nxb, s), SR(A, nxb, s);
    DBuf<uint64_t> sprefix(A, nx + 1, s);
    DBuf<uint32_t> row_nnz(A, nxb, s);
    // heavy rows' kept column bitmaps: words of every heavy row and of the
    // dense ones only, their word offsets, each row's smallest rank
    const bool keep_bm = ctx->keep_row_bitmaps != 0;
    DBuf<uint32_t> bm_w_all, bm_w_dense, row_rb;
    DBuf<uint64_t> bm_off_all, bm_off_dense;
    DBuf<uint8_t> row_class;
    if (keep_bm) {
        bm_w_all.reset(A, nxb, s);
        bm_w_dense.reset(A, nxb, s);
        row_rb.reset(A, nxb, s);
        bm_off_all.reset(A, nxb, s);
        bm_off_dense.reset(A, nxb, s);
    }
    if (nx) {
        DBuf<uint8_t> rflag(A, nx, s);
        row_class.reset(A, nx, s);
        DBuf<uint32_t> mrow(A, nx, s), row_k0(A, nx + 1, s);
        k_bmatch<<<grid_for(nx), kThreads, 0, s>>>(xkeys, nx, kbx, kby, d_bp, run_key, run_start, cnts + kCntRuns,
                                                    ctab, pos, cnt, rflag);
        count_launch();
        GS_CUDA(cudaGetLastError());
        run_key.release();
        run_start.release();
        RowArrays ra{};
        ra.xprefix = xprefix;
        ra.mpre = mpre;
        ra.mrun = mrun;
        ra.mrow = mrow;
        ra.row_start = row_start;
        ra.row_k0 = row_k0;
        ra.row_xf = row_xf;
        ra.row_job = row_job;
        ra.row_prod = row_prod;
        ra.row_class = row_class;
        ra.row_nnz = row_nnz;
        ra.row_xi = row_xi;
        ra.H = H;
        ra.SR = SR;
        ra.L = L;
        ra.sprefix = sprefix;
        ra.lpre = lpre;
        ra.lk0 = lk0;
        ra.ustart = ustart;
        ra.lrun = lrun;
        ra.lrow = lrow;
        ra.loff = loff;
        DBuf<uint32_t> row_mx, longs;
        if (by_free && any_light) {
            longs.reset(A, nx / kOrderScan + 1, s);
            ra.longs = longs;
        }
        if (keep_bm) {
            row_mx.reset(A, nx, s);
            ra.row_rb = row_rb;
            ra.row_mx = row_mx;
        }
        launch_x_rows(xkeys, nx, kbx, d_bp, cnt, rflag, ra, cnts, scan_state(flags_x), s);
        xk0.release();
        xk1.release();
        if (any_wide)
            launch_wide_tables(reinterpret_cast<const WideTab *>(tabs.get() + o_wt), g, std::max(nx, ny), row_job, row_xf,
                               cols, d_acc, cnts, plan_err, s);
        const uint64_t *range = nullptr;
        if (nshards > 1) {
            k_shard_range<<<1, 32, 0, s>>>(xprefix, row_start, cnts + kCntRows, shard, nshards, cnts + kCntRange,
                                           plan_err);
            count_launch();
            GS_CUDA(cudaGetLastError());
            range = cnts + kCntRange;
        }
        launch_row_classes(nx, d_bp, d_acc, range, ra, cnts, scan_state(flags_x + zf_x), s);
        mark(3);
        launch_light_units(nx, light_bin, ra, cnts, scan_state(flags_x + 2 * zf_x), s);
        launch_matched_runs(nx, pos, cnt, rank, ra, cnts, plan_err, s);
        if (longs.get()) launch_light_order(nx, pos, cnt, ra, cnts, plan_err, ctx->sm_count, s);
        if (keep_bm)
            launch_heavy_bitmaps(nx, ra, bm_w_all, bm_w_dense, bm_off_all, bm_off_dense, cnts,
                                 scan_state(flags_x + 3 * zf_x), s);
    } else {
        GS_CUDA(cudaMemsetAsync(xprefix.get(), 0, 8, s));
        GS_CUDA(cudaMemsetAsync(mpre.get(), 0, 4, s));
        GS_CUDA(cudaMemsetAsync(row_start.get(), 0, 4, s));
        mark(3);
    }
    // counters and the jobs' error words, copied at once
    const size_t head_bytes = 8 * kCnts + 4 * (size_t)g;
    std::vector<uint8_t> h_head;
    uint8_t *head = static_cast<uint8_t *>(ctx->h_pin);
    if (!head || head_bytes > gsparc_ctx::kPinBytes) {
        h_head.resize(head_bytes);
        head = h_head.data();
    }
    d2h(head, reinterpret_cast<const uint8_t *>(zero.get()), head_bytes, s);
    GS_CUDA(cudaStreamSynchronize(s));
    uint64_t hc_cnt[kCnts];
    std::memcpy(hc_cnt, head, sizeof(hc_cnt));
    std::vector<unsigned int> jerr(g);
    std::memcpy(jerr.data(), head + sizeof(hc_cnt), 4 * (size_t)g);
    unsigned int herr = (unsigned int)hc_cnt[kCntErr];
    uint64_t ir = hc_cnt[kCntProducts];
    GS_REQUIRE(!(herr & kScanErr), GSPARC_EINTERNAL, kLookBackGaveUp);
    const uint64_t bm_words_all = hc_cnt[kCntBmAll], bm_words_dense = hc_cnt[kCntBmDense];
    const uint64_t nrows = hc_cnt[kCntRows], nh = hc_cnt[kCntHeavy], nl = hc_cnt[kCntLight],
                   nu = hc_cnt[kCntUnits], nsr = hc_cnt[kCntStream];
    if (nshards > 1) ir = hc_cnt[kCntRange + 2];  // the shard's products
    bst.ir_nnz += ir;
    bst.rows += nrows;
    bst.heavy_rows += nh;
    bst.stream_rows += nsr;

    // Narrow rows: units of about `slice` products (some 24 CTAs' worth an SM,
    // so that the last ones end together), their columns' marks and the partial
    // sums of rows of several units.  Where these do not fit a sixteenth of the
    // memory left, the windowed kernel takes the rows.
    const uint64_t slice = std::min<uint64_t>(std::max<uint64_t>(ir / ((uint64_t)ctx->sm_count * 24), kNarrowSlice),
                                              1ull << 20);
    const uint64_t narrow_cols = hc_cnt[kCntNarrowCols], nbm_words = hc_cnt[kCntNarrow] * (kNarrowCols / 32),
                   nparts = 2 * (ir / slice) * narrow_cols;
    // the output of the widest row, twice in two chunks, and the heavy rows'
    // cursors must fit beside what is optional
    const uint64_t out_need = 48 * hc_cnt[kCntCols] + 16 * nx + (1ull << 20);
    const auto fits = [&](uint64_t bytes, uint64_t part) {
        return bytes <= A.available() / part && bytes + out_need <= A.available();
    };
    const uint64_t nnarrow = fits(4 * nbm_words + 8 * nparts, 16) ? hc_cnt[kCntNarrow] : 0;
    const uint8_t *narrow_class = nnarrow ? row_class.get() : nullptr;

    // y_f of every Y entry for the heavy rows, where it fits 32 bits, the memory
    // allows, and rows past the light ones have a product for every entry
    DBuf<uint32_t> ycol;
    {
        int most = 0;
        for (Job *q : G)
            most = std::max(most, q->wide && q->key_words == 1 ? q->wide->nfbits_y : q->LY.nfbits);
        if (nh > nnarrow && most <= 32 && ir - hc_cnt[kCntLightProd] >= ny && fits(4 * ny, 16)) {
            ycol.reset(A, ny, s);
            launch_y_cols32(ykeys, ny, kby, d_acc, cols, rank, ycol, plan_err, s);
        }
    }

    // heavy rows largest first (H itself stays in row order for chunk planning)
    DBuf<uint32_t> H2;
    const uint32_t *Hs = H.get();
    if (nh > 1) {
        DBuf<uint8_t> hp0(A, nh, s), hp1(A, nh, s);
        H2.reset(A, nh, s);
        k_heavy_sizes<<<grid_for(nh), kThreads, 0, s>>>(H, nh, row_prod, narrow_class, hp0);
        count_launch();
        GS_CUDA(cudaGetLastError());
        size_t tmp = 0;
        GS_CUDA(cub::DeviceRadixSort::SortPairsDescending(nullptr, tmp, hp0.get(), hp1.get(), H.get(), H2.get(),
                                                          (int)nh, 0, 8, s));
        DBuf<uint8_t> t(A, tmp, s);
        GS_CUDA(cub::DeviceRadixSort::SortPairsDescending(t.get(), tmp, hp0.get(), hp1.get(), H.get(), H2.get(),
                                                          (int)nh, 0, 8, s));
        Hs = H2.get();
    }

    // ---- symbolic pass ----
    DBuf<uint32_t> cursor, pend;  // of the windowed kernel
    if (nh > nnarrow) {
        cursor.reset(A, nxb, s);
        pend.reset(A, nxb, s);
    }
    DBuf<uint64_t> row_off(A, nrows + 1, s);
    AccArgs aa{};
    aa.row_job = row_job;
    aa.jobs = d_acc;
    aa.row_start = row_start;
    aa.row_xf = row_xf;
    aa.pos = pos;
    aa.cnt = cnt;
    aa.xprefix = xprefix;
    aa.mpre = mpre;
    aa.mrun = mrun;
    aa.light_cap = (uint32_t)light_cap;
    aa.light_cols = hc_cnt[kCntCols];
    aa.ustart = ustart;
    aa.lk0 = lk0;
    aa.lrun = lrun;
    aa.lrow = lrow;
    aa.lpre = lpre;
    aa.loff = loff;
    // Light rows are merged once: the pass that counts their outputs writes them
    // to scratch, 12 B a product, which the chunks copy from; twice (the second
    // time in place) where that does not fit an eighth of the memory left, and
    // for plans, whose values change.
    const uint64_t light_prod = hc_cnt[kCntLightProd];
    const bool light_once = !keep && nu && fits(12 * light_prod, 8);
    DBuf<uint64_t> lout_keys, lpos;
    DBuf<float> lout_vals;
    if (light_once) {
        lout_keys.reset(A, light_prod, s);
        lout_vals.reset(A, light_prod, s);
        lpos.reset(A, nl, s);
        aa.lpos = lpos;
        aa.lout_keys = lout_keys;
        aa.lout_vals = lout_vals;
    }
    aa.xval = xvals;
    aa.yrank = rank;
    aa.yval = yvals;
    aa.ykeys = ykeys;
    aa.cols = cols;
    aa.any_wide = any_wide;
    aa.ycol = ycol.get() ? ycol.get() : rank.get();
    aa.col_is_key = ycol.get() != nullptr;
    aa.work_counter = ctx->d_flag + 1;
    aa.cursor = cursor;
    aa.pend = pend;
    aa.row_nnz = row_nnz;
    aa.row_off = row_off;
    aa.row_xi = row_xi;
    aa.err = ctx->d_flag;
    aa.heavy_cap = ctx->heavy_window_cap;
    DBuf<uint32_t> nbm, unit_off, part_off;
    DBuf<float2> part;
    if (nnarrow) {
        nbm.reset(A, nbm_words, s);
        unit_off.reset(A, nh + 1, s);
        part_off.reset(A, nh, s);
        part.reset(A, std::max<uint64_t>(nparts, 1), s);
        GS_CUDA(cudaMemsetAsync(nbm.get(), 0, 4 * nbm_words, s));
        launch_narrow_units(Hs, (uint32_t)nh, row_class, row_prod, slice, unit_off, part_off,
                            late_scan(flags_x + 4 * zf_x, 2), s);
        aa.row_class = row_class;
        aa.unit_off = unit_off;
        aa.part_off = part_off;
        aa.nbm = nbm;
        aa.part = part;
        aa.narrow_cols = (uint32_t)narrow_cols;
    }
    // Kept bitmaps take at most an eighth of the memory left (the rest is for
    // the output chunks): those of the heavy rows of at most kKeepBitsMax bits
    // per product if they fit, else of the dense rows (at most
    // kKeepBitsPerProduct), else none; the other heavy rows mark their windows.
    DBuf<uint32_t> hbm;
    DBuf<uint64_t> *bm_off = nullptr;
    if (keep_bm && nh) {
        const uint64_t room = A.available() / 8;
        if (bm_words_all && bm_words_all * 4 <= room)
            bm_off = &bm_off_all;
        else if (bm_words_dense && bm_words_dense * 4 <= room)
            bm_off = &bm_off_dense;
    }
    if (bm_off) {
        const uint64_t words = bm_off == &bm_off_all ? bm_words_all : bm_words_dense;
        hbm.reset(A, words, s);
        aa.hbm = hbm;
        aa.row_bmoff = *bm_off;
        aa.row_bmw = bm_off == &bm_off_all ? bm_w_all : bm_w_dense;
        aa.row_rb = row_rb;
        bst.kept_bitmap_bytes += words * 4;
    }
    if (bm_off != &bm_off_all) {
        bm_off_all.release();
        bm_w_all.release();
    }
    if (bm_off != &bm_off_dense) {
        bm_off_dense.release();
        bm_w_dense.release();
    }
    const int ghs = std::max(1, ctx->sm_count * heavy_blocks_per_sm(false));
    const int gh = std::max(1, ctx->sm_count * heavy_blocks_per_sm(true));
    const int gl = std::max(1, ctx->sm_count * light_blocks_per_sm());
    const int gs_grid = std::max(1, ctx->sm_count * stream_blocks_per_sm());
    {
        AccArgs b = aa;
        b.units = L;
        b.nunits = (uint32_t)nu;
        b.l0 = 0;
        b.l1 = (uint32_t)nl;
        b.work_counter = work;
        b.out_cap = light_prod;
        launch_light(b, light_once ? kLightValues : kLightCount,
                     (int)std::min<uint64_t>(gl, std::max<uint64_t>(1, nu)), s);
        b.units = Hs;
        b.nunits = (uint32_t)nh;
        if (nh > nnarrow) {
            b.work_counter = work + 1;
            launch_heavy(b, false, (int)std::min<uint64_t>(ghs, std::max<uint64_t>(1, nh)), s);
        }
        if (nnarrow) {
            b.work_counter = work + 2;
            launch_narrow(b, false, ctx->sm_count, s);
        }
    }
    launch_row_offsets(row_nnz, nrows, row_off, late_scan(flags_x + 6 * zf_x, 1), s);
    const UnitLists ul{L, nl, H, nh, SR, nsr};
    k_after_counts<<<grid_for(std::max<uint64_t>(nl + nh + nsr, (uint64_t)g + 1)), kThreads, 0, s>>>(
        ul, row_off, row_job, nrows, xprefix, d_xoffs, g, ctx->d_flag, d_jo);
    count_launch();
    GS_CUDA(cudaGetLastError());
    // What no later pass of this group reads goes back before the output is taken,
    // while the symbolic pass runs (between the readback and its launch the same
    // cost 4 us a call).  The planning's arrays are sized for a row an X nonzero, so
    // the output has more need of them: with all of them held, 6e5 rows beside a row
    // of 1e6 outputs needed 196 MB, now 162.
    row_nnz.release();
    aa.row_nnz = nullptr;
    if (!nl || light_once) {
        ustart.release();
        lk0.release();
        lrun.release();
        lrow.release();
        lpre.release();
        loff.release();
    }
    if (!nsr) {
        SR.release();
        sprefix.release();
        // single-run rows alone take y_f from the sorted keys
        yk0.release();
        yk1.release();
        if (keep) keep->ykeys.release();
        aa.ykeys = nullptr;
    }
    if (!nh) row_prod.release();
    if (!bm_off) row_rb.release();
    if (!nnarrow) {
        mpre.release();
        mrun.release();
        row_class.release();
    }
    std::vector<JobOut> jo(g + 2);
    const size_t jo_bytes = sizeof(JobOut) * (size_t)(g + 2);
    void *jo_at = ctx->h_pin && jo_bytes <= gsparc_ctx::kPinBytes ? ctx->h_pin : jo.data();
    d2h(static_cast<uint8_t *>(jo_at), reinterpret_cast<const uint8_t *>(d_jo), jo_bytes, s);
    GS_CUDA(cudaStreamSynchronize(s));
    if (jo_at != jo.data()) std::memcpy(jo.data(), jo_at, jo_bytes);
    const uint64_t max_unit = jo[g + 1].row0;
    herr = (unsigned int)jo[g + 1].out_off;
    bst.bytes_d2h += sizeof(JobOut) * (g + 1) + 64 + 4 * g + 8;
    GS_REQUIRE(!(herr & 2u), GSPARC_EINTERNAL, "light unit over capacity");
    GS_REQUIRE(!(herr & kScanErr), GSPARC_EINTERNAL, kLookBackGaveUp);
    const uint64_t ntot = jo[g].out_off;
    bst.nnz += ntot;
    mark(4);

    // per-job counts; jobs with an out-of-range index fail alone
    std::vector<uint64_t> job_nnz(g);
    for (int j = 0; j < g; ++j) {
        gsparc_job &J = *G[j]->job;
        gsparc_stats &st = J.stats;
        st.ir_nnz = nshards > 1 ? ir : jo[j + 1].ir_off - jo[j].ir_off;
        st.nnz = jo[j + 1].out_off - jo[j].out_off;
        st.rows = jo[j + 1].row0 - jo[j].row0;
        st.heavy_rows = jo[j + 1].heavy0 - jo[j].heavy0;
        job_nnz[j] = st.nnz;
        if (jerr[j] & 1u) {
            J.status = GSPARC_EINVAL;
            set_last_error("an index is not smaller than its mode size");
        }
    }

    // ---- chunk plan (memory-aware partitioning of the output) ----
    // Units (light units, heavy rows) tile the output in row order.  A chunk
    // takes the units that start in [k*C, (k+1)*C) of the output; with units
    // of at most max_unit outputs and C >= max_unit every chunk is non-empty
    // and holds fewer than C + max_unit <= cap outputs.
    // a chunk's output buffers (two when chunks overlap delivery) must fit
    // the memory left; the caller's max_chunk_nnz can only lower that
    uint64_t cap = std::min<uint64_t>(A.available() / 3 / 12, 1ull << 31);
    if (max_chunk_nnz) cap = std::min(cap, max_chunk_nnz);
    cap = std::max<uint64_t>(cap, 1);
    struct Chunk {
        uint64_t lu0, lu1;  // light rows [lu0, lu1)
        uint64_t h0, h1;    // heavy rows [h0, h1) of the chunk-grouped heavy list
        uint64_t s0, s1;    // stream rows [s0, s1)
        uint64_t first, n;
    };
    std::vector<Chunk> chunks;
    DBuf<uint32_t> Hc;  // heavy rows grouped by chunk, largest first inside a chunk
    const uint32_t *Hchunk = Hs;
    // Jobs that complete one by one get chunk cuts at job boundaries after
    // kFirstCutProducts, 2x that, 4x that, ... products.
    const bool progressive = done_fn && g > 1 && ntot > 0;
    if (ntot <= cap && !progressive) {
        if (ntot || nl || nh || nsr) chunks.push_back({0, nl, 0, nh, 0, nsr, 0, ntot});
    } else {
        uint64_t C = std::max(cap > max_unit ? cap - max_unit : 1, std::max<uint64_t>(max_unit, 1));
        C = std::max<uint64_t>(C, (ntot + (1ull << 20) - 1) >> 20);  // at most 2^20 uniform chunks
        GS_REQUIRE(2 * 12 * (C + max_unit) <= A.available(), GSPARC_ENOMEM,
                   "one output row does not fit the HBM budget");
        std::vector<uint64_t> target{0};
        if (!progressive) {
            for (uint64_t t = C; t < ntot; t += C) target.push_back(t);
        } else {
            uint64_t acc = 0, thr = kFirstCutProducts;
            for (int j = 0; j < g; ++j) {
                const uint64_t end = jo[j + 1].out_off;
                while (end - target.back() > C) target.push_back(target.back() + C);
                acc += jo[j + 1].ir_off - jo[j].ir_off;
                if (acc >= thr && j + 1 < g && end > target.back() && end < ntot) {
                    target.push_back(end);
                    acc = 0;
                    thr *= 2;
                }
            }
        }
        target.push_back(ntot);
        const uint64_t K = target.size() - 1;
        const uint64_t M = nl + nh + nsr;
        DBuf<uint32_t> urow(A, M, s);
        DBuf<uint64_t> uoff(A, M, s);
        k_merge_starts<<<grid_for(M), kThreads, 0, s>>>(ul, row_off, urow, uoff);
        count_launch();
        GS_CUDA(cudaGetLastError());
        DBuf<uint64_t> d_target(A, K + 1, s);
        h2d(d_target.get(), target.data(), K + 1, s);
        DBuf<uint64_t> cinfo(A, kChunkInfo * (K + 1), s);
        k_chunk_bounds<<<grid_for(K + 1), kThreads, 0, s>>>(urow, uoff, M, d_target, K, ul, nrows, ntot, cinfo);
        count_launch();
        GS_CUDA(cudaGetLastError());
        std::vector<uint64_t> ci(kChunkInfo * (K + 1));
        d2h(ci.data(), cinfo.get(), kChunkInfo * (K + 1), s);
        if (nh) {
            // heavy rows grouped by chunk (stable in the largest-first order)
            DBuf<uint64_t> hk0(A, nh, s), hk1(A, nh, s);
            Hc.reset(A, nh, s);
            k_heavy_chunk_keys<<<grid_for(nh), kThreads, 0, s>>>(Hs, nh, row_prod, aa.row_class, cinfo, K, hk0);
            count_launch();
            GS_CUDA(cudaGetLastError());
            const int bits = kChunkProdBits + 1 + ceil_log2(K);
            GS_REQUIRE(bits <= 64, GSPARC_EINTERNAL, "too many output chunks");
            size_t tmp = 0;
            GS_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tmp, hk0.get(), hk1.get(), Hs, Hc.get(), (int)nh, 0,
                                                    bits, s));
            DBuf<uint8_t> t(A, tmp, s);
            GS_CUDA(cub::DeviceRadixSort::SortPairs(t.get(), tmp, hk0.get(), hk1.get(), Hs, Hc.get(), (int)nh, 0,
                                                    bits, s));
            Hchunk = Hc.get();
        }
        GS_CUDA(cudaStreamSynchronize(s));
        bst.bytes_d2h += 8 * kChunkInfo * (K + 1);
        for (uint64_t k = 0; k < K; ++k) {
            const uint64_t *a = &ci[kChunkInfo * k], *b = &ci[kChunkInfo * (k + 1)];
            if (b[1] > a[1]) chunks.push_back({a[2], b[2], a[3], b[3], a[4], b[4], a[1], b[1] - a[1]});
        }
    }
    bst.chunks += chunks.size();
    if (nnarrow && Hchunk != Hs)  // the chunks' own order
        launch_narrow_units(Hchunk, (uint32_t)nh, row_class, row_prod, slice, unit_off, part_off,
                            late_scan(flags_x + 5 * zf_x, 3), s);
    row_prod.release();

    if (keep) {
        // a plan keeps what the numeric pass needs, in arrays of the sizes that
        // turned out (a copy each, where the memory has room for it), and stops here
        const auto fit = [&](auto &b, uint64_t n, auto &at) {
            using T = std::remove_reference_t<decltype(*b.get())>;
            n = std::max<uint64_t>(n, 1);
            if (b.size() <= n || sizeof(T) * n + 256 > A.available()) return;
            std::remove_reference_t<decltype(b)> c(A, n, s);
            GS_CUDA(cudaMemcpyAsync(c.get(), b.get(), sizeof(T) * n, cudaMemcpyDeviceToDevice, s));
            b = std::move(c);
            at = b.get();
        };
        if (Hc.get()) H2.release();  // the list that heavy_list() takes
        if (Hc.get() || H2.get()) H.release();
        const uint32_t *list = nullptr;  // the lists' addresses are taken when a chunk is launched
        fit(L, nl, list);
        fit(H, nh, list);
        fit(SR, nsr, list);
        const uint64_t *pre = nullptr;
        fit(sprefix, nsr + 1, pre);
        fit(ustart, nu + 1, aa.ustart);
        fit(lk0, nl + 1, aa.lk0);
        fit(lpre, nl + 1, aa.lpre);
        fit(lrun, hc_cnt[kCntLightRuns], aa.lrun);
        fit(lrow, hc_cnt[kCntLightRuns], aa.lrow);
        fit(loff, hc_cnt[kCntLightRuns], aa.loff);
        fit(row_start, nrows + 1, aa.row_start);
        fit(row_xf, nrows, aa.row_xf);
        fit(row_job, nrows, aa.row_job);
        fit(row_xi, nrows, aa.row_xi);
        if (aa.col_is_key && !nl && !nnarrow && !any_wide)
            cols.release();  // no row looks a column up
        else
            fit(cols, hc_cnt[kCntCols], aa.cols);
        if (nnarrow) fit(row_class, nrows, aa.row_class);
        if (bm_off) {
            fit(row_rb, nrows, aa.row_rb);
            fit(*bm_off, nrows, aa.row_bmoff);
            fit(bm_off == &bm_off_all ? bm_w_all : bm_w_dense, nrows, aa.row_bmw);
        }
        keep->g = g;
        keep->nx = nx;
        keep->ny = ny;
        keep->ntot = ntot;
        keep->nu = nu;
        keep->nh = nh;
        keep->nsr = nsr;
        keep->gl = gl;
        keep->gh = gh;
        keep->gs_grid = gs_grid;
        keep->job_first.resize(g + 1);
        for (int j = 0; j <= g; ++j) keep->job_first[j] = jo[j].out_off;
        keep->jobs = G;
        keep->d_lx = d_lx;  // in tabs
        keep->d_ly = d_ly;
        keep->d_xoffs = d_xoffs;
        keep->d_yoffs = d_yoffs;
        keep->tabs = std::move(tabs);
        keep->d_acc = std::move(d_acc);
        keep->rank = std::move(rank);
        keep->ycol = std::move(ycol);
        keep->pos = std::move(pos);
        keep->cnt = std::move(cnt);
        keep->mpre = std::move(mpre);
        keep->mrun = std::move(mrun);
        keep->ustart = std::move(ustart);
        keep->lk0 = std::move(lk0);
        keep->lrun = std::move(lrun);
        keep->lrow = std::move(lrow);
        keep->lpre = std::move(lpre);
        keep->loff = std::move(loff);
        keep->row_start = std::move(row_start);
        keep->L = std::move(L);
        keep->H = std::move(H);
        keep->H2 = std::move(H2);
        keep->SR = std::move(SR);
        keep->row_xi = std::move(row_xi);
        keep->cursor = std::move(cursor);
        keep->pend = std::move(pend);
        keep->cols = std::move(cols);
        keep->xprefix = std::move(xprefix);
        keep->row_xf = std::move(row_xf);
        keep->sprefix = std::move(sprefix);
        keep->row_off = std::move(row_off);
        keep->row_job = std::move(row_job);
        keep->Hc = std::move(Hc);
        if (bm_off) {  // kept bitmaps are part of what the numeric pass reads
            keep->hbm = std::move(hbm);
            keep->row_rb = std::move(row_rb);
            keep->row_bmoff = std::move(*bm_off);
            keep->row_bmw = std::move(bm_off == &bm_off_all ? bm_w_all : bm_w_dense);
        }
        keep->chunks.clear();
        for (auto &c : chunks) keep->chunks.push_back({c.lu0, c.lu1, c.h0, c.h1, c.s0, c.s1, c.first, c.n});
        if (nnarrow) {
            keep->nnarrow = nnarrow;
            keep->nbm = std::move(nbm);
            keep->unit_off = std::move(unit_off);
            keep->part_off = std::move(part_off);
            keep->part = std::move(part);
            keep->row_class = std::move(row_class);
        }
        keep->sm_count = ctx->sm_count;
        keep->flags.reset(A, 4, s);
        GS_CUDA(cudaMemsetAsync(keep->flags.get(), 0, 16, s));
        keep->aa = aa;  // the moved buffers keep their device addresses
        keep->aa.err = keep->flags.get();
        keep->aa.work_counter = keep->flags.get() + 1;
        unsigned int e = 0;
        d2h(&e, ctx->d_flag, 1, s);
        GS_CUDA(cudaStreamSynchronize(s));
        GS_REQUIRE(!(e & kScanErr), GSPARC_EINTERNAL, kLookBackGaveUp);
        tm.total += planning_times();
        return;
    }

    // ---- numeric pass, chunk by chunk, double-buffered against delivery ----
    const int nbuf = chunks.size() > 1 ? 2 : 1;
    uint64_t bufn = 0;
    for (auto &c : chunks) bufn = std::max(bufn, c.n);
    DBuf<uint64_t> out_k[2];
    DBuf<float> out_v[2];
    DBuf<uint64_t> out_k2[2];  // 128-bit keys of jobs whose sink asks for two key words
    bool any_kw2 = false;
    for (Job *q : G) any_kw2 |= q->key_words == 2;
    for (int i = 0; i < nbuf; ++i) {
        out_k[i].reset(A, std::max<uint64_t>(bufn, 1), s);
        out_v[i].reset(A, std::max<uint64_t>(bufn, 1), s);
        if (any_kw2) out_k2[i].reset(A, 2 * std::max<uint64_t>(bufn, 1), s);
    }
    std::vector<cudaEvent_t> kev(2 * chunks.size(), nullptr);
    for (auto &e : kev) GS_CUDA(cudaEventCreate(&e));
    cudaStream_t s2 = ctx->copy_stream;

    // FP64 verification of every chunk before delivery (off unless asked for)
    const bool verify = ctx->verify_budget != 0 && nrows > 0 && ntot > 0;
    VerifyState vs;
    DBuf<VerifyEntry> v_list;
    DBuf<unsigned long long> v_cnt;
    DBuf<double> v_acc;
    DBuf<VerifyOut> v_out;
    if (verify) {
        v_list.reset(A, nrows, s);
        v_cnt.reset(A, 2, s);
        v_out.reset(A, g, s);
        GS_CUDA(cudaMemsetAsync(v_out.get(), 0, sizeof(VerifyOut) * g, s));
        uint64_t cap = std::min<uint64_t>(bufn, 1ull << 25);
        cap = std::max<uint64_t>(1, std::min<uint64_t>(cap, A.available() / 2 / sizeof(double)));
        v_acc.reset(A, cap, s);
        vs.list = v_list.get();
        vs.cnt = v_cnt.get();
        vs.acc = v_acc.get();
        vs.acc_cap = cap;
        vs.out = v_out.get();
        vs.threshold = verify_threshold(ctx->verify_budget, ir);
        vs.salt = 0x5eed5eed5eedull;
        GS_CUDA(cudaStreamSynchronize(s));
    }
    double t_out = 0;
    std::vector<uint64_t> job_first(g + 1);
    for (int j = 0; j <= g; ++j) job_first[j] = jo[j].out_off;
    int next_done = 0;  // jobs before it were reported complete

    // Consecutive chunks go to two streams, so the next chunk's kernels start
    // on SMs the current chunk's kernels leave idle at their tails.  Each
    // stream has its own work counter; the buffer a chunk writes was delivered
    // (host-synchronously) before it is enqueued.  A device sink may enqueue
    // its own copies of a chunk on the engine's stream, which only orders them
    // before later chunks on that stream: groups with one stay on one stream.
    bool device_sink = false;
    for (Job *q : G) device_sink |= q->job->sink.kind == GSPARC_SINK_DEVICE;
    cudaStream_t sa = ctx->alt_stream && !device_sink && chunks.size() > 1 ? ctx->alt_stream : s;
    cudaEvent_t ev_ready = nullptr, ev_alt = nullptr;
    GS_CUDA(cudaEventCreateWithFlags(&ev_ready, cudaEventDisableTiming));
    GS_CUDA(cudaEventCreateWithFlags(&ev_alt, cudaEventDisableTiming));
    GS_CUDA(cudaEventRecord(ev_ready, s));
    GS_CUDA(cudaStreamWaitEvent(sa, ev_ready, 0));
    auto enqueue = [&](size_t ci) {
        const Chunk &c = chunks[ci];
        const int bi = (int)(ci % nbuf);
        const cudaStream_t sc = (ci & 1) ? sa : s;
        unsigned int *counter = ctx->d_flag + ((ci & 1) && sa != s ? 5 : 1);
        AccArgs b = aa;
        // the first chunk has counters of its own, cleared with the rest
        const auto next_counter = [&](int k) {
            b.work_counter = ci == 0 ? work + 3 + k : counter;
            if (ci) GS_CUDA(cudaMemsetAsync(counter, 0, 4, sc));
        };
        b.chunk_base = c.first;
        b.out_keys = out_k[bi];
        b.out_vals = out_v[bi];
        b.out_cap = c.n;
        b.units = L;
        b.nunits = (uint32_t)nu;
        b.l0 = (uint32_t)c.lu0;
        b.l1 = (uint32_t)c.lu1;
        next_counter(0);
        GS_CUDA(cudaEventRecord(kev[2 * ci], sc));
        if (light_once) {
            launch_light_copy(b, ctx->sm_count, sc);
        } else {
            launch_light(b, kLightFinal, (int)std::min<uint64_t>(gl, std::max<uint64_t>(1, nu)), sc);
        }
        b.units = Hchunk + c.h0;
        b.nunits = (uint32_t)(c.h1 - c.h0);
        if (nh > nnarrow) {
            next_counter(1);
            launch_heavy(b, true, (int)std::min<uint64_t>(gh, std::max<uint64_t>(1, b.nunits)), sc);
        }
        if (nnarrow) {
            b.unit_off += c.h0;
            b.part_off += c.h0;
            next_counter(2);
            launch_narrow(b, true, ctx->sm_count, sc);
        }
        b.units = SR.get() + c.s0;
        b.nunits = (uint32_t)(c.s1 - c.s0);
        b.sprefix = sprefix.get() + c.s0;
        launch_stream(b, gs_grid, sc);
        GS_CUDA(cudaEventRecord(kev[2 * ci + 1], sc));
    };
    auto deliver = [&](size_t ci) {
        const Chunk &c = chunks[ci];
        const int bi = (int)(ci % nbuf);
        auto t0 = std::chrono::steady_clock::now();
        GS_CUDA(cudaStreamWaitEvent(s2, kev[2 * ci + 1], 0));
        GS_CUDA(cudaEventSynchronize(kev[2 * ci + 1]));
        const uint64_t c0 = c.first, c1 = c.first + c.n;
        if (verify) {
            // before any wide-key remap: the chunk still holds the engine's keys
            verify_chunk(aa, vs, nrows, c0, c1, out_k[bi].get(), out_v[bi].get(), s2);
            GS_CUDA(cudaStreamSynchronize(s2));  // the buffer is rewritten two chunks on
        }
        // jobs overlapping [c0, c1)
        int j = (int)(std::upper_bound(job_first.begin(), job_first.end(), c0) - job_first.begin()) - 1;
        for (j = std::max(j, 0); j < g && job_first[j] < c1; ++j) {
            gsparc_job &J = *G[j]->job;
            const uint64_t a0 = std::max(c0, job_first[j]), a1 = std::min(c1, job_first[j + 1]);
            if (a1 <= a0 || J.status != GSPARC_OK) continue;
            if (G[j]->wide && G[j]->key_words == 2) {
                // relabeled output keys back to x_f << Y_nfbits | y_f in 128 bits
                uint64_t *k2 = out_k2[bi].get() + 2 * (a0 - c0);
                wide_remap_keys128(*G[j]->wide, out_k[bi].get() + (a0 - c0), k2, a1 - a0, s2);
                GS_CUDA(cudaStreamSynchronize(s2));
                deliver_slice(J.sink, k2, out_v[bi].get() + (a0 - c0), a1 - a0, a0 - job_first[j], job_nnz[j],
                              s2, J.stats, bst.bytes_d2h, 2);
                continue;
            }
            deliver_slice(J.sink, out_k[bi].get() + (a0 - c0), out_v[bi].get() + (a0 - c0), a1 - a0,
                          a0 - job_first[j], job_nnz[j], s2, J.stats, bst.bytes_d2h);
        }
        t_out += std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
        // jobs whose whole output is now delivered are complete (unless a
        // device-side check of the chunk failed)
        if (done_fn && next_done < g && job_first[next_done + 1] <= c1) {
            unsigned int e = 0;
            d2h(&e, ctx->d_flag, 1, s2);
            GS_CUDA(cudaStreamSynchronize(s2));
            GS_REQUIRE(!(e & (6u | kScanErr)), GSPARC_EINTERNAL, "numeric pass failed a device-side check");
        }
        if (done_fn)
            for (; next_done < g && job_first[next_done + 1] <= c1; ++next_done) {
                Job *q = G[next_done];
                if (!q->done && q->job->status == GSPARC_OK) {
                    q->done = true;
                    (*done_fn)(q->job);
                }
            }
    };
    try {
        for (size_t ci = 0; ci < chunks.size(); ++ci) {
            enqueue(ci);
            if (ci >= 1) deliver(ci - 1);
        }
        if (!chunks.empty()) deliver(chunks.size() - 1);
    } catch (...) {
        cudaStreamSynchronize(s2);
        cudaStreamSynchronize(sa);
        cudaStreamSynchronize(s);
        for (auto e : kev) cudaEventDestroy(e);
        cudaEventDestroy(ev_ready);
        cudaEventDestroy(ev_alt);
        throw;
    }
    GS_CUDA(cudaEventRecord(ev_alt, sa));
    GS_CUDA(cudaStreamWaitEvent(s, ev_alt, 0));
    cudaEventDestroy(ev_ready);
    cudaEventDestroy(ev_alt);
    if (verify) {
        std::vector<VerifyOut> vo(g);
        d2h(vo.data(), v_out.get(), g, s2);
        GS_CUDA(cudaStreamSynchronize(s2));
        for (int j = 0; j < g; ++j) {
            verify_fill_stats(vo[j], G[j]->job->stats);
            verify_fill_stats(vo[j], bst);
        }
    }
    mark(5);
    unsigned int hflags_own[4] = {0, 0, 0, 0};
    unsigned int *hflags = ctx->h_pin ? static_cast<unsigned int *>(ctx->h_pin) : hflags_own;
    d2h(hflags, ctx->d_flag, 4, s);
    GS_CUDA(cudaStreamSynchronize(s));
    bst.heavy_windows += hflags[2];
    GS_REQUIRE(!(hflags[0] & 2u), GSPARC_EINTERNAL, "light unit over capacity");
    GS_REQUIRE(!(hflags[0] & kScanErr), GSPARC_EINTERNAL, kLookBackGaveUp);
    GS_REQUIRE(!(hflags[0] & 4u), GSPARC_EINTERNAL, "numeric pass wrote past its chunk (symbolic count mismatch)");
    const double planned = planning_times(), end = at(5);
    tm.contract += end - planned;
    tm.total += end;
    tm.out += t_out;
    // numeric kernel time: first chunk's start to the last chunk's end (chunks
    // on the two streams overlap)
    {
        float span = 0.f;
        for (size_t i = 0; i + 1 < kev.size(); i += 2) {
            float t = 0.f;
            GS_CUDA(cudaEventElapsedTime(&t, kev[0], kev[i + 1]));
            span = std::max(span, t);
        }
        tm.numeric += span;
    }
    for (auto e : kev) cudaEventDestroy(e);
}

}  // namespace

// Checks every job on its own (a bad job fails alone: its status says why)
// and prepares the ones that pass: layouts, relabeling of keys over 64 bits.
void validate_jobs(gsparc_ctx *ctx, gsparc_job *jobs, int njobs, cudaStream_t s, std::vector<Job> &js,
                   gsparc_stats &bst) {
    js.reserve(njobs);
    for (int i = 0; i < njobs; ++i) {
        gsparc_job &J = jobs[i];
        std::memset(&J.stats, 0, sizeof(J.stats));
        J.status = GSPARC_OK;
        try {
            GS_REQUIRE(J.x && J.y, GSPARC_EINVAL, "null tensor");
            GS_REQUIRE(J.ncmodes >= 1 && J.ncmodes <= kMaxOrder && J.cx && J.cy, GSPARC_EINVAL, "bad contract modes");
            GS_REQUIRE(J.accum >= -1 && J.accum <= 1, GSPARC_EINVAL, "accum must be -1, 0 or 1");
            const gsparc_sink &k = J.sink;
            GS_REQUIRE(k.kind >= GSPARC_SINK_DISCARD && k.kind <= GSPARC_SINK_HOST, GSPARC_EINVAL, "bad sink kind");
            GS_REQUIRE(k.kind != GSPARC_SINK_HOST || (k.host_keys && k.host_vals && k.host_capacity), GSPARC_EINVAL,
                       "host sink needs host_keys, host_vals and host_capacity");
            GS_REQUIRE(k.kind != GSPARC_SINK_DEVICE || k.on_chunk, GSPARC_EINVAL, "device sink needs on_chunk");
            Job q;
            q.job = &J;
            q.tx = J.x;
            q.ty = J.y;
            q.LX = make_layout(J.x->order, J.x->dims, J.ncmodes, J.cx);
            q.LY = make_layout(J.y->order, J.y->dims, J.ncmodes, J.cy);
            GS_REQUIRE(J.x->order > J.ncmodes && J.y->order > J.ncmodes, GSPARC_EUNSUPPORTED,
                       "every operand needs at least one free mode");
            for (int m = 0; m < J.ncmodes; ++m)
                GS_REQUIRE(q.LX.bits[J.cx[m]] == q.LY.bits[J.cy[m]], GSPARC_EINVAL,
                           "contract modes of X and Y have different bit widths (mode sizes differ)");
            // a discarded output of more than 64 bits needs no key words at all:
            // run it on the 128-bit path and deliver nothing
            q.key_words = k.key_words ? k.key_words
                                      : (k.kind == GSPARC_SINK_DISCARD && q.LX.nfbits + q.LY.nfbits > 64 ? 2 : 1);
            GS_REQUIRE(q.key_words == 1 || q.key_words == 2, GSPARC_EINVAL, "sink key_words must be 0, 1 or 2");
            GS_REQUIRE(q.LX.nfbits + q.LY.nfbits <= 64 * q.key_words, GSPARC_EUNSUPPORTED,
                       "output key wider than 64 bits (X free bits + Y free bits > 64): set sink.key_words = 2");
            GS_REQUIRE(J.x->nnz < kMaxGroupNnz && J.y->nnz < kMaxGroupNnz, GSPARC_EUNSUPPORTED,
                       "operand with more than 2^31 nonzeros");
            const Layout LX0 = q.LX, LY0 = q.LY;
            if (q.LX.nbits() > 64 || q.LY.nbits() > 64 || q.key_words == 2) {
                // the reference's 128-bit key path: relabel onto 64-bit keys (128-bit
                // output keys are built from the rank tables at delivery)
                q.wide = make_wide(ctx->arena, J.x, q.LX, J.y, q.LY, s);
                q.tx = &q.wide->x2;
                q.ty = &q.wide->y2;
                q.LX = make_layout(2, q.tx->dims, 1, q.wide->cx2);
                q.LY = make_layout(2, q.ty->dims, 1, q.wide->cy2);
            }
            q.light_max = J.accum == GSPARC_ACCUM_DENSE ? 0 : (ctx->light_row_max ? ctx->light_row_max : kLightRowMax);
            q.width = std::max(q.LX.nbits(), q.LY.nbits());
            J.stats.nnz_x = J.x->nnz;
            J.stats.nnz_y = J.y->nnz;
            J.stats.nbits_x = LX0.nbits();
            J.stats.nbits_y = LY0.nbits();
            J.stats.ncbits = LX0.ncbits;
            J.stats.nfbits_x = LX0.nfbits;
            J.stats.nfbits_y = LY0.nfbits;
            J.stats.accumulator = J.accum;
            bst.nnz_x += J.x->nnz;
            bst.nnz_y += J.y->nnz;
            js.push_back(q);
        } catch (const Error &e) {
            J.status = e.st;
            set_last_error(e.msg);
        }
    }

}

// Groups of jobs whose keys, with the job id above them, fit 64 bits: widest
// keys first; a group of n jobs needs ceil(log2 n) id bits.
std::vector<std::vector<Job *>> make_groups(std::vector<Job> &js) {
    std::vector<Job *> order;
    for (auto &q : js) order.push_back(&q);
    std::stable_sort(order.begin(), order.end(), [](const Job *a, const Job *b) { return a->width > b->width; });
    std::vector<std::vector<Job *>> groups;
    {
        size_t i = 0;
        while (i < order.size()) {
            std::vector<Job *> G;
            uint64_t sx = 0, sy = 0;
            const int w = order[i]->width;  // widest of the group (sorted descending)
            while (i < order.size()) {
                Job *q = order[i];
                const uint64_t n1 = G.size() + 1;
                if (!G.empty() && (w + ceil_log2(n1) > 64 || (int)n1 > kMaxGroupJobs ||
                                   sx + q->job->x->nnz > kMaxGroupNnz || sy + q->job->y->nnz > kMaxGroupNnz))
                    break;
                G.push_back(q);
                sx += q->job->x->nnz;
                sy += q->job->y->nnz;
                ++i;
            }
            groups.push_back(std::move(G));
        }
    }

    return groups;
}

void sptc_batch(gsparc_ctx *ctx, gsparc_job *jobs, int njobs, uint64_t max_chunk_nnz, gsparc_stats *st_out,
                cudaStream_t s, int shard, int nshards, const JobDoneFn *done_fn) {
    GS_REQUIRE(ctx, GSPARC_EINVAL, "null context");
    GS_REQUIRE(njobs >= 0 && (njobs == 0 || jobs), GSPARC_EINVAL, "bad job array");
    GS_REQUIRE(nshards >= 1 && shard >= 0 && shard < nshards, GSPARC_EINVAL, "bad shard");
    GS_REQUIRE(nshards == 1 || njobs == 1, GSPARC_EINVAL, "row shards apply to a single contraction");
    gsparc_stats bst;
    std::memset(&bst, 0, sizeof(bst));
    const uint64_t launches0 = launch_count();

    std::vector<Job> js;
    validate_jobs(ctx, jobs, njobs, s, js, bst);
    std::vector<std::vector<Job *>> groups = make_groups(js);

    // completion reports: at most one per job, early ones from run_group
    std::vector<char> reported(njobs, 0);
    JobDoneFn report;
    const JobDoneFn *report_fn = nullptr;
    if (done_fn) {
        report = [&](gsparc_job *J) {
            reported[J - jobs] = 1;
            (*done_fn)(J);
        };
        report_fn = &report;
    }

    Times tm;
    for (auto &G : groups) {
        try {
            run_group(ctx, G, max_chunk_nnz, shard, nshards, tm, bst, s, report_fn);
        } catch (const Error &e) {
            // the group's jobs fail together (except those already complete);
            // later groups still run
            for (Job *q : G)
                if (!q->done && q->job->status == GSPARC_OK) q->job->status = e.st;
            set_last_error(e.msg);
            cudaStreamSynchronize(s);
        }
    }

    bst.t_linearize_ms = tm.lin;
    bst.t_sort_ms = tm.sort;
    bst.t_match_ms = tm.match;
    bst.t_plan_ms = tm.plan;
    bst.t_contract_ms = tm.contract;
    bst.t_output_ms = tm.out;
    bst.t_total_ms = tm.total;
    bst.t_numeric_kernel_ms = tm.numeric;
    bst.kernel_launches = launch_count() - launches0;
    bst.accumulator = GSPARC_ACCUM_AUTO;
    for (int i = 0; i < njobs; ++i) {
        gsparc_stats &st = jobs[i].stats;
        st.t_linearize_ms = tm.lin;
        st.t_sort_ms = tm.sort;
        st.t_match_ms = tm.match;
        st.t_plan_ms = tm.plan;
        st.t_contract_ms = tm.contract;
        st.t_output_ms = tm.out;
        st.t_total_ms = tm.total;
    }
    if (st_out) *st_out = bst;
    if (done_fn)
        for (int i = 0; i < njobs; ++i)
            if (!reported[i]) (*done_fn)(&jobs[i]);
    for (int i = 0; i < njobs; ++i)
        if (jobs[i].status != GSPARC_OK) {
            if (njobs == 1) fail(jobs[i].status, last_error());
            fail(jobs[i].status, std::string("job ") + std::to_string(i) + " failed (" +
                                     gsparc_status_string(jobs[i].status) + "); last message: " + last_error());
        }
}

}  // namespace gs

// ---- plans: the coordinate-only work done once, the numeric pass replayed ----

struct gsparc_plan {
    gsparc_ctx *ctx = nullptr;
    std::vector<gsparc_job> jobs;  // copies of the caller's jobs (modes copied too)
    std::vector<std::vector<int>> modes;
    std::vector<gs::Job> js;
    std::vector<std::unique_ptr<gs::GroupPlan>> groups;
    std::vector<uint64_t> group_off;               // first output of each group
    std::vector<std::pair<int, int>> chunk_of;     // plan chunk -> (group, group chunk)
    std::vector<uint64_t> job_first, job_nnz;      // per caller job
    uint64_t total = 0;
};

namespace gs {

void plan_create(gsparc_ctx *ctx, const gsparc_job *jobs, int njobs, uint64_t max_chunk_nnz, gsparc_plan **out,
                 uint64_t *total, cudaStream_t s) {
    GS_REQUIRE(ctx && out && njobs >= 1 && jobs, GSPARC_EINVAL, "bad argument");
    *out = nullptr;
    auto P = std::make_unique<gsparc_plan>();
    P->ctx = ctx;
    P->jobs.assign(jobs, jobs + njobs);
    P->modes.resize(njobs);
    for (int i = 0; i < njobs; ++i) {
        gsparc_job &J = P->jobs[i];
        GS_REQUIRE(J.ncmodes >= 1 && J.ncmodes <= kMaxOrder && J.cx && J.cy, GSPARC_EINVAL, "bad contract modes");
        auto &m = P->modes[i];
        m.assign(J.cx, J.cx + J.ncmodes);
        m.insert(m.end(), J.cy, J.cy + J.ncmodes);
        J.cx = m.data();
        J.cy = m.data() + J.ncmodes;
        J.sink = gsparc_sink{};
        J.sink.kind = GSPARC_SINK_DISCARD;
    }
    gsparc_stats bst;
    std::memset(&bst, 0, sizeof(bst));
    validate_jobs(ctx, P->jobs.data(), njobs, s, P->js, bst);
    for (int i = 0; i < njobs; ++i)
        if (P->jobs[i].status != GSPARC_OK)
            fail(P->jobs[i].status, "job " + std::to_string(i) + ": " + last_error());
    std::vector<std::vector<Job *>> groups = make_groups(P->js);
    Times tm;
    P->job_first.assign(njobs, 0);
    P->job_nnz.assign(njobs, 0);
    for (auto &G : groups) {
        auto gp = std::make_unique<GroupPlan>();
        run_group(ctx, G, max_chunk_nnz, 0, 1, tm, bst, s, nullptr, gp.get());
        for (Job *q : G)
            if (q->job->status != GSPARC_OK) fail(q->job->status, last_error());
        P->group_off.push_back(P->total);
        for (size_t c = 0; c < gp->chunks.size(); ++c) P->chunk_of.push_back({(int)P->groups.size(), (int)c});
        for (int j = 0; j < gp->g; ++j) {
            const int i = (int)(gp->jobs[j]->job - P->jobs.data());
            P->job_first[i] = P->total + gp->job_first[j];
            P->job_nnz[i] = gp->job_first[j + 1] - gp->job_first[j];
        }
        P->total += gp->ntot;
        P->groups.push_back(std::move(gp));
    }
    if (total) *total = P->total;
    *out = P.release();
}

// One chunk of a plan's output into keys/vals (first = the chunk's first
// output).  Launches only: memsets, value gathers, the numeric kernels and
// (for jobs with keys over 64 bits) the output key map.
void plan_execute(gsparc_plan *P, uint64_t chunk, uint64_t *keys, float *vals, uint64_t capacity,
                  cudaStream_t s) {
    GS_REQUIRE(P && chunk < P->chunk_of.size(), GSPARC_EINVAL, "no such chunk");
    const int gi = P->chunk_of[chunk].first, ci = P->chunk_of[chunk].second;
    GroupPlan &gp = *P->groups[gi];
    const GroupPlan::Chunk &c = gp.chunks[ci];
    GS_REQUIRE(c.n <= capacity && (c.n == 0 || (keys && vals)), GSPARC_EINVAL,
               "output arrays smaller than the chunk (gsparc_plan_chunk gives its size)");
    AccArgs b = gp.aa;
    b.chunk_base = c.first;
    b.out_keys = keys;
    b.out_vals = vals;
    b.out_cap = c.n;
    b.units = gp.L.get();
    b.nunits = (uint32_t)gp.nu;
    b.l0 = (uint32_t)c.lu0;
    b.l1 = (uint32_t)c.lu1;
    GS_CUDA(cudaMemsetAsync(gp.flags.get() + 1, 0, 4, s));
    launch_light(b, kLightFinal, (int)std::min<uint64_t>(gp.gl, std::max<uint64_t>(1, b.nunits)), s);
    b.units = gp.heavy_list() + c.h0;
    b.nunits = (uint32_t)(c.h1 - c.h0);
    if (gp.nh > gp.nnarrow) {
        GS_CUDA(cudaMemsetAsync(gp.flags.get() + 1, 0, 4, s));
        launch_heavy(b, true, (int)std::min<uint64_t>(gp.gh, std::max<uint64_t>(1, b.nunits)), s);
    }
    if (gp.nnarrow) {
        b.unit_off += c.h0;
        b.part_off += c.h0;
        GS_CUDA(cudaMemsetAsync(gp.flags.get() + 1, 0, 4, s));
        launch_narrow(b, true, gp.sm_count, s);
    }
    b.units = gp.SR.get() + c.s0;
    b.nunits = (uint32_t)(c.s1 - c.s0);
    b.sprefix = gp.sprefix.get() + c.s0;
    launch_stream(b, gp.gs_grid, s);
    for (int j = 0; j < gp.g; ++j) {
        if (!gp.jobs[j]->wide || gp.jobs[j]->key_words == 1) continue;  // written with final keys
        const uint64_t a0 = std::max(c.first, gp.job_first[j]), a1 = std::min(c.first + c.n, gp.job_first[j + 1]);
        if (a1 > a0) wide_remap_keys(*gp.jobs[j]->wide, keys + (a0 - c.first), a1 - a0, s);
    }
}

// Fetches the operands' current values into the plan's sorted value arrays.
void plan_refresh(gsparc_plan *P, cudaStream_t s) {
    GS_REQUIRE(P, GSPARC_EINVAL, "null plan");
    for (auto &g : P->groups) {
        GroupPlan &gp = *g;
        if (gp.nx) {
            k_bvals<<<grid_for(gp.nx), kThreads, 0, s>>>(gp.d_lx, gp.d_xoffs, gp.g, gp.nx, gp.xperm, gp.xvals);
            count_launch();
        }
        if (gp.ny) {
            k_bvals<<<grid_for(gp.ny), kThreads, 0, s>>>(gp.d_ly, gp.d_yoffs, gp.g, gp.ny, gp.yperm, gp.yvals);
            count_launch();
        }
        GS_CUDA(cudaGetLastError());
    }
}

// Waits for `s`, reads and clears the device-side error words of every group.
void plan_check(gsparc_plan *P, cudaStream_t s) {
    GS_REQUIRE(P, GSPARC_EINVAL, "null plan");
    for (auto &gp : P->groups) {
        unsigned int f = 0;
        d2h(&f, gp->flags.get(), 1, s);
        GS_CUDA(cudaMemsetAsync(gp->flags.get(), 0, 4, s));
        GS_CUDA(cudaStreamSynchronize(s));
        GS_REQUIRE(!(f & 2u), GSPARC_EINTERNAL, "light unit over capacity");
        GS_REQUIRE(!(f & 4u), GSPARC_EINTERNAL, "numeric pass wrote past its chunk");
    }
}

void plan_destroy(gsparc_plan *P) {
    if (!P) return;
    const int dev = P->ctx->device;
    int prev = -1;
    cudaGetDevice(&prev);
    if (prev != dev) cudaSetDevice(dev);
    cudaDeviceSynchronize();  // the buffers may still be read by executions in flight
    delete P;
    if (prev >= 0 && prev != dev) cudaSetDevice(prev);
}

uint64_t plan_nchunks(const gsparc_plan *P) { return P->chunk_of.size(); }

void plan_chunk(const gsparc_plan *P, uint64_t k, uint64_t *first, uint64_t *nnz) {
    GS_REQUIRE(k < P->chunk_of.size(), GSPARC_EINVAL, "no such chunk");
    const GroupPlan &gp = *P->groups[P->chunk_of[k].first];
    const GroupPlan::Chunk &c = gp.chunks[P->chunk_of[k].second];
    if (first) *first = P->group_off[P->chunk_of[k].first] + c.first;
    if (nnz) *nnz = c.n;
}

void plan_job_output(const gsparc_plan *P, int job, uint64_t *first, uint64_t *nnz) {
    GS_REQUIRE(job >= 0 && job < (int)P->job_first.size(), GSPARC_EINVAL, "no such job");
    if (first) *first = P->job_first[job];
    if (nnz) *nnz = P->job_nnz[job];
}

}  // namespace gs
