// narrow.cu -- heavy rows over a narrow column space.
//
// When a job has at most kNarrowCols distinct columns, a long row needs no
// windows, bitmaps or searches: every warp keeps its own (sum, error) pair per
// column in shared memory and adds the products it meets by TwoSum, without
// atomics; the warps' and then the units' pairs are added in a fixed order.
// Rows are cut into slices of about equal products, so a few hundred rows of
// millions of products fill the GPU (the windowed kernel gives a row to one
// CTA: 200 rows kept 100 SMs busy).
//
// A warp takes 32 runs at a time, flattens them by a shuffle scan and steps
// through their entries 32 at a time (a lane's run: a reduction over the lanes'
// run starts and a popcount).  Inside one run of a job whose Y repeats no
// coordinate the columns of a step are distinct; where a step spans runs,
// lanes of the same column take turns: each writes its lane number to the
// column's tag and the one that reads itself back adds.
//
// A run of at least kLongRun entries is added by itself first: its X value and
// address are the warp's, its columns are distinct, so its steps need neither a
// search nor turns and four are in flight.  The line lies where a run's last,
// partly empty step costs no more than the search it saves: 32, 64 and 128 give
// the same (1.394, 1.390, 1.407 ms; 1.69 ms without, at the size below).
//
// The symbolic pass only marks columns and stops as soon as all are marked.
//
// Bound: shared-memory latency of the read-add-write of a step and the loads
// of the Y entries from L2.  1e7 x 1e7 nonzeros, 6.6e8 products onto 200 x 300
// outputs, against the windowed kernel: numeric 4637 -> 1390 us, symbolic
// 2081 -> 171 us.
#include "blockops.cuh"
#include "kernels.cuh"
#include "rows.h"

namespace gs {

namespace {
using namespace dev;

constexpr int NT = 256;
constexpr int NW = NT / 32;
constexpr uint32_t FULL = 0xffffffffu;
constexpr uint32_t INF = 0xffffffffu;
constexpr int ILP = 4;
constexpr uint32_t kLongRun = 64;  // runs of so many entries are added by themselves

// Last p in [0, n) with off[p] <= u (off[0] <= u < off[n]); 32 probes a step,
// all lanes of a warp.
__device__ __forceinline__ uint32_t warp_find(const uint32_t *__restrict__ off, uint32_t n, uint32_t u) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t lo = 0, hi = n;
    while (hi - lo > 1) {
        const uint32_t step = (hi - lo + 31) / 32;
        const uint64_t q = (uint64_t)lo + (uint64_t)(lane + 1) * step;
        const uint32_t below = __popc(__ballot_sync(FULL, q < hi && off[q] <= u));
        lo += below * step;
        hi = min(hi, lo + step);
    }
    return lo;
}

// First k in [k0, k1] (matched nonzeros) with at least `want` products before it.
__device__ __forceinline__ uint32_t run_at(const AccArgs &a, uint32_t k0, uint32_t k1, uint64_t want) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t lo = k0, hi = k1;  // every k < lo is below, hi is not (or is k1)
    while (lo < hi) {
        const uint32_t step = (hi - lo + 31) / 32;
        const uint64_t q = (uint64_t)lo + (uint64_t)lane * step;
        const uint32_t below = __popc(__ballot_sync(FULL, q < hi && a.xprefix[a.mrun[q < hi ? q : lo]] < want));
        if (below == 0) return lo;
        const uint64_t last = (uint64_t)lo + (uint64_t)(below - 1) * step;  // below `want`
        hi = (uint32_t)min((uint64_t)hi, last + step);
        lo = (uint32_t)last + 1;
    }
    return lo;
}

// The products of x with N entries, 32 apart, of one run (no column twice) into
// the warp's pairs; TAIL: only those below `left`.
template <int N, bool TAIL>
__device__ __forceinline__ void add_words(float2 *my, const uint32_t *__restrict__ rank, const float *__restrict__ yv,
                                          float x, int left) {
    uint32_t c[N];
    float y[N];
    float2 z[N];
#pragma unroll
    for (int e = 0; e < N; ++e) {
        c[e] = 0;
        if (!TAIL || 32 * e < left) {
            c[e] = rank[32 * e];
            y[e] = yv[32 * e];
        }
    }
#pragma unroll
    for (int e = 0; e < N; ++e)
        if (!TAIL || 32 * e < left) z[e] = my[c[e]];
#pragma unroll
    for (int e = 0; e < N; ++e)
        if (!TAIL || 32 * e < left) {
            const float pr = __fmul_rn(x, y[e]);  // not contracted into the sum
            const float pe = fmaf(x, y[e], -pr);
            float sum, err;
            two_sum(z[e].x, pr, sum, err);
            my[c[e]] = make_float2(sum, z[e].y + (err + pe));
        }
}

template <bool NUMERIC>
__global__ void __launch_bounds__(NT) k_narrow(AccArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const uint32_t nc = a.narrow_cols, ncp = (nc + 3u) & ~3u;
    float2 *acc = reinterpret_cast<float2 *>(smem_raw);                             // [NW][ncp]
    uint8_t *tags = reinterpret_cast<uint8_t *>(acc + (NUMERIC ? NW * ncp : 0));    // [NW][ncp]
    __shared__ uint32_t s_bits[kNarrowCols / 32];
    __shared__ uint32_t s_u[5];
    __shared__ uint32_t s_base[NUMERIC ? NW : 1][32], s_len[NUMERIC ? NW : 1][32];
    __shared__ float s_xv[NUMERIC ? NW : 1][32];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t le = 0xffffffffu >> (31 - lane);
    float2 *my = acc + warp * ncp;
    uint8_t *tag = tags + warp * ncp;
    if (*a.err & kScanErr) return;  // the units were not written
    const uint32_t ubase = a.unit_off[0], nunits = a.unit_off[a.nunits] - ubase;
    if (NUMERIC)
        for (uint32_t c = tid; c < NW * ncp; c += NT) acc[c] = make_float2(0.f, 0.f);

    for (;;) {
        __syncthreads();
        if (warp == 0) {
            uint32_t u = 0;
            if (lane == 0) u = atomicAdd(a.work_counter, 1u);
            u = __shfl_sync(FULL, u, 0);
            if (lane == 0) s_u[0] = INF;
            if (u < nunits) {
                const uint32_t at = warp_find(a.unit_off, a.nunits, ubase + u);
                if (lane == 0) {
                    s_u[0] = a.units[at];
                    s_u[1] = ubase + u - a.unit_off[at];            // slice
                    s_u[2] = a.unit_off[at + 1] - a.unit_off[at];   // slices of the row
                    s_u[3] = a.part_off[at];                        // its first partial sums
                }
            }
        }
        __syncthreads();
        const uint32_t row = s_u[0];
        if (row == INF) break;
        const uint32_t slice = s_u[1], nu = s_u[2];
        const BatchJob job = a.jobs[a.row_job[row]];
        const uint32_t xs = a.row_start[row], xe = a.row_start[row + 1];
        const uint32_t k0 = a.mpre[xs], k1 = a.mpre[xe];
        const uint64_t P0 = a.xprefix[xs], P = a.xprefix[xe] - P0;
        uint32_t *gbits = a.nbm + (uint64_t)a.row_xi[row] * (kNarrowCols / 32);
        const uint32_t full = lane < job.ncols / 32 ? FULL
                              : lane == job.ncols / 32 ? (1u << (job.ncols & 31)) - 1u : 0u;  // a word per lane
        static_assert(kNarrowCols == 1024, "a lane per word of marks");
        if (!NUMERIC) {
            if (tid < 32) s_bits[tid] = __ldcg(gbits + tid);
            __syncthreads();
        }

        // this warp's runs: its share of the slice's products
        const uint64_t share = (uint64_t)slice * NW + warp, shares = (uint64_t)nu * NW;
        const uint32_t ka = run_at(a, k0, k1, P0 + (uint64_t)((unsigned __int128)P * share / shares));
        const uint32_t kb =
            share + 1 == shares ? k1 : run_at(a, k0, k1, P0 + (uint64_t)((unsigned __int128)P * (share + 1) / shares));

        for (uint32_t kk = ka; kk < kb; kk += 32) {
            if (!NUMERIC && __all_sync(FULL, (volatile uint32_t &)s_bits[lane] == full)) break;
            uint32_t base = 0, len = 0;
            float xv = 0.f;
            if (kk + lane < kb) {
                const uint32_t i = a.mrun[kk + lane];
                base = a.pos[i];
                len = a.cnt[i];
                if (NUMERIC) xv = a.xval[i];
            }
            if (NUMERIC && !job.ydup) {
                uint32_t longs = __ballot_sync(FULL, len >= kLongRun);
                for (; longs; longs &= longs - 1u) {
                    const int k = __ffs(longs) - 1;
                    const uint32_t n = __shfl_sync(FULL, len, k);
                    const uint32_t *rk = a.yrank + (uint64_t)__shfl_sync(FULL, base, k) + lane;
                    const float *yv = a.yval + (rk - a.yrank);
                    const float x = __shfl_sync(FULL, xv, k);
                    uint32_t t = 0;
                    for (; t + 32 * ILP <= n; t += 32 * ILP) add_words<ILP, false>(my, rk + t, yv + t, x, 0);
                    for (; t < n; t += 64) add_words<2, true>(my, rk + t, yv + t, x, (int)(n - t - lane));
                    __syncwarp();
                }
                // the other runs move to the first lanes: the walk below counts run
                // starts, so an empty lane between two runs would shift the rest
                const uint32_t rest = __ballot_sync(FULL, len != 0 && len < kLongRun);
                if (rest >> lane & 1u) {
                    const uint32_t p = __popc(rest & (le >> 1));
                    s_base[warp][p] = base;
                    s_len[warp][p] = len;
                    s_xv[warp][p] = xv;
                }
                __syncwarp();
                len = 0;
                if (lane < (uint32_t)__popc(rest)) {
                    base = s_base[warp][lane];
                    len = s_len[warp][lane];
                    xv = s_xv[warp][lane];
                }
                __syncwarp();
            }
            uint32_t off = len;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(FULL, off, o);
                if (lane >= (uint32_t)o) off += y;
            }
            const uint32_t tot = __shfl_sync(FULL, off, 31);
            off -= len;
            base -= off;                       // entry t of the batch is Y entry base + t
            const uint32_t at = len ? off : INF;  // lanes past the last run start nothing
            uint32_t kp = INF;                 // runs that start before the step, minus one
            for (uint32_t t = 0; t < tot; t += 32 * ILP) {
                uint32_t r[ILP], several[ILP];
                float x[ILP], y[ILP];
#pragma unroll
                for (int e = 0; e < ILP; ++e) {
                    const uint32_t te = t + 32 * e;
                    const uint32_t m = __reduce_or_sync(FULL, at - te < 32u ? 1u << (at - te) : 0u);
                    const uint32_t k = (kp + __popc(m & le)) & 31u;
                    kp += __popc(m);
                    several[e] = m & ~1u;  // runs start inside the step
                    const uint32_t j = __shfl_sync(FULL, base, k) + te + lane;
                    if (NUMERIC) x[e] = __shfl_sync(FULL, xv, k);
                    r[e] = INF;
                    if (te + lane < tot) {
                        r[e] = a.yrank[j];
                        if (NUMERIC) y[e] = a.yval[j];
                    }
                }
#pragma unroll
                for (int e = 0; e < ILP; ++e) {
                    const uint32_t c = r[e];
                    bool todo = c != INF;
                    if (!NUMERIC) {
                        if (todo && !((volatile uint32_t &)s_bits[c >> 5] >> (c & 31) & 1u))
                            atomicOr(&s_bits[c >> 5], 1u << (c & 31));
                        continue;
                    }
                    float pr = 0.f, pe = 0.f;
                    if (todo) {
                        pr = __fmul_rn(x[e], y[e]);  // not contracted into the sum
                        pe = fmaf(x[e], y[e], -pr);
                    }
                    auto add = [&] {
                        const float2 z = my[c];
                        float sum, err;
                        two_sum(z.x, pr, sum, err);
                        my[c] = make_float2(sum, z.y + (err + pe));
                    };
                    if (!several[e] && !job.ydup) {
                        if (todo) add();
                        __syncwarp();
                    } else {
                        while (__any_sync(FULL, todo)) {
                            if (todo) tag[c] = (uint8_t)lane;
                            __syncwarp();
                            if (todo && tag[c] == lane) {
                                add();
                                todo = false;
                            }
                            __syncwarp();
                        }
                    }
                }
            }
        }
        __syncthreads();
        if (!NUMERIC) {
            if (tid < 32 && s_bits[tid]) atomicOr(gbits + tid, s_bits[tid]);
            continue;
        }
        // the warps' pairs, in warp order
        const uint64_t o0 = a.row_off[row] - a.chunk_base, xf_hi = shl(a.row_xf[row], job.y_nfbits);
        float2 *part = a.part + (uint64_t)(s_u[3] + slice) * nc;
        for (uint32_t c0 = 0; c0 < job.ncols; c0 += NT) {
            const uint32_t c = c0 + tid;
            if (c >= job.ncols) break;
            float s = 0.f, e = 0.f;
#pragma unroll
            for (int w = 0; w < NW; ++w) {
                const float2 z = acc[w * ncp + c];
                float ns, err;
                two_sum(s, z.x, ns, err);
                s = ns;
                e += err + z.y;
                acc[w * ncp + c] = make_float2(0.f, 0.f);
            }
            if (nu > 1) {
                part[c] = make_float2(s, e);
                continue;
            }
            uint32_t slot = 0;  // marked columns before c
            for (uint32_t w = 0; w < c / 32; ++w) slot += __popc(gbits[w]);
            const uint32_t b = gbits[c >> 5];
            if (!(b >> (c & 31) & 1u)) continue;
            slot += __popc(b & ((1u << (c & 31)) - 1u));
            if (o0 + slot < a.out_cap) {
                a.out_keys[o0 + slot] = xf_hi | a.cols[job.cols_off + c];
                a.out_vals[o0 + slot] = s + e;
            } else {
                atomicOr(a.err, 4u);
            }
        }
    }
}

// Rows of several units: their partial pairs in unit order.  A CTA per row.
__global__ void __launch_bounds__(NT) k_narrow_sum(AccArgs a) {
    if (*a.err & kScanErr) return;
    for (uint32_t at = blockIdx.x; at < a.nunits; at += gridDim.x) {
        const uint32_t nu = a.unit_off[at + 1] - a.unit_off[at];
        if (nu < 2) continue;
        const uint32_t row = a.units[at];
        const BatchJob job = a.jobs[a.row_job[row]];
        const uint32_t *gbits = a.nbm + (uint64_t)a.row_xi[row] * (kNarrowCols / 32);
        const uint64_t o0 = a.row_off[row] - a.chunk_base, xf_hi = shl(a.row_xf[row], job.y_nfbits);
        const float2 *part = a.part + (uint64_t)a.part_off[at] * a.narrow_cols;
        for (uint32_t c = threadIdx.x; c < job.ncols; c += NT) {
            const uint32_t b = gbits[c >> 5];
            if (!(b >> (c & 31) & 1u)) continue;
            uint32_t slot = __popc(b & ((1u << (c & 31)) - 1u));
            for (uint32_t w = 0; w < c / 32; ++w) slot += __popc(gbits[w]);
            float s = 0.f, e = 0.f;
            for (uint32_t u = 0; u < nu; ++u) {
                const float2 z = part[(uint64_t)u * a.narrow_cols + c];
                float ns, err;
                two_sum(s, z.x, ns, err);
                s = ns;
                e += err + z.y;
            }
            if (o0 + slot < a.out_cap) {
                a.out_keys[o0 + slot] = xf_hi | a.cols[job.cols_off + c];
                a.out_vals[o0 + slot] = s + e;
            } else {
                atomicOr(a.err, 4u);
            }
        }
    }
}

// Outputs of every narrow row of a list (a warp per row).
__global__ void __launch_bounds__(NT) k_narrow_count(AccArgs a) {
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t at = blockIdx.x * NW + (threadIdx.x >> 5); at < a.nunits; at += gridDim.x * NW) {
        const uint32_t row = a.units[at];
        if (a.row_class[row] != kRowNarrow) continue;
        const uint32_t n = __reduce_add_sync(
            FULL, (uint32_t)__popc(a.nbm[(uint64_t)a.row_xi[row] * (kNarrowCols / 32) + lane]));
        if (lane == 0) a.row_nnz[row] = n;
    }
}

// Units of every row of a heavy list (0: not a narrow row) and partial sums of
// the rows of several units, as prefix sums.
__global__ void __launch_bounds__(kScanThreads)
    k_narrow_units(const uint32_t *__restrict__ list, uint32_t n, const uint8_t *__restrict__ row_class,
                   const uint64_t *__restrict__ row_prod, uint64_t slice, uint32_t *__restrict__ unit_off,
                   uint32_t *__restrict__ part_off, ScanState st) {
    __shared__ ScanShared<2> sh;
    const uint32_t tile = next_tile(st, sh);
    const uint32_t i0 = tile * kScanTile + threadIdx.x * kScanItems;
    uint32_t c[kScanItems];
    uint64_t x[2] = {0, 0};
#pragma unroll
    for (int q = 0; q < kScanItems; ++q) {
        c[q] = 0;
        if (i0 + q < n) {
            const uint32_t row = list[i0 + q];
            if (row_class[row] == kRowNarrow) c[q] = (uint32_t)((row_prod[row] + slice - 1) / slice);
            x[0] += c[q];
            x[1] += c[q] > 1 ? c[q] : 0;
        }
    }
    if (!tile_scan<2>(st, sh, tile, x)) return;
#pragma unroll
    for (int q = 0; q < kScanItems; ++q)
        if (i0 + q < n) {
            unit_off[i0 + q] = (uint32_t)x[0];
            part_off[i0 + q] = (uint32_t)x[1];
            x[0] += c[q];
            x[1] += c[q] > 1 ? c[q] : 0;
        }
    if ((uint64_t)(tile + 1) * kScanTile >= n && threadIdx.x == 0) unit_off[n] = (uint32_t)sh.through[0];
}

size_t narrow_smem(bool numeric, uint32_t cols) {
    const size_t ncp = (cols + 3u) & ~3u;
    return numeric ? NW * ncp * (sizeof(float2) + 1) : 0;
}

// The kernel's shared memory limit is the function's, not the launch's: every
// call sets the same one, the widest job's, so that no thread lowers it between
// another thread's setting and its launch.
template <bool NUMERIC>
int narrow_grid(int sm_count, uint32_t cols) {
    int n = 0;
    const size_t sm = narrow_smem(NUMERIC, cols);
    GS_CUDA(cudaFuncSetAttribute(k_narrow<NUMERIC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)narrow_smem(NUMERIC, kNarrowCols)));
    GS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_narrow<NUMERIC>, NT, sm));
    return sm_count * std::max(n, 1);
}

}  // namespace

void launch_narrow(const AccArgs &a, bool numeric, int sm_count, cudaStream_t s) {
    if (a.nunits == 0) return;
    const size_t sm = narrow_smem(numeric, a.narrow_cols);
    const int rows = (int)std::min<uint32_t>(a.nunits, (uint32_t)sm_count * 8);
    if (numeric) {
        k_narrow<true><<<narrow_grid<true>(sm_count, a.narrow_cols), NT, sm, s>>>(a);
        k_narrow_sum<<<rows, NT, 0, s>>>(a);
    } else {
        k_narrow<false><<<narrow_grid<false>(sm_count, a.narrow_cols), NT, sm, s>>>(a);
        k_narrow_count<<<(rows + NW - 1) / NW, NT, 0, s>>>(a);
    }
    count_launch(2);
    GS_CUDA(cudaGetLastError());
}

void launch_narrow_units(const uint32_t *list, uint32_t n, const uint8_t *row_class, const uint64_t *row_prod,
                         uint64_t slice, uint32_t *unit_off, uint32_t *part_off, const ScanState &st, cudaStream_t s) {
    if (n == 0) return;
    k_narrow_units<<<(unsigned)scan_tiles(n), kScanThreads, 0, s>>>(list, n, row_class, row_prod, slice, unit_off,
                                                                    part_off, st);
    count_launch();
    GS_CUDA(cudaGetLastError());
}

}  // namespace gs
