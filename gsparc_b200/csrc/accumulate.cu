// accumulate.cu -- light rows of the accumulation of matched products.
//
// Output row r is one X free index x_f (X is sorted free-major, so its
// nonzeros are contiguous).  Its products are the Y runs matched by the row's
// X nonzeros; every Y run is sorted by column (the Y free index, carried as a
// dense rank among Y's distinct free indices).  Rows of few products are done
// here: units of them are expanded, their sorted runs merged and compressed on
// chip (expand-sort-compress; reference ESC:
// include/gsparc/contraction.cuh:100-141,506-537), with a compensated
// sequential sum per output key.  Longer rows: rowwin.cu (windows of columns)
// and narrow.cu (few columns); rows of one run: stream.cu.  Sums that are
// exactly zero stay in the output, as in the reference's ESC
// (include/gsparc/contraction.cuh:532-537).
//
// Two passes: a symbolic one that counts each row's distinct columns, and a
// numeric one that writes each row's sorted output at its final offset.
#include "blockops.cuh"
#include "kernels.cuh"

namespace gs {

namespace {
using namespace dev;

// ------------------------------------------------------------------ light
// A unit's products are its rows' matched Y runs, laid out run after run; every
// run is sorted by column rank already, so a row of R runs needs only
// ceil(log2 R) rounds of pairwise merging, not a full sort.  An entry is one
// word, rank << 12 | entry before merging (K: 32 bits where the group has fewer
// than 2^20 columns), so entries are distinct and a merge is stable.  In a round
// every thread makes 8 consecutive entries of the output: one search finds
// where its first one splits the two groups (merge path), then each next one
// costs a compare and one shared load; the outputs wait in registers for the
// barrier, so one copy of the entries is enough.  Places are padded by one word
// in 32, or the 8-entry stride of the threads would meet in 4 banks.
//
// Afterwards a thread holds 8 merged entries: heads (first of a row and rank)
// are counted and scanned, each head sums its entries (its own thread's, then
// the next ones' where they go on), and the outputs leave in slot order.
//
// kLightCount counts the outputs of every row, kLightValues also writes them to
// scratch (a.lout_*), from where k_light_copy moves them once the output offsets
// are known; kLightFinal (plans, and where the scratch does not fit) redoes the
// merge of a chunk's light rows and writes them in place.
//
// Bound: instruction issue and the barriers around a unit's start, whose run
// table comes through dependent global loads.  Both passes together, us (ncu),
// with a bitonic sort of 64-bit keys / merge rounds by one search an entry, both
// in units of neighbouring rows / this: a batch of 24 mixed contractions 2000 /
// 848 / 314, 1e7 products in rows of about 490 -- / 1078 / 172, 1e6 products in
// rows of about 200 between single-run rows 460 / 243 / 61.
constexpr int kPer = 8;
constexpr int kIdBits = 12;
static_assert(kLightCap <= 1 << kIdBits, "an entry's number fits the key");

template <int C>
struct LightShape {
    static constexpr int T = C / kPer;
    static constexpr int WORDS = C / 32;
};

__device__ __forceinline__ uint32_t padded(uint32_t p) { return p + (p >> 5); }

// Entry p's run among those that start at the set bits of `bits` (pre: the
// runs that start before every word).
__device__ __forceinline__ uint32_t run_of(const uint32_t *bits, const uint16_t *pre, uint32_t p) {
    return pre[p >> 5] + __popc(bits[p >> 5] & (0xffffffffu >> (31 - (p & 31)))) - 1;
}

template <int MODE, int C, class K>
__global__ void __launch_bounds__(LightShape<C>::T) k_light(AccArgs a) {
    constexpr int T = LightShape<C>::T, WORDS = LightShape<C>::WORDS, NW = T / 32;
    constexpr bool VALUES = MODE != kLightCount;
    constexpr K kNone = ~(K)0;  // above every entry
    extern __shared__ __align__(16) unsigned char smem_raw[];
    K *key = reinterpret_cast<K *>(smem_raw);                     // [C + C / 32] entries
    uint32_t *rrow = reinterpret_cast<uint32_t *>(key + C + WORDS);  // [C] light row of every run
    uint32_t *rj0 = rrow + C;                                     // [C] first Y entry of every run
    float *xv = reinterpret_cast<float *>(rj0 + C);               // [C] (values) X value of every run
    uint32_t *sbits = reinterpret_cast<uint32_t *>(xv + (VALUES ? C : 0));  // [WORDS] a run starts at entry p
    uint32_t *rbits = sbits + WORDS;                              // [WORDS] a row starts at entry p
    uint16_t *off = reinterpret_cast<uint16_t *>(rbits + WORDS);  // [C + 2] first entry of every run
    uint16_t *rf = off + C + 2;                                   // [C] first run of the run's row
    uint16_t *re = rf + C;                                        // [C] end of the row's runs
    uint16_t *rs = re + C;                                        // [C] (first run of a row) outputs before the row
    uint16_t *spre = rs + C;                                      // [WORDS] runs starting before the word
    // after the sums: the outputs by slot
    uint32_t *orank = rj0;  // [C]
    float *oval = xv;       // [C]
    uint16_t *orun = off;   // [C]
    __shared__ uint32_t s_wsum[NW + 1];
    __shared__ uint32_t s_unit, s_maxr, s_first, s_last;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t p0 = tid * kPer;  // this thread's merged entries: p0 .. p0 + 7

    // the units that hold the light rows [a.l0, a.l1)
    if (tid < 2) {
        const uint32_t want = tid ? a.l1 - 1 : a.l0;  // the last unit that starts at or before it
        uint32_t lo = 0, hi = a.nunits;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (a.ustart[mid] <= want)
                lo = mid;
            else
                hi = mid;
        }
        (tid ? s_last : s_first) = lo;
    }
    __syncthreads();

    for (;;) {
        if (tid == 0) {
            s_unit = atomicAdd(a.work_counter, 1u);
            s_maxr = 0;
        }
        if (tid < WORDS) sbits[tid] = rbits[tid] = 0;
        __syncthreads();
        const uint32_t u = s_first + s_unit;
        if (u > s_last) break;
        const uint32_t l0 = max(a.ustart[u], a.l0), l1 = min(a.ustart[u + 1], a.l1);
        const uint32_t k0 = a.lk0[l0], nr = a.lk0[l1] - k0;  // the unit's runs
        const uint64_t P0 = a.lpre[l0];
        const uint32_t P = (uint32_t)(a.lpre[l1] - P0);
        if (P > (uint32_t)C) {  // planner guarantees otherwise
            if (tid == 0) atomicOr(a.err, 2u);
            __syncthreads();
            continue;
        }
        // runs (nr <= P)
        for (uint32_t k = tid; k < nr; k += T) {
            const uint32_t i = a.lrun[k0 + k], l = a.lrow[k0 + k];
            const uint32_t o = (uint32_t)(a.loff[k0 + k] - P0);
            const uint32_t f = a.lk0[l] - k0, e = a.lk0[l + 1] - k0;
            off[k] = (uint16_t)o;
            rj0[k] = a.pos[i];
            rrow[k] = l;
            rf[k] = (uint16_t)f;
            re[k] = (uint16_t)e;
            if (VALUES) xv[k] = a.xval[i];
            atomicOr(&sbits[o >> 5], 1u << (o & 31));
            if (k == f) {
                atomicOr(&rbits[o >> 5], 1u << (o & 31));
                atomicMax(&s_maxr, e - f);
            }
        }
        if (tid == 0) off[nr] = (uint16_t)P;
        __syncthreads();
        const uint32_t maxr = s_maxr;
        if (warp == 0) {  // runs starting before every word of flags
            uint32_t c[WORDS / 32], sum = 0;
#pragma unroll
            for (int q = 0; q < WORDS / 32; ++q) {
                c[q] = sum;
                sum += __popc(sbits[lane * (WORDS / 32) + q]);
            }
            uint32_t x = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= (uint32_t)o) x += y;
            }
#pragma unroll
            for (int q = 0; q < WORDS / 32; ++q) spre[lane * (WORDS / 32) + q] = (uint16_t)(x - sum + c[q]);
        }
        __syncthreads();

        // expand (a warp's lanes take consecutive entries)
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const uint32_t p = tid + T * q;
            if (p < P) {
                const uint32_t k = run_of(sbits, spre, p);
                key[padded(p)] = ((K)a.yrank[rj0[k] + p - off[k]] << kIdBits) | p;
            }
        }
        __syncthreads();

        // merge rounds: groups of 2^l runs of a row, two by two
        const uint32_t kp = p0 < P ? run_of(sbits, spre, p0) : 0u;  // run of this thread's first place
        const uint32_t mine = p0 < P ? min(P - p0, (uint32_t)kPer) : 0u;
        for (uint32_t l = 0; (1u << l) < maxr; ++l) {
            K out[kPer];
            if (mine) {
                uint32_t f = rf[kp], e = re[kp];
                uint32_t sa = f + ((kp - f) >> (l + 1) << (l + 1));  // the pair's first run
                uint32_t as = off[sa], ae = off[min(sa + (1u << l), e)], be = off[min(sa + (2u << l), e)];
                // how the pair's first p0 - as entries split
                const uint32_t d = p0 - as;
                uint32_t lo = d > be - ae ? d - (be - ae) : 0u, hi = min(d, ae - as);
                while (lo < hi) {
                    const uint32_t mid = (lo + hi) >> 1;
                    if (key[padded(as + mid)] < key[padded(ae + d - 1 - mid)])
                        lo = mid + 1;
                    else
                        hi = mid;
                }
                uint32_t x = as + lo, y = ae + d - lo;
                K kx = x < ae ? key[padded(x)] : kNone, ky = y < be ? key[padded(y)] : kNone;
#pragma unroll
                for (int q = 0; q < kPer; ++q) {
                    out[q] = kNone;
                    if ((uint32_t)q < mine) {
                        if (p0 + q == be) {  // the next pair
                            sa = min(sa + (2u << l), e);
                            if (sa == e) e = re[sa];  // of the next row
                            x = be;
                            ae = off[min(sa + (1u << l), e)];
                            be = off[min(sa + (2u << l), e)];
                            y = ae;
                            kx = key[padded(x)];
                            ky = y < be ? key[padded(y)] : kNone;
                        }
                        const bool left = kx < ky;
                        out[q] = left ? kx : ky;
                        const uint32_t nx = (left ? x : y) + 1, end = left ? ae : be;
                        const K v = nx < end ? key[padded(nx)] : kNone;
                        if (left) {
                            x = nx;
                            kx = v;
                        } else {
                            y = nx;
                            ky = v;
                        }
                    }
                }
            }
            __syncthreads();
#pragma unroll
            for (int q = 0; q < kPer; ++q)
                if ((uint32_t)q < mine) key[padded(p0 + q)] = out[q];
            __syncthreads();
        }

        // heads and their slots
        K my[kPer];
        uint32_t heads = 0;
        {
            uint32_t prev = p0 > 0 && mine ? (uint32_t)(key[padded(p0 - 1)] >> kIdBits) : 0u;
            const uint32_t starts = mine ? (rbits[p0 >> 5] >> (p0 & 31)) & 0xffu : 0u;
#pragma unroll
            for (int q = 0; q < kPer; ++q) {
                my[q] = (uint32_t)q < mine ? key[padded(p0 + q)] : kNone;
                const uint32_t rk = (uint32_t)(my[q] >> kIdBits);
                if ((uint32_t)q < mine && ((starts >> q & 1u) || rk != prev)) heads |= 1u << q;
                prev = rk;
            }
            const uint32_t n = __popc(heads);
            uint32_t inc = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= (uint32_t)o) inc += y;
            }
            if (lane == 31) s_wsum[warp] = inc;
            __syncthreads();
            uint32_t slot = inc - n, all = 0;
#pragma unroll
            for (int w = 0; w < NW; ++w) {
                if (w < (int)warp) slot += s_wsum[w];
                all += s_wsum[w];
            }
            // outputs before every row
            for (uint32_t b = starts & ((1u << mine) - 1u); b; b &= b - 1) {
                const uint32_t q = __ffs(b) - 1;
                rs[run_of(sbits, spre, p0 + q)] = (uint16_t)(slot + __popc(heads & ((1u << q) - 1u)));
            }
            __syncthreads();
            if (MODE != kLightFinal) {
                for (uint32_t k = tid; k < nr; k += T)
                    if (k == rf[k]) {
                        a.row_nnz[a.units[rrow[k]]] = (re[k] < nr ? rs[re[k]] : all) - rs[k];
                        if (MODE == kLightValues) a.lpos[rrow[k]] = P0 + rs[k];
                    }
            }
            if (VALUES) {
                float v[kPer];
                float pr[kPer], pe[kPer];
#pragma unroll
                for (int q = 0; q < kPer; ++q) {
                    pr[q] = pe[q] = 0.f;
                    if ((uint32_t)q < mine) {
                        const uint32_t id = (uint32_t)my[q] & ((1u << kIdBits) - 1u), k = run_of(sbits, spre, id);
                        const float x = xv[k], y = a.yval[rj0[k] + id - off[k]];
                        pr[q] = __fmul_rn(x, y);  // not contracted into the sum
                        pe[q] = fmaf(x, y, -pr[q]);
                    }
                }
                // each head's entries in order; a head's value ends up at its place
                float sum = 0.f, c = 0.f;
                int at = -1;
#pragma unroll
                for (int q = 0; q < kPer; ++q) {
                    v[q] = 0.f;
                    if (heads >> q & 1u) {
                        at = q;
                        sum = 0.f + pr[q];  // as from an empty accumulator: a product that
                        c = 0.f + pe[q];    // underflows to -0 alone gives +0 on every path but the copied rows'
                    } else {
                        float ns, err;
                        two_sum(sum, pr[q], ns, err);
                        sum = ns;
                        c += err + pe[q];
                    }
                    if ((uint32_t)q < mine) v[q] = sum + c;
                }
                // the last head's entries of the following threads
                if (at >= 0 && mine == kPer) {
                    const uint32_t rk = (uint32_t)(my[kPer - 1] >> kIdBits);
                    for (uint32_t p = p0 + kPer; p < P && !(rbits[p >> 5] >> (p & 31) & 1u); ++p) {
                        const K w = key[padded(p)];
                        if ((uint32_t)(w >> kIdBits) != rk) break;
                        const uint32_t id = (uint32_t)w & ((1u << kIdBits) - 1u), k = run_of(sbits, spre, id);
                        const float x = xv[k], y = a.yval[rj0[k] + id - off[k]];
                        const float pq = __fmul_rn(x, y);
                        float ns, err;
                        two_sum(sum, pq, ns, err);
                        sum = ns;
                        c += err + fmaf(x, y, -pq);
                    }
                }
                const float last = sum + c;
                uint32_t krun[kPer];
#pragma unroll
                for (int q = 0; q < kPer; ++q)
                    if (heads >> q & 1u) krun[q] = rf[run_of(sbits, spre, p0 + q)];
                __syncthreads();  // rj0, xv and off are read
#pragma unroll
                for (int q = 0; q < kPer; ++q)
                    if (heads >> q & 1u) {
                        // a head's value stands at the entry before the next head
                        const uint32_t rest = heads & (0xfffffffeu << q);
                        float z = last;
                        if (rest) {
                            const int nq = __ffs(rest) - 2;
#pragma unroll
                            for (int t = 0; t < kPer; ++t)
                                if (t == nq) z = v[t];
                        }
                        const uint32_t o = slot + __popc(heads & ((1u << q) - 1u));
                        orank[o] = (uint32_t)(my[q] >> kIdBits);
                        oval[o] = z;
                        orun[o] = (uint16_t)krun[q];
                    }
                __syncthreads();
                uint64_t *ok = MODE == kLightFinal ? a.out_keys : a.lout_keys;
                float *ov = MODE == kLightFinal ? a.out_vals : a.lout_vals;
                for (uint32_t o = tid; o < all; o += T) {
                    const uint32_t k = orun[o], row = a.units[rrow[k]];
                    int y_nfbits;
                    const uint64_t *cols;
                    uint32_t ncols;
                    row_job_params(a, row, y_nfbits, cols, ncols);
                    const uint64_t to =
                        MODE == kLightFinal ? a.row_off[row] - a.chunk_base + (o - rs[k]) : P0 + o;
                    if (to < a.out_cap) {
                        ok[to] = shl(a.row_xf[row], y_nfbits) | cols[orank[o]];
                        ov[to] = oval[o];
                    } else {
                        atomicOr(a.err, 4u);
                    }
                }
            }
        }
        __syncthreads();
    }
}

// The outputs of a chunk's light rows from scratch to their places, a warp a row.
__global__ void __launch_bounds__(256) k_light_copy(AccArgs a) {
    const uint32_t lane = threadIdx.x & 31, step = gridDim.x * 8;
    for (uint32_t l = a.l0 + blockIdx.x * 8 + (threadIdx.x >> 5); l < a.l1; l += step) {
        const uint32_t row = a.units[l];
        const uint64_t o0 = a.row_off[row] - a.chunk_base, from = a.lpos[l];
        const uint32_t n = (uint32_t)(a.row_off[row + 1] - a.row_off[row]);
        if (o0 + n > a.out_cap) {
            if (lane == 0) atomicOr(a.err, 4u);
            continue;
        }
        const unsigned long long *sk = (const unsigned long long *)a.lout_keys + from;
        const float *sv = a.lout_vals + from;
        for (uint32_t i = lane; i < n; i += 32) {
            __stcs((unsigned long long *)a.out_keys + o0 + i, __ldcs(sk + i));
            __stcs(a.out_vals + o0 + i, __ldcs(sv + i));
        }
    }
}

template <int C, class K>
size_t light_smem(bool values) {
    // key | rrow, rj0 | xv | sbits, rbits | off, rf, re, rs, spre
    return sizeof(K) * (C + C / 32) + (size_t)C * 8 + (values ? (size_t)C * 4 : 0) + C / 4 +
           2 * ((size_t)4 * C + 2 + C / 32);
}

template <int MODE, int C, class K>
void launch_light_as(const AccArgs &a, int grid, cudaStream_t s) {
    const size_t sm = light_smem<C, K>(MODE != kLightCount);
    GS_CUDA(cudaFuncSetAttribute(k_light<MODE, C, K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    k_light<MODE, C, K><<<grid, LightShape<C>::T, sm, s>>>(a);
}

template <int MODE>
void launch_light_mode(const AccArgs &a, int grid, cudaStream_t s) {
    const bool narrow_key = a.light_cols < 1ull << (32 - kIdBits);  // the largest key stays free
    if (a.light_cap <= (uint32_t)kLightCap / 2) {
        if (narrow_key)
            launch_light_as<MODE, kLightCap / 2, uint32_t>(a, grid, s);
        else
            launch_light_as<MODE, kLightCap / 2, uint64_t>(a, grid, s);
    } else {
        if (narrow_key)
            launch_light_as<MODE, kLightCap, uint32_t>(a, grid, s);
        else
            launch_light_as<MODE, kLightCap, uint64_t>(a, grid, s);
    }
}

}  // namespace

int light_blocks_per_sm() { return 5; }

// a.light_cap products at most in a unit: the capacity the planner packed for.
void launch_light(const AccArgs &a, int mode, int grid, cudaStream_t s) {
    if (a.nunits == 0 || a.l1 <= a.l0) return;
    if (mode == kLightCount)
        launch_light_mode<kLightCount>(a, grid, s);
    else if (mode == kLightValues)
        launch_light_mode<kLightValues>(a, grid, s);
    else
        launch_light_mode<kLightFinal>(a, grid, s);
    count_launch();
    GS_CUDA(cudaGetLastError());
}

void launch_light_copy(const AccArgs &a, int sm_count, cudaStream_t s) {
    if (a.l1 <= a.l0) return;
    k_light_copy<<<std::min<unsigned>((a.l1 - a.l0 + 7) / 8, (unsigned)sm_count * 8u), 256, 0, s>>>(a);
    count_launch();
    GS_CUDA(cudaGetLastError());
}

}  // namespace gs
