// accumulate.cu -- symbolic and numeric accumulation of matched products.
//
// Output row r is one X free index x_f (X is sorted free-major, so its
// nonzeros are contiguous).  Its products are the Y runs matched by the row's
// X nonzeros; every Y run is sorted by column (the Y free index, carried as a
// dense rank among Y's distinct free indices).  Two accumulators:
//
//  * heavy rows (many products): a dense window of kHeavyW columns in shared
//    memory sweeps the row's column range; each run keeps a cursor, so every
//    window takes exactly the run entries that fall inside it.  Sums are
//    compensated: the hardware add returns the old value, from which the exact
//    rounding error of that addition is rebuilt (TwoSum) and accumulated in a
//    second word; each product's own rounding error (fma) goes there too.
//    Touched cells are tracked in a bitmap so exact-zero sums still count
//    (the reference's ESC keeps them, include/gsparc/contraction.cuh:532-537).
//  * light rows (few products): units of consecutive rows are expanded, their
//    sorted runs merged and compressed on chip (expand-sort-compress; reference
//    ESC: include/gsparc/contraction.cuh:100-141,506-537), with a compensated
//    sequential sum per output key.
//
// Both run twice: a symbolic pass that only counts each row's distinct
// columns, and a numeric pass that writes each row's sorted output at its
// final offset.
#include "blockops.cuh"
#include "kernels.cuh"

namespace gs {

namespace {
using namespace dev;

// Threads of a light CTA: 256 for units of up to 2048 products (the default
// rows of up to 1024 products), 512 for 4096, so a thread holds 8 entries.
template <int C>
struct LightShape {
    static constexpr int T = C / 8;
};

// ------------------------------------------------------------------ light
// A unit's products are its rows' matched Y runs, laid out run after run; every
// run is sorted by column rank already, so a row of R runs needs only
// ceil(log2 R) rounds of pairwise merging, not a full sort: in round l the
// groups of 2^l consecutive runs of a row are merged two by two, an entry's
// new position being its offset in its own group plus the number of entries
// of the sibling group before it (a binary search in shared memory; ties keep
// the left group first, so the order is stable and the sums deterministic).
// The entries are held in registers between the two barriers of a round, so
// one copy of (rank, product id) is enough.  A warp owns 32 * PER consecutive
// entries, lane-strided, which makes the head flags a ballot and their scan a
// popcount.
//
// Bound: shared-memory latency of the binary searches and the barriers around
// a unit's start (its run table comes through dependent global loads).
// Against the bitonic sort of (row, rank) pairs this replaced, in a batch of 24
// mixed contractions (light rows of 2 to some hundred runs): symbolic
// 851 -> 305 us, numeric 1149 -> 540 us.  Searches of a thread's 8 entries in
// step (a fixed number of probes for the warp's longest group) were slower:
// 385 us symbolic.
template <bool NUMERIC, int C>
__global__ void __launch_bounds__(LightShape<C>::T) k_light(AccArgs a) {
    constexpr int T = LightShape<C>::T;
    constexpr int NW = T / 32;
    constexpr int PER = C / T;  // entries per thread
    constexpr int WORDS = C / 32;
    static_assert(WORDS <= T, "one thread per flag word");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint32_t *key = reinterpret_cast<uint32_t *>(smem_raw);  // [C] column ranks, merged in place
    uint32_t *rrow = key + C;                                // [C] row of every run
    uint32_t *rj0 = rrow + C;                                // [C] first Y entry of every run ...
    uint16_t *hs = reinterpret_cast<uint16_t *>(rj0);        // ... then [C] heads before every entry
    uint32_t *sbits = rj0 + C;                               // [WORDS] bit p: a run starts at entry p
    uint16_t *pid = reinterpret_cast<uint16_t *>(sbits + WORDS);  // [C] product (entry before merging)
    uint16_t *off = pid + C;                                 // [C + 2] first entry of every run
    uint16_t *rf = off + C + 2;                              // [C] first run of the run's row
    uint16_t *re = rf + C;                                   // [C] end of the row's runs
    uint16_t *spre = re + C;                                 // [WORDS] runs starting before the word
    float *xv = reinterpret_cast<float *>(spre + WORDS + (WORDS & 1));  // [C] (numeric) X value of every run
    float *yv = xv + C;                                      // [C] (numeric) Y value of every product
    __shared__ uint32_t s_wsum[NW + 1];
    __shared__ uint32_t s_unit, s_maxr;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t le = 0xffffffffu >> (31 - lane);  // lanes up to this one
    const uint32_t p0 = warp * (32 * PER) + lane;    // this thread's entries: p0 + 32 q

    for (;;) {
        if (tid == 0) {
            s_unit = atomicAdd(a.work_counter, 1u);
            s_maxr = 0;
        }
        if (tid < WORDS) sbits[tid] = 0;
        __syncthreads();
        const uint32_t u = s_unit;
        if (u >= a.nunits) break;
        const uint32_t r0 = a.units[2 * u], r1 = a.units[2 * u + 1];
        const uint32_t xs = a.row_start[r0], xe = a.row_start[r1];
        const uint64_t P0 = a.xprefix[xs];
        const uint32_t P = (uint32_t)(a.xprefix[xe] - P0);
        const uint32_t k0 = a.mpre[xs], nr = a.mpre[xe] - k0;  // the unit's runs (nr <= P)
        if (P > (uint32_t)C) {  // planner guarantees otherwise
            if (tid == 0) atomicOr(a.err, 2u);
            __syncthreads();
            continue;
        }
        // runs
        for (uint32_t k = tid; k < nr; k += T) {
            const uint32_t i = a.mrun[k0 + k];
            uint32_t lo = r0, hi = r1;  // largest r in [r0, r1) with row_start[r] <= i
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) >> 1;
                if (a.row_start[mid] <= i)
                    lo = mid;
                else
                    hi = mid;
            }
            const uint32_t o = (uint32_t)(a.xprefix[i] - P0);
            const uint32_t f = a.mpre[a.row_start[lo]] - k0, e = a.mpre[a.row_start[lo + 1]] - k0;
            off[k] = (uint16_t)o;
            rj0[k] = a.pos[i];
            rrow[k] = lo;
            rf[k] = (uint16_t)f;
            re[k] = (uint16_t)e;
            if (NUMERIC) xv[k] = a.xval[i];
            atomicOr(&sbits[o >> 5], 1u << (o & 31));
            if (k == f) atomicMax(&s_maxr, e - f);
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

        // expand
        uint16_t kk[PER];  // run of every entry (of its place: groups keep their places)
#pragma unroll
        for (int q = 0; q < PER; ++q) {
            const uint32_t p = p0 + 32 * q;
            kk[q] = 0;
            if (p < P) {
                const uint32_t k = spre[p >> 5] + __popc(sbits[p >> 5] & le) - 1;  // p & 31 == lane
                kk[q] = (uint16_t)k;
                const uint32_t j = rj0[k] + p - off[k];
                key[p] = a.yrank[j];
                pid[p] = (uint16_t)p;
                if (NUMERIC) yv[p] = a.yval[j];
            }
        }
        __syncthreads();

        // merge rounds
        for (uint32_t l = 0; (1u << l) < maxr; ++l) {
            uint32_t x[PER], np[PER];  // rank; product id and new place (16 bits each)
#pragma unroll
            for (int q = 0; q < PER; ++q) {
                const uint32_t p = p0 + 32 * q;
                np[q] = p;
                x[q] = 0;
                if (p < P) {
                    const uint32_t k = kk[q], f = rf[k], e = re[k];
                    const uint32_t g = (k - f) >> l, right = g & 1u, s0 = f + ((g ^ 1u) << l);
                    uint32_t to = p;
                    if (s0 < e) {
                        const uint32_t v = key[p];
                        const uint32_t slo = off[s0];
                        uint32_t lo = slo, hi = off[min(s0 + (1u << l), e)];
                        // sibling entries before this one: those below v, or up to v for an entry
                        // of the right group (ranks are below 2^31)
                        while (lo < hi) {
                            const uint32_t mid = (lo + hi) >> 1;
                            if (key[mid] < v + right)
                                lo = mid + 1;
                            else
                                hi = mid;
                        }
                        // a right group's sibling starts where the merged group does
                        to = right ? p - off[f + (g << l)] + lo : p + lo - slo;
                        x[q] = v;
                    }
                    np[q] = to | ((uint32_t)pid[p] << 16);
                }
            }
            __syncthreads();
#pragma unroll
            for (int q = 0; q < PER; ++q) {
                const uint32_t to = np[q] & 0xffffu;
                if (to != p0 + 32 * q) {  // entries that stay are in place already
                    key[to] = x[q];
                    pid[to] = (uint16_t)(np[q] >> 16);
                }
            }
            __syncthreads();
        }

        // heads: the first entry of every (row, rank); heads before every entry
        uint32_t bal[PER], mine = 0;
#pragma unroll
        for (int q = 0; q < PER; ++q) {
            const uint32_t p = p0 + 32 * q;
            const bool h = p < P && (p == off[rf[kk[q]]] || key[p] != key[p - 1]);
            bal[q] = __ballot_sync(0xffffffffu, h);
            mine += __popc(bal[q]);
        }
        if (lane == 0) s_wsum[warp] = mine;
        __syncthreads();
        uint32_t run = 0;
#pragma unroll
        for (int w = 0; w < NW; ++w)
            if (w < (int)warp) run += s_wsum[w];
#pragma unroll
        for (int q = 0; q < PER; ++q) {
            const uint32_t p = p0 + 32 * q;
            if (p < P) hs[p] = (uint16_t)(run + __popc(bal[q] & (le >> 1)));
            run += __popc(bal[q]);
        }
        if (warp == NW - 1 && lane == 0) s_wsum[NW] = run;  // all heads
        __syncthreads();

        if (!NUMERIC) {
            const uint32_t all = s_wsum[NW];
            for (uint32_t k = tid; k < nr; k += T)
                if (k == rf[k]) {
                    const uint32_t e = off[re[k]];
                    a.row_nnz[rrow[k]] = (e < P ? hs[e] : all) - hs[off[k]];
                }
        } else {
            // every entry's product and its rounding error, in merged order
            float pr[PER], pe[PER];
#pragma unroll
            for (int q = 0; q < PER; ++q) {
                const uint32_t p = p0 + 32 * q;
                pr[q] = pe[q] = 0.f;
                if (p < P) {
                    const uint32_t id = pid[p], w = id >> 5;
                    const uint32_t kr = spre[w] + __popc(sbits[w] & (0xffffffffu >> (31 - (id & 31)))) - 1;
                    const float xf = xv[kr], yf = yv[id];
                    pr[q] = xf * yf;
                    pe[q] = fmaf(xf, yf, -pr[q]);
                }
            }
            __syncthreads();  // xv and yv are read
            float *spr = xv, *spe = yv;
#pragma unroll
            for (int q = 0; q < PER; ++q) {
                const uint32_t p = p0 + 32 * q;
                if (p < P) {
                    spr[p] = pr[q];
                    spe[p] = pe[q];
                }
            }
            __syncthreads();
            // a head sums its entries and writes the output
#pragma unroll
            for (int q0 = 0; q0 < PER; q0 += 4) {
                uint64_t o[4], out[4];
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    const int q = q0 + v;
                    const uint32_t p = p0 + 32 * q;
                    o[v] = ~0ull;
                    out[v] = 0;
                    if ((bal[q] >> lane) & 1u) {
                        const uint32_t k = kk[q], row = rrow[k];
                        o[v] = a.row_off[row] - a.chunk_base + (uint32_t)(hs[p] - hs[off[rf[k]]]);
                        int y_nfbits;
                        const uint64_t *cols;
                        uint32_t ncols;
                        row_job_params(a, row, y_nfbits, cols, ncols);
                        out[v] = shl(a.row_xf[row], y_nfbits) | cols[key[p]];
                    }
                }
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    const int q = q0 + v;
                    const uint32_t p = p0 + 32 * q;
                    if (!((bal[q] >> lane) & 1u)) continue;
                    const uint32_t end = off[re[kk[q]]], rk = key[p];
                    float sum = pr[q], c = pe[q];
                    for (uint32_t e = p + 1; e < end && key[e] == rk; ++e) {
                        float ns, err;
                        two_sum(sum, spr[e], ns, err);
                        sum = ns;
                        c += err + spe[e];
                    }
                    if (o[v] < a.out_cap) {
                        a.out_keys[o[v]] = out[v];
                        a.out_vals[o[v]] = sum + c;
                    } else {
                        atomicOr(a.err, 4u);
                    }
                }
            }
        }
        __syncthreads();
    }
}

template <int C>
size_t light_smem(bool numeric) {
    // key, rrow, rj0 | sbits | pid, off, rf, re, spre | xv, yv
    return (size_t)C * 12 + C / 8 + 2 * ((size_t)4 * C + 2 + C / 32 + ((C / 32) & 1)) +
           (numeric ? (size_t)C * 8 : 0);
}

template <bool NUMERIC, int C>
void launch_light_as(const AccArgs &a, int grid, cudaStream_t s) {
    const size_t sm = light_smem<C>(NUMERIC);
    GS_CUDA(cudaFuncSetAttribute(k_light<NUMERIC, C>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    k_light<NUMERIC, C><<<grid, LightShape<C>::T, sm, s>>>(a);
}

}  // namespace

int light_blocks_per_sm() { return 4; }

// a.light_cap products at most in a unit: the capacity the planner packed for.
void launch_light(const AccArgs &a, bool numeric, int grid, cudaStream_t s) {
    if (a.nunits == 0) return;
    if (a.light_cap <= (uint32_t)kLightCap / 2) {
        if (numeric)
            launch_light_as<true, kLightCap / 2>(a, grid, s);
        else
            launch_light_as<false, kLightCap / 2>(a, grid, s);
    } else {
        if (numeric)
            launch_light_as<true, kLightCap>(a, grid, s);
        else
            launch_light_as<false, kLightCap>(a, grid, s);
    }
    count_launch();
    GS_CUDA(cudaGetLastError());
}

}  // namespace gs
