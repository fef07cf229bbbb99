// scan.cuh -- one-kernel prefix sums for the planning kernels.
//
// A CTA takes the next tile of kScanTile items from a ticket (so every tile
// before it belongs to a CTA that is already running), scans its items on
// chip and finds what the tiles before it add up to by a decoupled look-back:
// every tile publishes its own sums, then its inclusive sums; a warp reads the
// published words of 32 tiles at a time until it meets an inclusive one.  So a
// planning step that computes per-item values, their prefix sums and the
// lists that follow from them is one launch and one pass over its inputs.
//
// The waits are on tiles whose CTAs are resident and publish before they wait,
// so every wait ends; it is bounded all the same (kScanPolls), and one that
// runs out sets bit 8 of the error word, on which this tile and every later
// one return without writing (kernels that follow in the stream check the bit).
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

namespace gs {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;  // consecutive items of a thread
constexpr int kScanTile = kScanThreads * kScanItems;
constexpr uint32_t kScanPolls = 1u << 20;
constexpr unsigned int kScanErr = 8u;

inline uint64_t scan_tiles(uint64_t n) { return (n + kScanTile - 1) / kScanTile; }

// Words of a scan of at most n items: flags (zero at launch) and values.
inline uint64_t scan_flag_words(uint64_t n) { return 1 + scan_tiles(n); }
constexpr int kMaxScanSums = 5;  // sums of one scan (V) at most
template <int V>
uint64_t scan_value_words(uint64_t n) {
    return 2 * V * scan_tiles(n);
}

// flag[0] is the ticket, flag[1 + t] tile t's state (0 nothing, 1 its own sums
// at val[2 t V], 2 also the inclusive sums at val[(2 t + 1) V]).
struct ScanState {
    uint32_t *flag;
    uint64_t *val;
    unsigned int *err;
};

#ifdef __CUDACC__

namespace dev {

static __device__ __forceinline__ uint32_t ld_acquire(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

static __device__ __forceinline__ void st_release(uint32_t *p, uint32_t v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// One warp: excl = the sums of every tile before `tile`, whose own sums are
// tot (the same in every lane).  False when a wait ran out.
template <int V>
__device__ __forceinline__ bool look_back(const ScanState &st, uint32_t tile, const uint64_t (&tot)[V],
                                          uint64_t (&excl)[V]) {
    static_assert(V <= kMaxScanSums, "the sums of a tile fit the buffer");
    const uint32_t lane = threadIdx.x & 31;
#pragma unroll
    for (int v = 0; v < V; ++v) excl[v] = 0;
    uint64_t *mine = st.val + 2ull * V * tile;
    if (tile > 0) {
        if (lane == 0) {
#pragma unroll
            for (int v = 0; v < V; ++v) mine[v] = tot[v];
            st_release(st.flag + 1 + tile, 1u);
        }
        uint32_t polls = 0;
        for (int64_t base = (int64_t)tile - 1; base >= 0;) {
            const int64_t t = base - lane;
            const uint32_t f = t < 0 ? 2u : ld_acquire(st.flag + 1 + t);
            if (__any_sync(0xffffffffu, f == 0)) {
                unsigned int e = 0;
                if (lane == 0) e = (++polls > kScanPolls) ? atomicOr(st.err, kScanErr) | kScanErr : ld_acquire(st.err);
                if (__shfl_sync(0xffffffffu, e, 0) & kScanErr) return false;
                __nanosleep(32);
                continue;
            }
            const uint32_t inclusive = __ballot_sync(0xffffffffu, f == 2u);
            const uint32_t last = inclusive ? __ffs(inclusive) - 1 : 31;
#pragma unroll
            for (int v = 0; v < V; ++v) {
                uint64_t x = (lane <= last && t >= 0) ? __ldcg(st.val + (2 * t + (f == 2u)) * V + v) : 0ull;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
                excl[v] += x;
            }
            if (inclusive) break;
            base -= 32;
        }
    }
    if (lane == 0) {
#pragma unroll
        for (int v = 0; v < V; ++v) mine[V + v] = excl[v] + tot[v];
        st_release(st.flag + 1 + tile, 2u);
    }
    return true;
}

template <int V>
struct ScanShared {
    uint64_t warp[kScanThreads / 32][V];
    uint64_t base[V], through[V];
    uint32_t tile, ok;
};

// The CTA's next tile (all threads).
template <int V>
__device__ __forceinline__ uint32_t next_tile(const ScanState &st, ScanShared<V> &sh) {
    if (threadIdx.x == 0) sh.tile = atomicAdd(st.flag, 1u);
    __syncthreads();
    return sh.tile;
}

// x: this thread's sums; becomes the sums of every item before this thread's
// first one.  sh.through: the sums up to the end of the tile.
template <int V>
__device__ __forceinline__ bool tile_scan(const ScanState &st, ScanShared<V> &sh, uint32_t tile, uint64_t (&x)[V]) {
    constexpr int NW = kScanThreads / 32;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint64_t inc[V];
#pragma unroll
    for (int v = 0; v < V; ++v) {
        inc[v] = x[v];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint64_t y = __shfl_up_sync(0xffffffffu, inc[v], o);
            if (lane >= (uint32_t)o) inc[v] += y;
        }
        if (lane == 31) sh.warp[warp][v] = inc[v];
    }
    __syncthreads();
    if (warp == 0) {
        uint64_t tot[V], excl[V];
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const uint64_t w = lane < NW ? sh.warp[lane][v] : 0ull;
            uint64_t y = w;
#pragma unroll
            for (int o = 1; o < NW; o <<= 1) {
                const uint64_t z = __shfl_up_sync(0xffffffffu, y, o);
                if (lane >= (uint32_t)o) y += z;
            }
            tot[v] = __shfl_sync(0xffffffffu, y, NW - 1);
            if (lane < NW) sh.warp[lane][v] = y - w;
        }
        const bool ok = look_back<V>(st, tile, tot, excl);
        if (lane == 0) {
            sh.ok = ok;
#pragma unroll
            for (int v = 0; v < V; ++v) {
                sh.base[v] = excl[v];
                sh.through[v] = excl[v] + tot[v];
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int v = 0; v < V; ++v) x[v] = sh.base[v] + sh.warp[warp][v] + inc[v] - x[v];
    return sh.ok;
}

}  // namespace dev

#endif

}  // namespace gs
