// Block scans and decoupled look-back, shared by the kernels that scan in one launch.
#pragma once

#include <cuda_runtime.h>

#include "gbh_internal.cuh"

namespace gbh {

// Records a device-side consistency failure (checked by the host after the call).
__device__ __forceinline__ void dev_error(DevInfo *info, int where) {
    atomicExch(&info->err, 1);
    info->err_where = where;
}

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// Block-wide exclusive scan of one value per thread (kBlock threads, at most 1,024); s_warp holds
// kBlock / 32 + 1 words. Returns the exclusive prefix and the total.
template <int kBlock>
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t *s_warp, uint32_t &total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t incl = warp_incl_scan(v);
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        const uint32_t w = lane < (kBlock / 32) ? s_warp[lane] : 0;
        const uint32_t wi = warp_incl_scan(w);
        if (lane < (kBlock / 32)) s_warp[lane] = wi - w;
        if (lane == (kBlock / 32) - 1) s_warp[kBlock / 32] = wi;
    }
    __syncthreads();
    const uint32_t r = s_warp[warp] + incl - v;
    total = s_warp[kBlock / 32];
    __syncthreads();
    return r;
}

// Polls of a look-back wait before the block gives up and records an error: far beyond any wait of a
// running predecessor.
constexpr int kLbSpinLimit = 1 << 22;

// Look-back words are read and written whole (value and flag in one word); nothing else is passed
// through them, so volatile (uncached, untorn) accesses suffice.
__device__ __forceinline__ unsigned long long ld_volatile64(const unsigned long long *p) {
    return *reinterpret_cast<const volatile unsigned long long *>(p);
}
__device__ __forceinline__ void st_volatile64(unsigned long long *p, unsigned long long v) {
    *reinterpret_cast<volatile unsigned long long *>(p) = v;
}

// Look-back of one tile, called by one warp: publishes the tile's sum, then reads its predecessors'
// words 32 at a time (lane j the (j+1)-th tile back) and adds them down to the nearest published
// prefix, publishes its own inclusive prefix and returns the exclusive one (all lanes). Tiles are
// taken in counter order, so every tile a block waits for belongs to a block that is already
// running, and the first tile never waits; past kLbSpinLimit polls the warp records an error
// (reported as GBH_ERR_LIMIT) and publishes what it has, so that its successors are not held.
// status: one 64-bit word per tile (flag in the top 2 bits), zero at the start.
__device__ __forceinline__ unsigned long long look_back(unsigned long long *status, uint32_t tile,
                                                        unsigned long long total, DevInfo *info) {
    constexpr unsigned long long kAgg = 1ull << 62, kPre = 2ull << 62, kVal = (1ull << 62) - 1;
    const int lane = threadIdx.x & 31;
    unsigned long long excl = 0;
    if (tile == 0) {
        if (lane == 0) st_volatile64(status, kPre | total);
        return 0;
    }
    if (lane == 0) st_volatile64(status + tile, kAgg | total);
    int64_t t = int64_t(tile) - 1;
    int spins = 0;
    bool bad = false;
    for (;;) {
        const int64_t idx = t - lane;
        unsigned long long w = idx >= 0 ? ld_volatile64(status + idx) : kPre;  // before tile 0: prefix 0
        // every word up to the nearest prefix must be published; wait for the others
        for (;;) {
            const unsigned pre = __ballot_sync(0xffffffffu, (w >> 62) == 2);
            const unsigned upto = pre ? (pre & (0u - pre)) * 2u - 1u : 0xffffffffu;  // lanes to the first prefix
            const unsigned wait = __ballot_sync(0xffffffffu, !(w >> 62)) & upto;
            if (!wait) break;
            if (++spins > kLbSpinLimit) {
                bad = true;
                break;
            }
            if ((wait >> lane) & 1u) w = ld_volatile64(status + idx);
        }
        if (bad) break;
        const unsigned pre = __ballot_sync(0xffffffffu, (w >> 62) == 2);
        const unsigned upto = pre ? (pre & (0u - pre)) * 2u - 1u : 0xffffffffu;
        unsigned long long v = ((upto >> lane) & 1u) ? (w & kVal) : 0ull;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        excl += v;
        if (pre) break;
        t -= 32;
    }
    if (lane == 0) {
        if (bad) dev_error(info, kErrScanWait);
        st_volatile64(status + tile, kPre | ((excl + total) & kVal));
    }
    return excl;
}

// Words of a look-back scan over `tiles` tiles: the tile counter (in two words), then the tiles'.
__host__ __device__ inline int64_t lb_words_of(int64_t tiles) { return 2 + 2 * tiles; }

}  // namespace gbh
