// sort.cu — the collect, key and sort stages of the tree build (build.go:11-41, 62-113,
// morton.go:7-49), and the Morton order for callers without device allocation.
//
// Compiled with -fmad=false like tree.cu: the root cube and the keys are bit identical to the
// reference's. The reference sorts stably by 63-bit Morton key, so (key, state index) is a strict
// order and any sort by it gives the reference's order:
//   k_bbox                 root cube of the stars (one launch; the last block to finish reduces)
//   k_tile_sort            a block takes 1,024 bodies: keys, star count, a bitonic sort in registers
//   k_merge, 1 to L times  up to 16 sorted runs merged at once: every element's place is its place
//                          in its own run plus what binary searches find before it in the others;
//                          the last merge also writes the sorted copies (build.go:34-41)
// Runs hold alive non-hole bodies only: a tile's dead bodies and holes sort behind its stars and
// drop out, so no separate scan compacts them. 16,384 bodies sort in 2 launches, 147,456 in 3; plain
// states of more than 786,432 take radix passes (kMergeTiles), 3 launches each.
//
// Forests: tiles never straddle systems, and runs merge only within their system, so (system, key)
// order needs no extra passes.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>

#include "gbh_internal.cuh"
#include "lookback.cuh"

namespace gbh {

namespace {

constexpr int kThreads = 256;
constexpr int kPer = kSortTile / kThreads;  // elements a thread
static_assert(kPer == 4, "the bitonic stages below");
constexpr int kMaxWay = 16;                 // runs merged at once
constexpr int kBboxBlocks = 1024;
constexpr int kPartWords = 7;               // per block: 3 minima, 3 maxima, any star
constexpr unsigned kFull = 0xffffffffu;

inline unsigned blocks_for(int64_t n, int threads) {
    int64_t b = (n + threads - 1) / threads;
    return unsigned(b < 1 ? 1 : b);
}

__device__ __forceinline__ bool is_star(uint8_t alive, uint8_t kind) { return alive && kind != GBH_BLACK_HOLE; }

// Order-preserving map of a double to a signed 64-bit integer (an involution): min and max of
// the keys are the keys of the min and max, computed on the integer ALU instead of the slow
// FP64 pipe. (-0 orders before +0; the coordinates are not NaN.)
__device__ __forceinline__ long long ord_key(double v) {
    long long b = __double_as_longlong(v);
    return b ^ ((b >> 63) & 0x7fffffffffffffffll);
}
__device__ __forceinline__ double ord_val(long long k) { return __longlong_as_double(k ^ ((k >> 63) & 0x7fffffffffffffffll)); }

// Minima mn and maxima mx over the block, in thread 0 .. 5 of the result array (min x y z, max x y z).
__device__ __forceinline__ void block_minmax(long long mn[3], long long mx[3], long long out[6]) {
    __shared__ long long s[6][kThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        for (int o = 16; o > 0; o >>= 1) {
            mn[c] = min(mn[c], __shfl_xor_sync(kFull, mn[c], o));
            mx[c] = max(mx[c], __shfl_xor_sync(kFull, mx[c], o));
        }
        if (lane == 0) {
            s[c][warp] = mn[c];
            s[3 + c][warp] = mx[c];
        }
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        long long v = s[threadIdx.x][0];
        for (int w = 1; w < kThreads / 32; ++w) v = threadIdx.x < 3 ? min(v, s[threadIdx.x][w]) : max(v, s[threadIdx.x][w]);
        out[threadIdx.x] = v;
    }
    __syncthreads();
}

// One body's part of a bounding box. A non-finite coordinate of a star makes the box non-finite by
// itself (NaN and infinities map to keys beyond every finite one); a non-finite mass is folded in
// as the key of a NaN, so that the input can be rejected before keys are formed (collect,
// build.go:62-113, would carry a NaN into the root cube and every key).
__device__ __forceinline__ void add_star(long long mn[3], long long mx[3], double vx, double vy, double vz, bool bad_mass) {
    const long long x = ord_key(vx), y = ord_key(vy), z = ord_key(vz);
    mn[0] = min(mn[0], x);
    mx[0] = max(mx[0], bad_mass ? LLONG_MAX : x);
    mn[1] = min(mn[1], y);
    mx[1] = max(mx[1], y);
    mn[2] = min(mn[2], z);
    mx[2] = max(mx[2], z);
}

// Root cube (build.go:19-21): side = max(max extent * (1+1e-9), 1e-12), scale = 2^21 / side, and its
// FP32 views; called by one warp, lane L forms the opening base 2 half_L / theta of level L
// (half_L = side / 2^(L+1): halving is exact, so one exact scaling gives it). `geo` may be null.
__device__ __forceinline__ void root_cube(const double mn[3], const double mx[3], double theta, int lane, SysGeo *geo,
                                          DevInfo *info) {
    double side = fmax(mx[0] - mn[0], fmax(mx[1] - mn[1], mx[2] - mn[2]));
    side = fmax(side * (1 + 1e-9), 1e-12);
    if (lane <= kMaxLevel) {
        const float base = __double2float_rn(2 * ldexp(side, -(lane + 1)) / theta);
        if (info) info->crit_base[lane] = base;
        if (geo) geo->crit_base[lane] = base;
    }
    if (lane != 0) return;
    float hi[3], lo[3];
    for (int c = 0; c < 3; ++c) {
        hi[c] = __double2float_rn(mn[c]);
        lo[c] = __double2float_rn(mn[c] - double(hi[c]));
    }
    const float sh = __double2float_rn(side), sl = __double2float_rn(side - double(sh));
    const double scale = double(1 << kMortonBits) / side;
    if (info) {
        info->minx = mn[0];
        info->miny = mn[1];
        info->minz = mn[2];
        info->side = side;
        info->scale = scale;
        for (int c = 0; c < 3; ++c) {
            info->min_hi[c] = hi[c];
            info->min_lo[c] = lo[c];
        }
        info->side_hi = sh;
        info->side_lo = sl;
    }
    if (geo) {
        geo->minx = mn[0];
        geo->miny = mn[1];
        geo->minz = mn[2];
        geo->side = side;
        geo->scale = scale;
        for (int c = 0; c < 3; ++c) {
            geo->min_hi[c] = hi[c];
            geo->min_lo[c] = lo[c];
        }
        geo->side_hi = sh;
        geo->side_lo = sl;
    }
}

__device__ __forceinline__ bool finite3(const double v[3]) { return isfinite(v[0]) && isfinite(v[1]) && isfinite(v[2]); }

// The build's first kernel: bounding box of the stars, alive holes' accelerations zeroed
// (bh.go:99-101), the error record and the look-back words `lb` of the build's later scans cleared.
// The last block to finish (a counter that wraps to 0 by itself) reduces the blocks' parts (min and
// max are exact, so their order does not matter) and forms the root cube.
__global__ __launch_bounds__(kThreads) void k_bbox(int64_t n, const double *__restrict__ px,
                                                   const double *__restrict__ py, const double *__restrict__ pz,
                                                   const double *__restrict__ mass, const uint8_t *__restrict__ kind,
                                                   const uint8_t *__restrict__ alive, double theta, long long *part,
                                                   double *ax, double *ay, double *az, uint32_t *lb, int64_t lb_words,
                                                   DevInfo *info, SysGeo *geo) {
    pdl_begin();
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        info->err = 0;
        info->err_where = 0;
        info->nstars = 0;
        info->nnodes = 0;
        info->work = 0;
        info->nleaves = 0;
        info->ntargets = 0;
        info->theta = theta;
    }
    const int64_t stride = int64_t(gridDim.x) * kThreads, t0 = int64_t(blockIdx.x) * kThreads + threadIdx.x;
    for (int64_t w = t0; w < lb_words; w += stride) lb[w] = 0;
    long long mn[3] = {LLONG_MAX, LLONG_MAX, LLONG_MAX}, mx[3] = {LLONG_MIN, LLONG_MIN, LLONG_MIN};
    bool any = false;
    for (int64_t i = t0; i < n; i += stride) {
        const uint8_t al = alive ? alive[i] : 1, kd = kind ? kind[i] : 0;
        if (is_star(al, kd)) {
            any = true;
            add_star(mn, mx, px[i], py[i], pz[i], mass && !isfinite(mass[i]));
        } else if (ax && al && kd == GBH_BLACK_HOLE) {
            ax[i] = 0;
            ay[i] = 0;
            az[i] = 0;
        }
    }
    __shared__ long long box[6];
    __shared__ bool s_last;
    any = __syncthreads_or(any);
    block_minmax(mn, mx, box);
    if (threadIdx.x < 6) part[blockIdx.x * kPartWords + threadIdx.x] = box[threadIdx.x];
    if (threadIdx.x == 6) part[blockIdx.x * kPartWords + 6] = any;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicInc(&info->bbox_done, gridDim.x - 1) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    any = false;
    for (int c = 0; c < 3; ++c) {
        mn[c] = LLONG_MAX;
        mx[c] = LLONG_MIN;
    }
    for (unsigned b = threadIdx.x; b < gridDim.x; b += kThreads) {
        const long long *q = part + b * kPartWords;
        for (int c = 0; c < 3; ++c) {
            mn[c] = min(mn[c], __ldcg(q + c));
            mx[c] = max(mx[c], __ldcg(q + 3 + c));
        }
        any |= __ldcg(q + 6) != 0;
    }
    any = __syncthreads_or(any);
    block_minmax(mn, mx, box);
    if (threadIdx.x >= 32) return;
    double lo[3], hi[3];
    for (int c = 0; c < 3; ++c) {
        lo[c] = ord_val(box[c]);
        hi[c] = ord_val(box[3 + c]);
    }
    root_cube(lo, hi, theta, threadIdx.x, geo, info);
    if (threadIdx.x == 0 && any && !(finite3(lo) && finite3(hi))) dev_error(info, kErrNonFinite);  // GBH_ERR_ARG
}

// ---------------------------------------------------------------- forests

__global__ void k_sys_init(int32_t nsys, SysGeo *geo, DevInfo *info, double theta, uint32_t *lb, int64_t lb_words) {
    pdl_begin();
    const int32_t s = int32_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    for (int64_t w = s; w < lb_words; w += stride) lb[w] = 0;
    if (s == 0) {
        info->err = 0;
        info->err_where = 0;
        info->nnodes = 0;
        info->work = 0;
        info->nleaves = 0;
        info->ntargets = 0;
        info->theta = theta;
    }
    if (s >= nsys) return;
    for (int c = 0; c < 3; ++c) {
        geo[s].kmin[c] = LLONG_MAX;
        geo[s].kmax[c] = LLONG_MIN;
    }
    geo[s].star_hi = 0;  // k_tile_sort counts the system's stars here
}

// Each system's bounding box, a tile a block (a tile lies in one system), alive holes zeroed.
__global__ __launch_bounds__(kThreads) void k_bbox_sys(const int4 *__restrict__ tiles,
                                                       const int64_t *__restrict__ sys_off,
                                                       const double *__restrict__ px, const double *__restrict__ py,
                                                       const double *__restrict__ pz, const double *__restrict__ mass,
                                                       const uint8_t *__restrict__ kind,
                                                       const uint8_t *__restrict__ alive, SysGeo *geo, double *ax,
                                                       double *ay, double *az) {
    pdl_begin();
    const int4 t = tiles[blockIdx.x];
    const int64_t end = min(int64_t(t.x) + kSortTile, sys_off[t.y + 1]);
    long long mn[3] = {LLONG_MAX, LLONG_MAX, LLONG_MAX}, mx[3] = {LLONG_MIN, LLONG_MIN, LLONG_MIN};
    for (int64_t i = int64_t(t.x) + threadIdx.x; i < end; i += kThreads) {
        const uint8_t al = alive ? alive[i] : 1, kd = kind ? kind[i] : 0;
        if (is_star(al, kd)) {
            add_star(mn, mx, px[i], py[i], pz[i], mass && !isfinite(mass[i]));
        } else if (al && kd == GBH_BLACK_HOLE) {
            ax[i] = 0;
            ay[i] = 0;
            az[i] = 0;
        }
    }
    __shared__ long long box[6];
    block_minmax(mn, mx, box);
    if (threadIdx.x < 3) atomicMin(&geo[t.y].kmin[threadIdx.x], box[threadIdx.x]);
    else if (threadIdx.x < 6) atomicMax(&geo[t.y].kmax[threadIdx.x - 3], box[threadIdx.x]);
}

// Per system (a warp each): root cube, FP32 views, opening bases.
__global__ void k_sys_cube(int32_t nsys, double theta, SysGeo *geo) {
    pdl_begin();
    const int32_t s = int32_t(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (s >= nsys) return;
    double mn[3], mx[3];
    for (int c = 0; c < 3; ++c) {
        mn[c] = ord_val(geo[s].kmin[c]);
        mx[c] = ord_val(geo[s].kmax[c]);
    }
    root_cube(mn, mx, theta, threadIdx.x & 31, geo + s, nullptr);
}

// Star ranges of the systems (exclusive scan of their star counts) and the gsize-star groups of the
// mixed walk, which never straddle two systems. One block, 1,024 systems at a time.
constexpr int kSysScan = 1024;
__global__ __launch_bounds__(kSysScan) void k_sys_ranges(int32_t nsys, int32_t gsize, SysGeo *geo, DevInfo *info) {
    pdl_begin();
    __shared__ uint32_t s_w[2][32];
    __shared__ uint32_t s_run[2];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x < 2) s_run[threadIdx.x] = 0;
    for (int32_t s0 = 0; s0 < nsys; s0 += kSysScan) {
        const int32_t s = s0 + threadIdx.x;
        const uint32_t cnt = s < nsys ? uint32_t(geo[s].star_hi) : 0u;
        const uint32_t ng = (cnt + uint32_t(gsize) - 1) / uint32_t(gsize);
        const uint32_t ia = warp_incl_scan(cnt), ib = warp_incl_scan(ng);
        if (lane == 31) {
            s_w[0][warp] = ia;
            s_w[1][warp] = ib;
        }
        __syncthreads();
        if (warp < 2) {
            const uint32_t w = s_w[warp][lane];
            s_w[warp][lane] = warp_incl_scan(w) - w;
        }
        __syncthreads();
        const uint32_t lo = s_run[0] + s_w[0][warp] + ia - cnt, g = s_run[1] + s_w[1][warp] + ib - ng;
        __syncthreads();
        if (threadIdx.x == kSysScan - 1) {
            s_run[0] = lo + cnt;
            s_run[1] = g + ng;
        }
        if (s < nsys) {
            geo[s].star_lo = int32_t(lo);
            geo[s].star_hi = int32_t(lo + cnt);
            geo[s].group_lo = int32_t(g);
            geo[s].ngroups = int32_t(ng);
            if (cnt) {  // an empty system keeps its initial keys (a NaN box); one with stars must be finite
                double mn[3], mx[3];
                for (int c = 0; c < 3; ++c) {
                    mn[c] = ord_val(geo[s].kmin[c]);
                    mx[c] = ord_val(geo[s].kmax[c]);
                }
                if (!(finite3(mn) && finite3(mx))) dev_error(info, kErrNonFinite);
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        info->nstars = s_run[0];
        info->ngroups = s_run[1];
    }
}

// ---------------------------------------------------------------- keys

// morton.go:7-15.
__device__ __forceinline__ uint64_t spread(uint64_t v) {
    v &= (uint64_t(1) << kMortonBits) - 1;
    v = (v | v << 32) & 0x1f00000000ffffull;
    v = (v | v << 16) & 0x1f0000ff0000ffull;
    v = (v | v << 8) & 0x100f00f00f00f00full;
    v = (v | v << 4) & 0x10c30c30c30c30c3ull;
    v = (v | v << 2) & 0x1249249249249249ull;
    return v;
}

// cell(), build.go:23-25: uint64(min(2^21-1, max(0, (v-lo)*scale))), the limits applied to the
// truncated integer (the same cells; two FP64 operations instead of six).
__device__ __forceinline__ uint64_t cell(double v, double lo, double scale) {
    const int t = __double2int_rz((v - lo) * scale);
    return uint64_t(min((1 << kMortonBits) - 1, max(0, t)));
}

// ---------------------------------------------------------------- sort

// A tile is 1,024 bodies of one system: (first body, system, the system's first tile, its tiles).
// A plain state's tiles follow from the index.
template <bool kForest>
__device__ __forceinline__ int4 tile_at(const int4 *__restrict__ tiles, int32_t t, int32_t ntiles) {
    return kForest ? tiles[t] : make_int4(t * kSortTile, 0, 0, ntiles);
}

// Compare-exchange of two values: (a, b) ascending when up.
__device__ __forceinline__ void exchange(uint64_t &a, uint64_t &b, bool up) {
    const bool swap = (a > b) == up;
    const uint64_t t = swap ? b : a;
    b = swap ? a : b;
    a = t;
}

// Bitonic sort of the block's kSortTile distinct values, 4 a thread (value 4 t + j is e[j] of thread
// t): strides below 4 in registers, up to 64 by shuffles, the 6 stages beyond through shared memory.
__device__ __forceinline__ void bitonic_sort(uint64_t (&e)[kPer], uint64_t *s_e) {
    const int t = threadIdx.x;
#pragma unroll
    for (int size = 2; size <= kSortTile; size <<= 1) {
#pragma unroll
        for (int s = size >> 1; s > 0; s >>= 1) {
            const bool keep_min = ((4 * t & s) == 0) == ((4 * t & size) == 0);
            if (s >= 128) {  // the partner is in another warp
#pragma unroll
                for (int j = 0; j < kPer; ++j) s_e[j * kThreads + t] = e[j];
                __syncthreads();
#pragma unroll
                for (int j = 0; j < kPer; ++j) {
                    const uint64_t o = s_e[j * kThreads + (t ^ (s >> 2))];
                    if ((e[j] > o) == keep_min) e[j] = o;
                }
                __syncthreads();
            } else if (s >= 4) {
#pragma unroll
                for (int j = 0; j < kPer; ++j) {
                    const uint64_t o = __shfl_xor_sync(kFull, e[j], s >> 2);
                    if ((e[j] > o) == keep_min) e[j] = o;
                }
            } else if (s == 2) {
                const bool up = (4 * t & size) == 0;
                exchange(e[0], e[2], up);
                exchange(e[1], e[3], up);
            } else {
                exchange(e[0], e[1], size == 2 ? true : (4 * t & size) == 0);
                exchange(e[2], e[3], size == 2 ? false : (4 * t & size) == 0);
            }
        }
    }
}

// Keys of a tile's bodies, sorted by (key, state index), its stars in front. The network sorts one
// 64-bit word an element: 0, the key's upper 53 bits (down to the second axis of level 18 of 21) and
// the slot in the tile, which settles equal keys by state index; dead bodies, holes and slots beyond
// the tile have the top bit set, above every star (a star in the root cube's highest corner has a key
// of all ones). Where neighbours agree in all 53 bits (levels 18 to 21 tell them apart, if
// anything) each such run is then put in order by the whole key: short runs by counting, a tile with a
// longer one (a cluster far tighter than the rest, coincident stars) by the network once more. Against
// (key, index) pairs of three registers: 16,384 bodies 16.6 -> 11.6 us, the 1.1M-body forest 57 -> 40
// (ncu, cold caches).
// 1,024 bodies a tile spread a small state over more SMs than 2,048 would, and a million
// bodies are 6.7 tiles a SM. pos4 (may be null): each star's position and mass in one record, for
// the last merge's reads through the order.
constexpr int kSlotBits = 10;
constexpr uint64_t kNoStar = uint64_t(1) << 63;
// Runs of more stars than this take the network. 16,384 stars in clusters of 8: 80.5 us a build either
// way, of 16 85 by counting and 80.6 by the network, of 128 213 and 146, of 512 387 and 198 (clusters 1e-7
// of the whole wide; by radix passes, without tiles, 163, 163, 221 and 288).
constexpr int kRankRun = 8;
static_assert(kSortTile == 1 << kSlotBits, "a word holds the slot");
template <bool kForest>
__global__ __launch_bounds__(kThreads) void k_tile_sort(int64_t n, const int4 *__restrict__ tiles, int32_t ntiles,
                                                        const int64_t *__restrict__ sys_off,
                                                        const double *__restrict__ px, const double *__restrict__ py,
                                                        const double *__restrict__ pz,
                                                        const double *__restrict__ mass,
                                                        const uint8_t *__restrict__ kind,
                                                        const uint8_t *__restrict__ alive, SysGeo *geo,
                                                        uint64_t *__restrict__ keys, int32_t *__restrict__ order,
                                                        int32_t *__restrict__ tile_len, Pos4 *__restrict__ pos4,
                                                        DevInfo *info) {
    pdl_begin();
    __shared__ uint64_t s_key[kSortTile];  // by slot
    __shared__ uint64_t s_e[kSortTile + 1];
    const int t = threadIdx.x;
    const int4 tile = tile_at<kForest>(tiles, blockIdx.x, ntiles);
    const int64_t start = kForest ? int64_t(tile.x) : int64_t(blockIdx.x) * kSortTile;
    const int64_t end = kForest ? min(start + kSortTile, sys_off[tile.y + 1]) : min(start + kSortTile, n);
    const double minx = kForest ? geo[tile.y].minx : info->minx, miny = kForest ? geo[tile.y].miny : info->miny,
                 minz = kForest ? geo[tile.y].minz : info->minz, sc = kForest ? geo[tile.y].scale : info->scale;
    uint64_t e[kPer];
    int cnt = 0;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        const int slot = j * kThreads + t;
        const int64_t i = start + slot;
        uint64_t k = ~0ull;
        bool star = false;
        if (i < end) {
            const double x = px[i], y = py[i], z = pz[i], m = mass ? mass[i] : 0.0;
            star = is_star(alive ? alive[i] : 1, kind ? kind[i] : 0);
            if (star && pos4) pos4[i] = Pos4{x, y, z, m};
            if (star) k = spread(cell(x, minx, sc)) << 2 | spread(cell(y, miny, sc)) << 1 | spread(cell(z, minz, sc));
        }
        s_key[slot] = k;
        // a key has 63 bits: its upper 53 in bits 10 to 62, bit 63 for what is no star
        e[j] = (star ? k >> kSlotBits << kSlotBits : kNoStar) | uint64_t(slot);
        cnt += __syncthreads_count(star);
    }
    bool tie = false;
    for (int pass = 0;; ++pass) {
        bitonic_sort(e, s_e);
#pragma unroll
        for (int j = 0; j < kPer; ++j) s_e[4 * t + j] = e[j];
        if (t == 0) s_e[kSortTile] = ~0ull;
        __syncthreads();
        if (pass == 1) break;
        // whether the places p and p + d hold stars of equal words
        auto equal = [&](int p, int d) { return p + d < cnt && s_e[p] >> kSlotBits == s_e[p + d] >> kSlotBits; };
        bool many = false;
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            tie |= equal(4 * t + j, 1);
            many |= equal(4 * t + j, kRankRun);
        }
        tie = __syncthreads_or(tie);
        if (!tie || !__syncthreads_or(many)) break;
        // long runs: the network again, by (the run's first place, the key's lower bits, slot)
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const int p = 4 * t + j;
            if (p >= cnt) continue;  // behind the stars already
            int lo = 0, hi = p;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (s_e[mid] >> kSlotBits < e[j] >> kSlotBits) lo = mid + 1;
                else hi = mid;
            }
            const int slot = int(e[j] & (kSortTile - 1));
            e[j] = uint64_t(lo) << 2 * kSlotBits | (s_key[slot] & (kSortTile - 1)) << kSlotBits | uint64_t(slot);
        }
        tie = false;
        __syncthreads();
    }
    if (tie) {
        // rank every element of a run of equal words by its whole key and slot (a run of m takes m
        // steps a thread, at most kRankRun)
        int rank[kPer];
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const int p = 4 * t + j;
            rank[j] = p;
            if (p < cnt) {
                const uint64_t w = e[j] >> kSlotBits, k = s_key[e[j] & (kSortTile - 1)];
                for (int q = p - 1; q >= 0 && (s_e[q] >> kSlotBits) == w; --q)
                    if (s_key[s_e[q] & (kSortTile - 1)] > k) --rank[j];
                for (int q = p + 1; q < cnt && (s_e[q] >> kSlotBits) == w; ++q)
                    if (s_key[s_e[q] & (kSortTile - 1)] < k) ++rank[j];
            }
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kPer; ++j) s_e[rank[j]] = e[j];
        __syncthreads();
    }
    for (int p = t; p < cnt; p += kThreads) {
        const int slot = int(s_e[p] & (kSortTile - 1));
        keys[start + p] = s_key[slot];
        order[start + p] = int32_t(start) + slot;
    }
    if (t == 0) {
        tile_len[blockIdx.x] = cnt;
        if (kForest) atomicAdd(&geo[tile.y].star_hi, cnt);
        else atomicAdd(reinterpret_cast<unsigned long long *>(&info->nstars), static_cast<unsigned long long>(cnt));
    }
}

// Entries of the sorted run x[0, len) below ka, and below kb, by one warp: each round probes 32
// places of each remaining range at once (2 rounds for 1,024 entries, 3 for 32,768).
__device__ __forceinline__ int2 warp_count_below(const uint64_t *__restrict__ x, int32_t len, uint64_t ka, uint64_t kb) {
    const int lane = threadIdx.x & 31;
    int32_t lo[2] = {0, 0}, hi[2] = {len, len};
    const uint64_t k[2] = {ka, kb};
    while (hi[0] > lo[0] || hi[1] > lo[1]) {
        int32_t step[2], at[2];
        bool below[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            step[e] = (hi[e] - lo[e] + 31) >> 5;
            at[e] = lo[e] + (lane + 1) * step[e] - 1;
            below[e] = lo[e] < hi[e] && at[e] < hi[e] && x[at[e]] < k[e];
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int c = __popc(__ballot_sync(kFull, below[e]));
            lo[e] += c * step[e];
            hi[e] = min(hi[e], lo[e] + step[e] - 1);
            if (hi[e] < lo[e]) hi[e] = lo[e];  // step 0: this search is done
        }
    }
    return make_int2(lo[0], lo[1]);
}

// What the last merge writes besides the sorted keys: build.go:34-41 with SourceMass (sim.go:93-98),
// FP64 copies for the FP64 kernels, and the FP32 hi/lo split for the walks.
struct SortedOut {
    const Pos4 *pos4;
    const uint8_t *kind;
    int dm_off, fp64_copies;
    double *sx, *sy, *sz, *sm;
    float4 *st_hi, *st_lo;
    int32_t *sid_sorted;

    // Body i at sorted place `to`.
    __device__ __forceinline__ void write(int64_t to, int32_t i) const {
        const Pos4 p = pos4[i];
        const double m = dm_off && kind && kind[i] == GBH_DARK_MATTER ? 0.0 : p.m;
        if (fp64_copies) {  // read by the FP64 upsweep, walk and potential only
            sx[to] = p.x;
            sy[to] = p.y;
            sz[to] = p.z;
            sm[to] = m;
        }
        const float hx = __double2float_rn(p.x), hy = __double2float_rn(p.y), hz = __double2float_rn(p.z);
        st_hi[to] = make_float4(hx, hy, hz, __double2float_rn(m));
        st_lo[to] = make_float4(__double2float_rn(p.x - double(hx)), __double2float_rn(p.y - double(hy)),
                                __double2float_rn(p.z - double(hz)), 0.f);
    }
};

// The layout entry of a plain state's one system.
__device__ __forceinline__ void single_system(SysGeo *geo, const DevInfo *info) {
    geo[0].star_lo = 0;
    geo[0].star_hi = int32_t(info->nstars);
    geo[0].root = 0;
    geo[0].group_lo = 0;
    geo[0].ngroups = int32_t((info->nstars + 63) / 64);
}

// Merges up to K runs of G tiles each into one (the runs of one group follow each other). A block
// takes 256 consecutive elements of one run, a thread each. An element's place is its place in its
// own run plus, from searches, the elements of the group's earlier runs at or below its key and
// those of the later runs below it (the stable order: earlier runs hold lower state indices). The
// block's first and last element bound the searches in every other run: a warp a run finds the
// window (about 256 elements) and copies it to shared memory, where each thread searches it, four
// runs at a time (eight: 80 registers, 4-14 % slower builds). Windows that do not fit (runs much denser there than this one) are searched where
// they are. Bounds by one thread each and copies by the whole block, run after run, took 23 us for
// 16,384 bodies (16 runs), a chain of some 30 round trips to L2; this takes 18.6 (ncu, cold caches). Four elements a
// thread, galloping on from the first, were 6 % faster on 524,288 stars in random order and 16 %
// slower on a merger, whose tiles differ.
// A run's stars are stored from its first tile's first body on; len_in and len_out hold the runs'
// lengths by their first tile.
constexpr int kWindow = 4096;  // elements: 32 KB, so that 6 blocks share a SM (6,144: 2-5 % slower builds above 131k)

template <bool kForest, bool kLast>
__global__ __launch_bounds__(kThreads) void k_merge(int64_t n, const int4 *__restrict__ tiles, int32_t ntiles, int32_t G,
                                                    int32_t K, const uint64_t *__restrict__ kin,
                                                    const int32_t *__restrict__ vin, uint64_t *__restrict__ kout,
                                                    int32_t *__restrict__ vout, const int32_t *__restrict__ len_in,
                                                    int32_t *__restrict__ len_out, DevInfo *info, SysGeo *geo,
                                                    SortedOut o) {
    pdl_begin();
    constexpr int kBlocksPerTile = kSortTile / kThreads;
    __shared__ uint64_t s_win[kWindow];
    __shared__ const uint64_t *s_x[kMaxWay];  // the run's window
    __shared__ int32_t s_lo[kMaxWay], s_width[kMaxWay], s_off[kMaxWay];
    __shared__ int32_t s_used;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int32_t t = int32_t(blockIdx.x) / kBlocksPerTile, part = int32_t(blockIdx.x) % kBlocksPerTile;
    const int4 tile = tile_at<kForest>(tiles, t, ntiles);
    const int32_t rel = t - tile.z, run = rel / G, group = run / K, mine = run - group * K;
    const int32_t nruns = (tile.w + G - 1) / G;
    // first tile, length and first slot of the group's run r
    auto first_tile = [&](int r) { return tile.z + (group * K + r) * G; };
    auto run_len = [&](int r) { return group * K + r < nruns ? len_in[first_tile(r)] : 0; };
    auto run_start = [&](int r) { return kForest ? int64_t(tiles[first_tile(r)].x) : int64_t(first_tile(r)) * kSortTile; };
    if (!kLast && tid == 0 && part == 0 && rel == group * K * G) {
        int32_t sum = 0;
        for (int r = 0; r < K; ++r) sum += run_len(r);
        len_out[t] = sum;
    }
    if (kLast && !kForest && geo && blockIdx.x == 0 && tid == 0) single_system(geo, info);
    const int64_t slot0 = (kForest ? int64_t(tile.x) : int64_t(t) * kSortTile) + part * kThreads;
    const int64_t p0 = slot0 - run_start(mine);
    const int32_t own = run_len(mine);
    if (p0 >= own) return;  // uniform over the block
    const int32_t cnt = int32_t(own - p0 < kThreads ? own - p0 : kThreads);
    const uint64_t k = tid < cnt ? kin[slot0 + tid] : 0;
    const int32_t i = tid < cnt ? vin[slot0 + tid] : 0;
    const uint64_t k_lo = kin[slot0], k_hi = kin[slot0 + cnt - 1];
    if (tid == 0) s_used = 0;
    __syncthreads();
    for (int r = warp; r < K; r += kThreads / 32) {
        const int32_t len = r == mine ? 0 : run_len(r);
        int2 w = make_int2(0, 0);
        int32_t off = 0;
        const uint64_t *x = kin;
        if (len > 0) {
            x += run_start(r);
            const uint64_t more = r < mine ? 1 : 0;
            w = warp_count_below(x, len, k_lo + more, k_hi + more);
            x += w.x;
            if (lane == 0) off = atomicAdd(&s_used, w.y - w.x);
            off = __shfl_sync(kFull, off, 0);
            if (off + w.y - w.x <= kWindow) {
#pragma unroll 8
                for (int32_t q = lane; q < w.y - w.x; q += 32) s_win[off + q] = x[q];
            }
        }
        if (lane == 0) {
            s_x[r] = x;
            s_lo[r] = w.x;
            s_width[r] = w.y - w.x;
            s_off[r] = off;
        }
    }
    __syncthreads();
    int64_t rank = p0 + tid;
    for (int r = 0; r < K; ++r) rank += s_lo[r];
    auto search = [&](auto window) {  // window(r): in shared or global memory
        constexpr int kRuns = 4;
        for (int r0 = 0; r0 < K; r0 += kRuns) {
            decltype(window(0)) x[kRuns];
            int32_t len[kRuns], pos[kRuns];
#pragma unroll
            for (int q = 0; q < kRuns; ++q) {
                const int r = r0 + q < K ? r0 + q : mine;  // this block's own run: width 0
                x[q] = window(r);
                len[q] = s_width[r];
                pos[q] = 0;
            }
            int32_t widest = 0;
#pragma unroll
            for (int q = 0; q < kRuns; ++q) widest = max(widest, len[q]);
            for (int32_t w = widest ? 1 << (31 - __clz(widest)) : 0; w; w >>= 1)
#pragma unroll
                for (int q = 0; q < kRuns; ++q) {
                    const int32_t at = pos[q] + w;
                    if (at <= len[q] && x[q][at - 1] < k + (r0 + q < mine ? 1 : 0)) pos[q] = at;
                }
#pragma unroll
            for (int q = 0; q < kRuns; ++q) rank += pos[q];
        }
    };
    if (s_used <= kWindow) search([&](int r) { return const_cast<const uint64_t *>(s_win) + s_off[r]; });
    else search([&](int r) { return s_off[r] + s_width[r] <= kWindow ? s_win + s_off[r] : s_x[r]; });
    if (tid >= cnt) return;
    const int64_t to = (kLast ? (kForest ? int64_t(geo[tile.y].star_lo) : 0) : run_start(0)) + rank;
    if (to >= n || i < 0 || i >= n) {
        dev_error(info, 10);
        return;
    }
    kout[to] = k;
    vout[to] = i;
    if (!kLast || !o.pos4) return;
    if (kForest) o.sid_sorted[to] = tile.y;
    o.write(to, i);
}

// Runs merged at once and the number of merges for up to `most` tiles a system: one merge of up to
// 16, else the fewest merges of at most 12 (more runs a merge cost each element more searches:
// 7 to 11 probes a run against one pass over the keys).
struct MergePlan {
    int levels, K;
};
MergePlan merge_plan(int64_t most) {
    if (most <= kMaxWay) return {1, int(most < 1 ? 1 : most)};
    for (int levels = 2;; ++levels)
        for (int K = 2; K <= 12; ++K) {
            int64_t p = 1;
            for (int l = 0; l < levels; ++l) p *= K;
            if (p >= most) return {levels, K};
        }
}

template <bool kForest>
cudaError_t run_sort(const Launch &L, int64_t n, const double *px, const double *py, const double *pz, const double *mass,
                     const uint8_t *kind, const uint8_t *alive, const int4 *tiles, int32_t ntiles, int64_t most,
                     const int64_t *sys_off, int32_t nsys, int32_t gsize, uint64_t *keys, uint64_t *keys_alt,
                     int32_t *order, int32_t *order_alt, int32_t *len, int32_t *len_alt, Pos4 *pos4, DevInfo *info,
                     SysGeo *geo, const SortedOut &out) {
    const MergePlan plan = merge_plan(most);
    // the merges ping-pong between the two buffers and end in keys / order
    uint64_t *kin = plan.levels & 1 ? keys_alt : keys, *kout = plan.levels & 1 ? keys : keys_alt;
    int32_t *vin = plan.levels & 1 ? order_alt : order, *vout = plan.levels & 1 ? order : order_alt;
    GBH_LAUNCH_AFTER(L, k_tile_sort<kForest>, unsigned(ntiles), kThreads, n, tiles, ntiles, sys_off, px, py, pz, mass,
                     kind, alive, geo, kin, vin, len, pos4, info);
    if (kForest) {
        GBH_LAUNCH_AFTER(L, k_sys_ranges, 1, kSysScan, nsys, gsize, geo, info);
    }
    int64_t G = 1;
    for (int l = 0; l < plan.levels; ++l) {
        const bool last = l + 1 == plan.levels;
        auto *kernel = last ? k_merge<kForest, true> : k_merge<kForest, false>;
        GBH_LAUNCH_AFTER(L, kernel, unsigned(ntiles) * (kSortTile / kThreads), kThreads, n, tiles, ntiles, int32_t(G),
                         plan.K, kin, vin, kout, vout, len, len_alt, info, geo, out);
        uint64_t *tk = kin;
        kin = kout;
        kout = tk;
        int32_t *tv = vin;
        vin = vout;
        vout = tv;
        int32_t *tl = len;
        len = len_alt;
        len_alt = tl;
        G *= plan.K;
    }
    return cudaSuccess;
}

// ---------------------------------------------------------------- large states
//
// Radix passes for plain states beyond kMergeTiles tiles: keys of the stars compacted in state order
// (one launch: star counts by look-back), then 8 stable passes of a digit histogram, its scan and a
// scatter, then the sorted copies.

// Whole build, CUDA events, merges against radix passes: Plummer spheres of 131,072 bodies 0.131 /
// 0.209 ms, 262,144 0.181 / 0.237, 393,216 0.237 / 0.287, 524,288 0.275 / 0.308, 786,432 0.400 /
// 0.397, 1,048,576 0.58 / 0.467 (each element searches more and longer runs, the passes stream).
// Forests take merges at any size; against passes over keys and system ids (as they were sorted before):
// one system of 1,048,576 among 63 of 100 0.49 / 0.91 ms, two of 1,048,576 0.89 / 1.35, 5,000 of 100
// 0.28 / 0.90, 20,000 of 50 0.85 / 2.56.
constexpr int64_t kMergeTiles = 768;
constexpr int kRsThreads = 256, kRsItems = 8, kRsTile = kRsThreads * kRsItems, kRsWarps = kRsThreads / 32,
              kRsBins = 256, kRsPasses = 8;
constexpr int kScanItems = 8, kScanTile = kThreads * kScanItems;
inline int64_t rs_tiles(int64_t n) { return (n + kRsTile - 1) / kRsTile; }
inline int64_t hist_scan_tiles(int64_t n) { return (rs_tiles(n) * kRsBins + kScanTile - 1) / kScanTile; }
inline int64_t sort_tiles(int64_t n) { return (n + kSortTile - 1) / kSortTile; }

// order[k] = i for the k-th star in state order; keys[k] its key (build.go:26-31); pos4 as k_tile_sort.
__global__ __launch_bounds__(kThreads) void k_compact_keys(int64_t n, const double *__restrict__ px,
                                                           const double *__restrict__ py,
                                                           const double *__restrict__ pz,
                                                           const double *__restrict__ mass,
                                                           const uint8_t *__restrict__ kind,
                                                           const uint8_t *__restrict__ alive,
                                                           uint64_t *__restrict__ keys, int32_t *__restrict__ order,
                                                           Pos4 *__restrict__ pos4, uint32_t *lb, DevInfo *info) {
    pdl_begin();
    __shared__ uint32_t s_warp[kThreads / 32 + 1];
    __shared__ uint32_t s_tile, s_prefix;
    const int t = threadIdx.x;
    if (t == 0) s_tile = atomicAdd(lb, 1u);
    __syncthreads();
    const uint32_t tile = s_tile;
    const int64_t start = int64_t(tile) * kSortTile;
    uint64_t k[kPer];
    uint32_t cnt = 0, star = 0;
    const double minx = info->minx, miny = info->miny, minz = info->minz, sc = info->scale;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        const int64_t i = start + j * kThreads + t;
        if (i >= n || !is_star(alive ? alive[i] : 1, kind ? kind[i] : 0)) continue;
        const double x = px[i], y = py[i], z = pz[i];
        pos4[i] = Pos4{x, y, z, mass ? mass[i] : 0.0};
        k[j] = spread(cell(x, minx, sc)) << 2 | spread(cell(y, miny, sc)) << 1 | spread(cell(z, minz, sc));
        star |= 1u << j;
        ++cnt;
    }
    // places in state order: item j of all threads before item j + 1, two items a scan
    uint32_t total, place[kPer], run = 0;
#pragma unroll
    for (int j = 0; j < kPer; j += 2) {
        const uint32_t e = block_excl_scan<kThreads>((star >> j & 1u) | (star >> (j + 1) & 1u) << 16, s_warp, total);
        place[j] = run + (e & 0xffffu);
        place[j + 1] = run + (total & 0xffffu) + (e >> 16);
        run += (total & 0xffffu) + (total >> 16);
    }
    if (t < 32) {
        const unsigned long long excl = look_back(reinterpret_cast<unsigned long long *>(lb + 2), tile, run, info);
        if (t == 0) {
            s_prefix = uint32_t(excl);
            if (tile == gridDim.x - 1) info->nstars = int64_t(excl) + run;
        }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kPer; ++j)
        if (star >> j & 1u) {
            keys[s_prefix + place[j]] = k[j];
            order[s_prefix + place[j]] = int32_t(start) + j * kThreads + t;
        }
}

__global__ __launch_bounds__(kRsThreads) void k_rs_hist(const uint64_t *__restrict__ keys, const DevInfo *info, int shift,
                                                        uint32_t ntiles, uint32_t *__restrict__ hist) {
    pdl_begin();
    __shared__ uint32_t h[kRsBins];
    const int64_t n = info->nstars;
    h[threadIdx.x] = 0;
    __syncthreads();
    const int64_t base = int64_t(blockIdx.x) * kRsTile;
    if (base < n) {
#pragma unroll
        for (int it = 0; it < kRsItems; ++it) {
            const int64_t idx = base + it * kRsThreads + threadIdx.x;
            if (idx < n) atomicAdd(&h[uint32_t(keys[idx] >> shift) & (kRsBins - 1)], 1u);
        }
    }
    __syncthreads();
    hist[size_t(threadIdx.x) * ntiles + blockIdx.x] = h[threadIdx.x];
}

// Exclusive scan of the digit table in one launch (look-back over its tiles).
__global__ __launch_bounds__(kThreads) void k_rs_scan(uint32_t *hist, int64_t n, uint32_t *lb, DevInfo *info) {
    pdl_begin();
    __shared__ uint32_t s_warp[kThreads / 32 + 1];
    __shared__ uint32_t s_tile, s_prefix;
    if (threadIdx.x == 0) s_tile = atomicAdd(lb, 1u);
    __syncthreads();
    const uint32_t tile = s_tile;
    const int64_t base = int64_t(tile) * kScanTile + int64_t(threadIdx.x) * kScanItems;
    uint32_t v[kScanItems], sum = 0, total;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        v[k] = base + k < n ? hist[base + k] : 0;
        sum += v[k];
    }
    uint32_t run = block_excl_scan<kThreads>(sum, s_warp, total);
    if (threadIdx.x < 32) {
        const unsigned long long excl = look_back(reinterpret_cast<unsigned long long *>(lb + 2), tile, total, info);
        if (threadIdx.x == 0) s_prefix = uint32_t(excl);
    }
    __syncthreads();
    run += s_prefix;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        if (base + k < n) hist[base + k] = run;
        run += v[k];
    }
}

// Stable scatter of one tile. Rank of a key = keys of the same digit earlier in the tile, in
// the order (item round, warp, lane) used to load them; offs holds the digit-major exclusive
// scan of the tile histograms, so equal digits keep their input order across tiles too.
__global__ __launch_bounds__(kRsThreads) void k_rs_scatter(const uint64_t *__restrict__ kin,
                                                           const int32_t *__restrict__ vin,
                                                           uint64_t *__restrict__ kout, int32_t *__restrict__ vout,
                                                           DevInfo *info, int shift, uint32_t ntiles,
                                                           const uint32_t *__restrict__ offs) {
    pdl_begin();
    __shared__ uint32_t s_run[kRsBins];
    __shared__ uint32_t s_goff[kRsBins];
    __shared__ uint32_t s_w[2][kRsWarps][kRsBins];
    const int64_t n = info->nstars;
    const int64_t base = int64_t(blockIdx.x) * kRsTile;
    if (base >= n) return;  // uniform over the block
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    s_run[tid] = 0;
    s_goff[tid] = offs[size_t(tid) * ntiles + blockIdx.x];
#pragma unroll
    for (int w = 0; w < kRsWarps; ++w) {
        s_w[0][w][tid] = 0;
        s_w[1][w][tid] = 0;
    }
    uint64_t k[kRsItems];
    int32_t v[kRsItems];
#pragma unroll
    for (int it = 0; it < kRsItems; ++it) {
        const int64_t idx = base + it * kRsThreads + tid;
        if (idx < n) {
            k[it] = kin[idx];
            v[it] = vin[idx];
        }
    }
    __syncthreads();
    const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
    for (int it = 0; it < kRsItems; ++it) {
        const int buf = it & 1;
        const bool valid = base + it * kRsThreads + tid < n;
        const uint32_t d = valid ? uint32_t(k[it] >> shift) & (kRsBins - 1) : 0u;
        const uint32_t peers = __match_any_sync(kFull, valid ? d : uint32_t(kRsBins + lane));
        const uint32_t rank = __popc(peers & lt);
        if (valid && rank == 0) s_w[buf][warp][d] = __popc(peers);
        __syncthreads();
        uint32_t run = s_run[tid];
#pragma unroll
        for (int w = 0; w < kRsWarps; ++w) {
            const uint32_t c = s_w[buf][w][tid];
            s_w[buf][w][tid] = run;
            run += c;
            s_w[buf ^ 1][w][tid] = 0;  // readers of the other buffer finished before this round's first barrier
        }
        s_run[tid] = run;
        __syncthreads();
        if (valid) {
            const uint32_t pos = s_goff[d] + s_w[buf][warp][d] + rank;
            if (pos < n) {
                kout[pos] = k[it];
                vout[pos] = v[it];
            } else {
                dev_error(info, 10);
            }
        }
    }
}

// The sorted copies through the order.
__global__ __launch_bounds__(kThreads) void k_gather(const int32_t *__restrict__ order, DevInfo *info, SysGeo *geo,
                                                     SortedOut o) {
    pdl_begin();
    const int64_t k = int64_t(blockIdx.x) * kThreads + threadIdx.x;
    if (k == 0) single_system(geo, info);
    if (k < info->nstars) o.write(k, order[k]);
}

cudaError_t sort_large(const Launch &L, TreeBufs &b, int64_t n, const double *px, const double *py, const double *pz,
                       const double *mass, const uint8_t *kind, const uint8_t *alive, const SortedOut &out) {
    uint32_t *lb = b.lb_state + b.lb_sort;
    GBH_LAUNCH_AFTER(L, k_compact_keys, unsigned(sort_tiles(n)), kThreads, n, px, py, pz, mass, kind, alive, b.keys,
                     b.order, b.pos4, lb, b.info);
    lb += lb_words_of(sort_tiles(n));
    const uint32_t ntiles = uint32_t(rs_tiles(n));
    uint64_t *kin = b.keys, *kout = b.keys_alt;
    int32_t *vin = b.order, *vout = b.order_alt;
    for (int p = 0; p < kRsPasses; ++p) {
        GBH_LAUNCH_AFTER(L, k_rs_hist, ntiles, kRsThreads, kin, b.info, 8 * p, ntiles, b.hist);
        GBH_LAUNCH_AFTER(L, k_rs_scan, unsigned(hist_scan_tiles(n)), kThreads, b.hist, int64_t(ntiles) * kRsBins, lb,
                         b.info);
        GBH_LAUNCH_AFTER(L, k_rs_scatter, ntiles, kRsThreads, kin, vin, kout, vout, b.info, 8 * p, ntiles, b.hist);
        lb += lb_words_of(hist_scan_tiles(n));
        uint64_t *tk = kin;
        kin = kout;
        kout = tk;
        int32_t *tv = vin;
        vin = vout;
        vout = tv;
    }
    GBH_LAUNCH_AFTER(L, k_gather, blocks_for(n, kThreads), kThreads, b.order, b.info, b.geo, out);
    return cudaSuccess;
}

}  // namespace

size_t sort_part_bytes() { return sizeof(long long) * kBboxBlocks * kPartWords; }
int64_t sort_lb_words(int64_t n) {
    return sort_tiles(n) <= kMergeTiles ? 0 : lb_words_of(sort_tiles(n)) + kRsPasses * lb_words_of(hist_scan_tiles(n));
}
int64_t sort_hist_words(int64_t n) { return sort_tiles(n) <= kMergeTiles ? 1 : rs_tiles(n) * kRsBins; }

cudaError_t sort_stars(const Launch &L, TreeBufs &b, int64_t n, const double *px, const double *py, const double *pz,
                       const double *mass, const uint8_t *kind, const uint8_t *alive, double *ax, double *ay,
                       double *az, double theta, int dm_off, bool exact, const ForestTiles *forest) {
    const SortedOut out = {b.pos4, kind, dm_off, exact ? 1 : 0, b.sx, b.sy, b.sz, b.sm, b.st_hi, b.st_lo, b.sid_sorted};
    if (!forest) {
        unsigned nb = blocks_for(n, kThreads);
        if (nb > unsigned(kBboxBlocks)) nb = kBboxBlocks;
        GBH_LAUNCH_AFTER(L, k_bbox, nb, kThreads, n, px, py, pz, mass, kind, alive, theta, b.bbox_part, ax, ay, az,
                         b.lb_state, b.lb_words, b.info, b.geo);
        const int32_t ntiles = int32_t(sort_tiles(n));
        if (ntiles > kMergeTiles) return sort_large(L, b, n, px, py, pz, mass, kind, alive, out);
        return run_sort<false>(L, n, px, py, pz, mass, kind, alive, nullptr, ntiles, ntiles, nullptr, 1, 64, b.keys,
                               b.keys_alt, b.order, b.order_alt, b.tile_len, b.tile_len + b.cap_tiles, b.pos4, b.info,
                               b.geo, out);
    }
    const int32_t nsys = b.nsys;
    const unsigned zb = blocks_for(b.lb_words > nsys ? b.lb_words : nsys, kThreads);
    GBH_LAUNCH_AFTER(L, k_sys_init, std::max(zb, blocks_for(nsys, kThreads)), kThreads, nsys, b.geo, b.info, theta,
                     b.lb_state, b.lb_words);
    if (forest->ntiles < 1) return cudaErrorInvalidValue;
    GBH_LAUNCH_AFTER(L, k_bbox_sys, unsigned(forest->ntiles), kThreads, forest->tiles, forest->sys_off, px, py, pz,
                     mass, kind, alive, b.geo, ax, ay, az);
    GBH_LAUNCH_AFTER(L, k_sys_cube, blocks_for(nsys, 4), 128, nsys, theta, b.geo);
    return run_sort<true>(L, n, px, py, pz, mass, kind, alive, forest->tiles, forest->ntiles, forest->most,
                          forest->sys_off, nsys, b.group == 32 ? 32 : 64, b.keys, b.keys_alt, b.order, b.order_alt,
                          b.tile_len, b.tile_len + b.cap_tiles, b.pos4, b.info, b.geo, out);
}

// ---------------------------------------------------------------- Morton order into caller-owned scratch

namespace {
inline size_t align256(size_t x) { return (x + 255) & ~size_t(255); }
}  // namespace

size_t morton_sort_scratch_bytes(int64_t nmax) {
    const int64_t tiles = (nmax + kSortTile - 1) / kSortTile;
    return align256(sizeof(DevInfo)) + align256(sort_part_bytes()) + align256(sizeof(uint64_t) * size_t(nmax)) +
           align256(sizeof(int32_t) * size_t(nmax)) + 2 * align256(sizeof(int32_t) * size_t(tiles));
}

// The collect, key and sort stages of the tree build (the same kernels), with every temporary
// carved out of one caller-provided device block instead of TreeBufs.
cudaError_t morton_sort(const Launch &L, int64_t n, const double *px, const double *py, const double *pz,
                        const uint8_t *kind, const uint8_t *alive, uint64_t *keys, int32_t *order, void *scratch,
                        size_t scratch_bytes, DevInfo **info_out) {
    if (morton_sort_scratch_bytes(n) > scratch_bytes) return cudaErrorInvalidValue;
    char *p = static_cast<char *>(scratch);
    auto take = [&](size_t bytes) {
        char *q = p;
        p += align256(bytes);
        return q;
    };
    const int32_t ntiles = int32_t((n + kSortTile - 1) / kSortTile);
    DevInfo *info = reinterpret_cast<DevInfo *>(take(sizeof(DevInfo)));
    long long *part = reinterpret_cast<long long *>(take(sort_part_bytes()));
    uint64_t *keys_alt = reinterpret_cast<uint64_t *>(take(sizeof(uint64_t) * size_t(n)));
    int32_t *order_alt = reinterpret_cast<int32_t *>(take(sizeof(int32_t) * size_t(n)));
    int32_t *len = reinterpret_cast<int32_t *>(take(sizeof(int32_t) * size_t(ntiles)));
    int32_t *len_alt = reinterpret_cast<int32_t *>(take(sizeof(int32_t) * size_t(ntiles)));
    *info_out = info;
    cudaError_t e = cudaMemsetAsync(info, 0, sizeof(DevInfo), L.stream);
    if (e != cudaSuccess || n == 0) return e;
    unsigned nb = blocks_for(n, kThreads);
    if (nb > unsigned(kBboxBlocks)) nb = kBboxBlocks;
    GBH_LAUNCH_AFTER(L, k_bbox, nb, kThreads, n, px, py, pz, nullptr, kind, alive, 0.9, part, nullptr, nullptr, nullptr,
                     nullptr, 0, info, nullptr);
    return run_sort<false>(L, n, px, py, pz, nullptr, kind, alive, nullptr, ntiles, ntiles, nullptr, 1, 64, keys, keys_alt,
                           order, order_alt, len, len_alt, nullptr, info, nullptr, SortedOut{});
}

}  // namespace gbh
