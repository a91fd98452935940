// tree.cu — octree construction and the FP64 kernels of the Barnes-Hut step.
//
// Compiled with -fmad=false: every FP64 a*b+c is a rounded multiply and a rounded add, as in
// the reference's arithmetic, so keys, node moments, the FP64 walk, the direct sum and the
// kick/drift are bit identical to it.
//
// Pipeline of tree_build (one stream, no host round trip):
//   sort_stars (sort.cu)                                            (collect, keys, sort, build.go:11-41, 62-113)
//   k_chains -> k_topology -> k_child_scan -> k_emit_nodes          (node set and links of buildNode, build.go:134-172)
//   k_upsweep                                                       (finish, build.go:176-217)
//
// Node set without recursion. A cell at level L is the set of sorted stars whose keys share
// their top 3L bits. The reference creates a node for the root and for every non-empty octant
// of a node that splits (count > leaf and level < 21). Counts shrink down the tree, so a
// non-root cell is a node exactly when its parent cell holds more than leaf stars. Every node
// starts at some sorted position i; the nodes starting at i form a chain of consecutive levels
// (a node and its first child share their first star). Sorting nodes by (first star, level) is
// the walk's pre-order, so the skip pointer of a node is the shallowest node that starts where
// it ends. The reference's serial build allocates each node's children as one block when the
// node is visited in that pre-order, so a prefix sum of child counts over pre-order gives every
// node its index in the reference's own serial layout.
#include <cuda_runtime.h>

#include <climits>

#include "gbh_internal.cuh"
#include "lookback.cuh"

namespace gbh {

namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

constexpr int kThreads = 256;

inline unsigned blocks_for(int64_t n, int threads) {
    int64_t b = (n + threads - 1) / threads;
    return unsigned(b < 1 ? 1 : b);
}

// ---------------------------------------------------------------- node set (chains)

// Sorted star range [lo, hi) of the system that sorted position i belongs to (the whole array
// for a plain state).
struct SysRange {
    int64_t lo, hi;
};
__device__ __forceinline__ SysRange sys_range(const int32_t *__restrict__ sid_sorted, const SysGeo *__restrict__ geo,
                                              int64_t i, int64_t n) {
    if (!sid_sorted) return SysRange{0, n};
    const SysGeo &g = geo[sid_sorted[i]];
    return SysRange{g.star_lo, g.star_hi};
}

// Shallowest level at which sorted position i starts a new cell (0 at the first star of its
// system, kNoCell if its key equals the previous one).
__device__ __forceinline__ int start_level(const uint64_t *__restrict__ keys, int64_t i, int64_t lo = 0) {
    if (i == lo) return 0;
    uint64_t x = keys[i] ^ keys[i - 1];
    if (x == 0) return kNoCell;
    int h = 63 - __clzll(static_cast<long long>(x));
    return kMaxLevel - h / 3;
}

__device__ __forceinline__ uint64_t prefix(uint64_t k, int L) { return L == 0 ? 0 : k >> (3 * (kMaxLevel - L)); }

// First position after i whose level-L cell differs from i's (galloping, then binary search).
__device__ int64_t cell_end(const uint64_t *__restrict__ keys, int64_t n, int64_t i, int L) {
    if (L == 0) return n;
    uint64_t P = prefix(keys[i], L);
    int64_t lo = i + 1, hi = n, step = 1;
    for (;;) {
        int64_t probe = i + step;
        if (probe >= n) break;
        if (prefix(keys[probe], L) != P) {
            hi = probe;
            break;
        }
        lo = probe + 1;
        step <<= 1;
    }
    while (lo < hi) {
        int64_t mid = (lo + hi) >> 1;
        if (prefix(keys[mid], L) == P) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// First position of i's level-L cell (not before lo_bound, the first star of its system).
__device__ int64_t cell_start(const uint64_t *__restrict__ keys, int64_t lo_bound, int64_t i, int L) {
    if (L == 0) return lo_bound;
    uint64_t P = prefix(keys[i], L);
    int64_t lo = lo_bound, hi = i, step = 1;
    for (;;) {
        int64_t probe = i - step;
        if (probe < lo_bound) break;
        if (prefix(keys[probe], L) != P) {
            lo = probe + 1;
            break;
        }
        hi = probe;
        step <<= 1;
    }
    while (lo < hi) {
        int64_t mid = (lo + hi) >> 1;
        if (prefix(keys[mid], L) == P) hi = mid;
        else lo = mid + 1;
    }
    return lo;
}

// Nodes that start at sorted position i of the system [lo, hi) (0 when none), from level L0 on.
__device__ __forceinline__ uint32_t chain_at(const uint64_t *__restrict__ keys, int64_t i, int64_t lo, int64_t hi,
                                             int leaf, int &L0) {
    L0 = start_level(keys, i, lo);
    if (L0 > kMaxLevel) return 0;
    // A level-L cell starting at i holds more than leaf stars exactly when the star leaf positions on
    // is still inside it (cells are contiguous runs of the sorted keys).
    const uint64_t ki = keys[i];
    const bool ahead = i + leaf < hi;
    const uint64_t ka = ahead ? keys[i + leaf] : 0;
    if (i > lo) {  // the parent cell (level L0-1) contains i-1 and i; the node exists iff it holds > leaf stars
        const int Lp = L0 - 1;
        const uint64_t P = prefix(ki, Lp);
        if (!(ahead && prefix(ka, Lp) == P)) {
            // at most leaf of its stars from i on: a of them, so leaf + 1 - a before i are needed
            int64_t x = i + 1, y = ahead ? i + leaf : hi;
            while (x < y) {
                const int64_t mid = (x + y) >> 1;
                if (prefix(keys[mid], Lp) == P) x = mid + 1;
                else y = mid;
            }
            const int64_t j = i - (leaf + 1 - (x - i));
            if (j < lo || prefix(keys[j], Lp) != P) return 0;
        }
    }
    if (!ahead) return 1;
    // the deepest level at which star i + leaf shares the cell; every such level from L0 to 20 splits
    const uint64_t d = ki ^ ka;
    const int S = d ? kMaxLevel - 1 - (63 - __clzll(static_cast<long long>(d))) / 3 : kMaxLevel - 1;
    const int last = S < kMaxLevel - 1 ? S : kMaxLevel - 1;
    return last >= L0 ? uint32_t(last - L0 + 2) : 1u;
}

// The nodes in pre-order, chain by chain: base[i] is the pre-order index of the first node at sorted
// position i (an exclusive scan of the chain lengths, by look-back), and each node gets its star,
// level | octant << 8 and an empty child mask. A block takes the next tile of 1,024 positions.
constexpr int kChainThreads = 512, kChainTile = 2 * kChainThreads;
inline int64_t chain_tiles(int64_t n) { return (n + kChainTile - 1) / kChainTile; }
__global__ __launch_bounds__(kChainThreads) void k_chains(const uint64_t *__restrict__ keys, DevInfo *info,
                                                          const int32_t *__restrict__ sid_sorted,
                                                          const SysGeo *__restrict__ geo, int leaf,
                                                          uint32_t *__restrict__ base, int32_t *__restrict__ pre_star,
                                                          uint32_t *__restrict__ pre_info,
                                                          uint32_t *__restrict__ pre_mask, uint32_t *lb,
                                                          int64_t cap_nodes) {
    pdl_begin();
    __shared__ uint32_t s_warp[kChainThreads / 32 + 1];
    __shared__ uint32_t s_tile, s_prefix;
    if (threadIdx.x == 0) s_tile = atomicAdd(lb, 1u);
    __syncthreads();
    const uint32_t tile = s_tile;
    const int64_t n = info->nstars;
    const int64_t i0 = int64_t(tile) * kChainTile + threadIdx.x;
    if (int64_t(tile) * kChainTile >= n) return;  // uniform
    uint32_t c[2] = {0, 0};
    int L0[2] = {0, 0};
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int64_t i = i0 + q * kChainThreads;
        if (i >= n) continue;
        const SysRange R = sys_range(sid_sorted, geo, i, n);
        c[q] = chain_at(keys, i, R.lo, R.hi, leaf, L0[q]);
    }
    uint32_t total;  // both halves in one scan: at most 512 x 22 nodes each
    const uint32_t excl = block_excl_scan<kChainThreads>(c[0] | c[1] << 16, s_warp, total);
    const uint32_t sum = (total & 0xffffu) + (total >> 16);
    if (threadIdx.x < 32) {
        const unsigned long long e = look_back(reinterpret_cast<unsigned long long *>(lb + 2), tile, sum, info);
        if (threadIdx.x == 0) s_prefix = uint32_t(e);
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int64_t i = i0 + q * kChainThreads;
        if (i >= n) continue;
        const uint32_t b = s_prefix + (q ? (total & 0xffffu) + (excl >> 16) : excl & 0xffffu);
        base[i] = b;
        if (i == n - 1) info->nnodes = int64_t(b) + c[q];
        const uint64_t key = keys[i];
        for (uint32_t t = 0; t < c[q]; ++t) {
            const int64_t p = int64_t(b) + t;
            if (p >= cap_nodes) {
                dev_error(info, 11);
                break;
            }
            const int L = L0[q] + int(t);
            pre_star[p] = int32_t(i);
            pre_info[p] = uint32_t(L) | (L == 0 ? 0u : uint32_t(key >> (3 * (kMaxLevel - L))) & 7u) << 8;
            pre_mask[p] = 0;
        }
    }
}

constexpr int kNextBlocks = 1024;  // most blocks of the kernels that find a block step's next event
// Tiles of the active-star lists (block steps).
constexpr int kTargetThreads = 256, kTargetItems = 4, kTargetTile = kTargetThreads * kTargetItems;
inline int64_t target_tiles(int64_t n) { return (n + kTargetTile - 1) / kTargetTile; }

// Grid of the per-node kernels below: they loop over the nodes, whose count only the device knows.
inline unsigned node_blocks(int64_t cap_nodes) {
    const unsigned nb = blocks_for(cap_nodes, kThreads);
    return nb < 2048u ? nb : 2048u;
}

// Parent (pre-order index) and end of every node's cell, one thread per node, so that the searches
// of all nodes run side by side; every node marks its octant in its parent's child mask. The
// parent is the node before in the same chain, or, for a chain's first node, the node at the
// start of the cell one level up.
__global__ __launch_bounds__(kThreads) void k_topology(const uint64_t *__restrict__ keys, DevInfo *info,
                                                       const uint32_t *__restrict__ base,
                                                       const int32_t *__restrict__ pre_star,
                                                       const uint32_t *__restrict__ pre_info, uint32_t *pre_mask,
                                                       int32_t *__restrict__ pre_parent, int32_t *__restrict__ pre_hi,
                                                       const int32_t *__restrict__ sid_sorted,
                                                       const SysGeo *__restrict__ geo, int64_t cap_nodes) {
    pdl_begin();
    const int64_t n = info->nstars, nn = info->nnodes < cap_nodes ? info->nnodes : cap_nodes;
    for (int64_t p = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; p < nn; p += int64_t(gridDim.x) * blockDim.x) {
        const int64_t i = pre_star[p];
        if (i < 0 || i >= n) {
            dev_error(info, 11);
            continue;
        }
        const uint32_t inf = pre_info[p];
        const int L = int(inf & 0xffu);
        const SysRange R = sys_range(sid_sorted, geo, i, n);
        int32_t par = -1;
        if (L > 0) {
            if (base[i] < uint32_t(p)) {
                par = int32_t(p) - 1;
            } else {
                const int64_t ps = cell_start(keys, R.lo, i, L - 1);
                par = int32_t(base[ps]) + (L - 1 - start_level(keys, ps, R.lo));
            }
            if (par < 0 || par >= nn) {
                dev_error(info, 11);
                par = -1;
            }
        }
        pre_parent[p] = par;
        pre_hi[p] = int32_t(cell_end(keys, R.hi, i, L));
        if (par >= 0) atomicOr(&pre_mask[par], 1u << (inf >> 8 & 0xffu));
    }
}

// Exclusive scan of the nodes' child counts (the bits of their masks), in one launch by look-back.
inline int64_t child_tiles(int64_t cap_nodes) { return (cap_nodes + kScanTile - 1) / kScanTile; }
__global__ __launch_bounds__(kScanThreads) void k_child_scan(const uint32_t *__restrict__ pre_mask,
                                                             uint32_t *__restrict__ child_base, int64_t cap_nodes,
                                                             uint32_t *lb, DevInfo *info) {
    pdl_begin();
    __shared__ uint32_t s_warp[kScanThreads / 32 + 1];
    __shared__ uint32_t s_tile, s_prefix;
    if (threadIdx.x == 0) s_tile = atomicAdd(lb, 1u);
    __syncthreads();
    const uint32_t tile = s_tile;
    const int64_t nn = info->nnodes < cap_nodes ? info->nnodes : cap_nodes;
    if (int64_t(tile) * kScanTile >= nn) return;  // uniform
    const int64_t p0 = int64_t(tile) * kScanTile + int64_t(threadIdx.x) * kScanItems;
    uint32_t v[kScanItems], sum = 0, total;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        v[k] = p0 + k < nn ? __popc(pre_mask[p0 + k]) : 0;
        sum += v[k];
    }
    uint32_t run = block_excl_scan<kScanThreads>(sum, s_warp, total);
    if (threadIdx.x < 32) {
        const unsigned long long e = look_back(reinterpret_cast<unsigned long long *>(lb + 2), tile, total, info);
        if (threadIdx.x == 0) s_prefix = uint32_t(e);
    }
    __syncthreads();
    run += s_prefix;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        if (p0 + k < nn) child_base[p0 + k] = run;
        run += v[k];
    }
}

// Links and ranges of every node in the reference layout (bh.go:59-67), one thread per node, and the
// list of leaves. A node's reference index: 1 + (children allocated before its parent's block) + its
// rank among the parent's non-empty octants, inside its system's block of the table (which starts
// at the pre-order index of the system's first chain). It is formed where it is needed (the node's
// own, its parent's, and that of the next node of the walk).
__global__ __launch_bounds__(kThreads) void k_emit_nodes(DevInfo *info, const uint32_t *__restrict__ base,
                                                         const int32_t *__restrict__ pre_star,
                                                         const int32_t *__restrict__ pre_parent,
                                                         const uint32_t *__restrict__ pre_info,
                                                         const uint32_t *__restrict__ pre_mask,
                                                         const int32_t *__restrict__ pre_hi,
                                                         const uint32_t *__restrict__ child_base,
                                                         gbh_node *__restrict__ nodes, int32_t *__restrict__ n_parent,
                                                         uint32_t *__restrict__ n_info, int32_t *__restrict__ n_arrive,
                                                         int32_t *__restrict__ leaves,
                                                         const int32_t *__restrict__ sid_sorted,
                                                         const SysGeo *__restrict__ geo, int64_t cap_nodes) {
    pdl_begin();
    const int64_t n = info->nstars, nn = info->nnodes < cap_nodes ? info->nnodes : cap_nodes;
    const int lane = threadIdx.x & 31;
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    // whole warps iterate together (the ballot below needs every lane)
    for (int64_t p0 = int64_t(blockIdx.x) * blockDim.x + (threadIdx.x & ~31); p0 < nn; p0 += stride) {
        const int64_t p = p0 + lane;
        int32_t r = -1;
        bool is_leaf = false;
        if (p < nn) {
            const int64_t i = pre_star[p];
            const int32_t pp = pre_parent[p];
            const uint32_t inf = pre_info[p], mask = pre_mask[p];
            const int64_t hi = pre_hi[p];
            const SysRange R = sys_range(sid_sorted, geo, i < 0 || i >= n ? 0 : i, n);
            const uint32_t root = base[R.lo];
            const uint32_t root_children = child_base[root];
            // the reference index of the node with octant word `w` under parent q (-1: the root)
            auto ref = [&](int32_t q, uint32_t w) {
                if (q < 0) return int32_t(root);
                return int32_t(root + 1 + (child_base[q] - root_children) +
                               __popc(pre_mask[q] & ((1u << (w >> 8 & 0xffu)) - 1u)));
            };
            r = ref(pp, inf);
            int32_t nx = -1;  // a system's walk ends at its own last node
            bool ok = i >= 0 && i < n && r >= 0 && r < nn && hi > i && hi <= R.hi;
            if (ok && hi < R.hi) {
                const uint32_t q = base[hi];
                ok = q < uint32_t(nn) && pre_star[q] == int32_t(hi);
                if (ok) nx = ref(pre_parent[q], pre_info[q]);
                ok = ok && nx >= 0 && nx < nn;
            }
            if (!ok) {
                dev_error(info, 12);
                r = -1;
            } else {
                is_leaf = mask == 0;
                gbh_node &nd = nodes[r];
                nd.first = mask ? int32_t(root + 1 + (child_base[p] - root_children)) : -1;
                nd.next = nx;
                nd.lo = int32_t(i);
                nd.hi = int32_t(hi);
                n_parent[r] = pp < 0 ? -1 : ref(pre_parent[pp], pre_info[pp]);
                n_info[r] = (inf & 0xffu) | uint32_t(__popc(mask)) << 8;
                n_arrive[r] = 0;
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, is_leaf);
        if (m) {
            uint32_t off = 0;
            if (lane == __ffs(m) - 1) off = atomicAdd(&info->nleaves, uint32_t(__popc(m)));
            off = __shfl_sync(0xffffffffu, off, __ffs(m) - 1);
            if (is_leaf) leaves[off + __popc(m & ((1u << lane) - 1u))] = r;
        }
    }
}

// ---------------------------------------------------------------- moments (finish, build.go:176-217)

struct Moments {
    double x, y, z, m, qxx, qyy, qzz, qxy, qxz, qyz;
};

// quadrupole.add, build.go:329-337.
__device__ __forceinline__ void quad_add(Moments &q, double m, double dx, double dy, double dz) {
    double r2 = dx * dx + dy * dy + dz * dz;
    q.qxx += m * (3 * dx * dx - r2);
    q.qyy += m * (3 * dy * dy - r2);
    q.qzz += m * (3 * dz * dz - r2);
    q.qxy += m * 3 * dx * dy;
    q.qxz += m * 3 * dx * dz;
    q.qyz += m * 3 * dy * dz;
}

// Geometric centre and half side of the level-L cell containing key, through the same
// rounded additions as the recursion c_child = c + offset(oct, bit) * half/2 (build.go:142-152).
__device__ __forceinline__ void cell_center(const SysGeo &inf, uint64_t key, int L, double &cx, double &cy,
                                            double &cz, double &half) {
    double h = inf.side / 2;
    cx = inf.minx + h;
    cy = inf.miny + h;
    cz = inf.minz + h;
    for (int l = 1; l <= L; ++l) {
        h = h / 2;
        uint32_t oct = uint32_t(key >> (3 * (kMaxLevel - l))) & 7u;
        cx = cx + ((oct >> 2 & 1u) ? h : -h);
        cy = cy + ((oct >> 1 & 1u) ? h : -h);
        cz = cz + ((oct & 1u) ? h : -h);
    }
    half = h;
}

__device__ __forceinline__ void write_node(gbh_node *nodes, PNode *pn, MNode *mn, int2 *mr, int32_t r, const Moments &q,
                                           double crit2) {
    gbh_node &nd = nodes[r];
    nd.x = q.x;
    nd.y = q.y;
    nd.z = q.z;
    nd.m = q.m;
    nd.qxx = q.qxx;
    nd.qyy = q.qyy;
    nd.qzz = q.qzz;
    nd.qxy = q.qxy;
    nd.qxz = q.qxz;
    nd.qyz = q.qyz;
    nd.crit2 = crit2;
    int32_t first = nd.first, next = nd.next, lo = nd.lo, hi = nd.hi;
    float fx = __double2float_rn(q.x), fy = __double2float_rn(q.y), fz = __double2float_rn(q.z);
    float fm = __double2float_rn(q.m), fc = __double2float_rn(crit2);
    PNode p;
    p.com = make_float4(fx, fy, fz, fm);
    p.q1 = make_float4(__double2float_rn(q.qxx), __double2float_rn(q.qyy), __double2float_rn(q.qzz),
                       __double2float_rn(q.qxy));
    p.q2 = make_float4(__double2float_rn(q.qxz), __double2float_rn(q.qyz), fc, 0.f);
    p.links = make_int4(first, next, lo, hi);
    pn[r] = p;
    MNode m;
    m.a = make_float4(fx, fy, fz, fc);
    m.b = make_float4(__double2float_rn(q.x - double(fx)), __double2float_rn(q.y - double(fy)),
                      __double2float_rn(q.z - double(fz)), fm);
    m.c = p.q1;
    m.d = make_float4(p.q2.x, p.q2.y, __int_as_float(first), __int_as_float(next));
    mn[r] = m;
    mr[r] = make_int2(lo, hi);
}

__device__ __forceinline__ double crit2_of(double theta, const Moments &q, double cx, double cy, double cz,
                                           double half) {
    double delta = sqrt((q.x - cx) * (q.x - cx) + (q.y - cy) * (q.y - cy) + (q.z - cz) * (q.z - cz));
    double crit = 2 * half / theta + delta;
    return crit * crit;
}

// Bottom-up moments: one thread per leaf; the last child to finish computes its parent.
__global__ __launch_bounds__(kThreads) void k_upsweep(const uint64_t *__restrict__ keys, const DevInfo *info,
                                                      const int32_t *__restrict__ leaves,
                                                      const double *__restrict__ sx, const double *__restrict__ sy,
                                                      const double *__restrict__ sz, const double *__restrict__ sm,
                                                      gbh_node *nodes, const int32_t *__restrict__ n_parent,
                                                      const uint32_t *__restrict__ n_info, int32_t *n_arrive, PNode *pn,
                                                      MNode *mn, int2 *mr, const int32_t *__restrict__ sid_sorted,
                                                      const SysGeo *__restrict__ geo, DevInfo *err_info) {
    const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= int64_t(info->nleaves)) return;
    const DevInfo inf = *info;
    const int32_t r = leaves[t];
    {
        int32_t lo = nodes[r].lo, hi = nodes[r].hi;
        int L = int(n_info[r] & 0xffu);
        Moments q = {};
        for (int32_t j = lo; j < hi; ++j) {
            double mj = sm[j];
            q.x = q.x + mj * sx[j];
            q.y = q.y + mj * sy[j];
            q.z = q.z + mj * sz[j];
            q.m = q.m + mj;
        }
        double cx, cy, cz, half;
        const SysGeo &g = geo[sid_sorted ? sid_sorted[lo] : 0];
        cell_center(g, keys[lo], L, cx, cy, cz, half);
        if (q.m > 0) {
            q.x = q.x / q.m;
            q.y = q.y / q.m;
            q.z = q.z / q.m;
        } else {
            q.x = cx;
            q.y = cy;
            q.z = cz;
        }
        for (int32_t j = lo; j < hi; ++j) quad_add(q, sm[j], sx[j] - q.x, sy[j] - q.y, sz[j] - q.z);
        write_node(nodes, pn, mn, mr, r, q, crit2_of(inf.theta, q, cx, cy, cz, half));
    }
    int32_t cur = r;
    for (int guard = 0; guard <= kMaxLevel + 1; ++guard) {
        int32_t par = n_parent[cur];
        if (par < 0) break;
        uint32_t nch = (n_info[par] >> 8) & 0xffu;
        __threadfence();
        int old = atomicAdd(&n_arrive[par], 1);
        if (old != int(nch) - 1) break;
        __threadfence();
        int32_t first = nodes[par].first;
        if (first < 0 || int64_t(first) + nch > inf.nnodes) {
            dev_error(err_info, 13);
            break;
        }
        Moments q = {};
        for (int32_t ch = first; ch < first + int32_t(nch); ++ch) {
            double cm = __ldcg(&nodes[ch].m);
            q.x = q.x + cm * __ldcg(&nodes[ch].x);
            q.y = q.y + cm * __ldcg(&nodes[ch].y);
            q.z = q.z + cm * __ldcg(&nodes[ch].z);
            q.m = q.m + cm;
        }
        int L = int(n_info[par] & 0xffu);
        double cx, cy, cz, half;
        const int32_t plo = nodes[par].lo;
        cell_center(geo[sid_sorted ? sid_sorted[plo] : 0], keys[plo], L, cx, cy, cz, half);
        if (q.m > 0) {
            q.x = q.x / q.m;
            q.y = q.y / q.m;
            q.z = q.z / q.m;
        } else {
            q.x = cx;
            q.y = cy;
            q.z = cz;
        }
        for (int32_t ch = first; ch < first + int32_t(nch); ++ch) {
            q.qxx = q.qxx + __ldcg(&nodes[ch].qxx);
            q.qyy = q.qyy + __ldcg(&nodes[ch].qyy);
            q.qzz = q.qzz + __ldcg(&nodes[ch].qzz);
            q.qxy = q.qxy + __ldcg(&nodes[ch].qxy);
            q.qxz = q.qxz + __ldcg(&nodes[ch].qxz);
            q.qyz = q.qyz + __ldcg(&nodes[ch].qyz);
            quad_add(q, __ldcg(&nodes[ch].m), __ldcg(&nodes[ch].x) - q.x, __ldcg(&nodes[ch].y) - q.y,
                     __ldcg(&nodes[ch].z) - q.z);
        }
        write_node(nodes, pn, mn, mr, par, q, crit2_of(inf.theta, q, cx, cy, cz, half));
        cur = par;
    }
}

// ---------------------------------------------------------------- FP64 walk (bh.go:106-155)

// The reference's per-star skip-pointer walk for the 32 stars of a warp in lockstep: the warp
// visits the union of its stars' nodes in pre-order, and each lane takes part in exactly the
// visits that its own walk makes (`resume` is the node its walk comes to next: a lane that
// accepts a node waits until the warp has passed the subtree, whose last skip pointer is the
// node's own). Every star so sees its nodes and leaf stars in the reference's order, and its sums
// keep their bits.
//
// The walk is bound by the FP64 pipe, which a warp instruction occupies for 64 cycles of its
// sub-partition however many lanes take part: neighbouring stars accept the same nodes, so the
// lanes share the instruction, while 32 separate walks in a warp drift apart and issue it for a few
// lanes at a time. One warp a block, so that few stars still spread over every SM. FP64 walk of
// 16,384 stars (theta 0.5, leaf 8): 24.4 ms with a thread a star, 8.0 ms so; 262,144 stars (leaf 24)
// 229 and 108 ms.
//
// accept(node, dx, dy, dz, d2) and pair(j) add the lane's own interaction. Returns the error code
// of a corrupt tree (each node is visited at most once), 0 otherwise.
template <class Accept, class Pair>
__device__ __forceinline__ int walk_lockstep(const gbh_node *__restrict__ nodes, int64_t nn, int64_t ns, bool valid,
                                             int32_t root, int32_t k, double x, double y, double z, int err_steps,
                                             int err_range, Accept accept, Pair pair) {
    if (nn <= 0) return 0;
    // a forest's warp may hold stars of several systems: one walk from each root
    unsigned todo = __ballot_sync(0xffffffffu, valid && root >= 0);
    while (todo) {
        const int32_t r0 = __shfl_sync(0xffffffffu, root, __ffs(todo) - 1);
        const bool mine = valid && root == r0;
        todo &= ~__ballot_sync(0xffffffffu, mine);
        int32_t resume = mine ? r0 : -2;
        int64_t steps = 0;
        for (int32_t i = r0; i >= 0;) {
            if (++steps > nn || i >= nn) return err_steps;
            const gbh_node &nd = nodes[i];
            const bool on = resume == i;
            const double dx = nd.x - x, dy = nd.y - y, dz = nd.z - z;
            const double d2 = dx * dx + dy * dy + dz * dz;
            const bool acc = on && d2 >= nd.crit2;
            const bool open = on && !acc;
            const int32_t first = nd.first, next = nd.next;
            const unsigned m_open = __ballot_sync(0xffffffffu, open);
            if (acc) {
                accept(nd, dx, dy, dz, d2);
                resume = next;
            }
            __syncwarp();
            if (!m_open) {
                i = next;
                continue;
            }
            if (first >= 0) {
                if (open) resume = first;
                i = first;
                continue;
            }
            const int32_t lo = nd.lo, hi = nd.hi;
            if (lo < 0 || hi > ns || lo > hi) return err_range;
            for (int32_t j = lo; j < hi; ++j)
                if (open && j != k) pair(j);
            __syncwarp();
            if (open) resume = next;
            i = next;
        }
    }
    return 0;
}

constexpr int kFp64Threads = 32;
__global__ __launch_bounds__(kFp64Threads) void k_walk_fp64(const DevInfo *info, const gbh_node *__restrict__ nodes,
                                                            const double *__restrict__ sx,
                                                            const double *__restrict__ sy,
                                                            const double *__restrict__ sz,
                                                            const double *__restrict__ sm,
                                                            const int32_t *__restrict__ order, double eps2, int quad,
                                                            int per, double *ax, double *ay, double *az,
                                                            const int32_t *__restrict__ targets,
                                                            const int32_t *__restrict__ sid_sorted,
                                                            const SysGeo *__restrict__ geo, DevInfo *err_info) {
    const int64_t t = int64_t(blockIdx.x) * per + threadIdx.x;
    const int64_t ns = info->nstars;
    const int64_t nt = targets ? int64_t(info->ntargets) : ns;
    if (t - threadIdx.x >= nt) return;  // the whole warp
    const bool valid = t < nt && int(threadIdx.x) < per;
    const int32_t k = valid ? (targets ? targets[t] : int32_t(t)) : 0;
    const double x = sx[k], y = sy[k], z = sz[k];
    double fax = 0, fay = 0, faz = 0;
    const int32_t root = sid_sorted ? geo[sid_sorted[k]].root : 0;  // the star's own system
    const int err = walk_lockstep(
        nodes, info->nnodes, ns, valid, root, k, x, y, z, 1, 7,
        [&](const gbh_node &nd, double dx, double dy, double dz, double d2) {
            double inv = 1 / (d2 + eps2);
            double inv3 = inv * sqrt(inv);
            double f = nd.m * inv3;
            if (quad) {
                double qx = nd.qxx * dx + nd.qxy * dy + nd.qxz * dz;
                double qy = nd.qxy * dx + nd.qyy * dy + nd.qyz * dz;
                double qz = nd.qxz * dx + nd.qyz * dy + nd.qzz * dz;
                double inv5 = inv3 * inv;
                f += 2.5 * (dx * qx + dy * qy + dz * qz) * inv5 * inv;
                fax -= qx * inv5;
                fay -= qy * inv5;
                faz -= qz * inv5;
            }
            fax += f * dx;
            fay += f * dy;
            faz += f * dz;
        },
        [&](int32_t j) {
            double ddx = sx[j] - x, ddy = sy[j] - y, ddz = sz[j] - z;
            double r2 = ddx * ddx + ddy * ddy + ddz * ddz + eps2;
            double f = sm[j] / (r2 * sqrt(r2));
            fax += f * ddx;
            fay += f * ddy;
            faz += f * ddz;
        });
    if (err && threadIdx.x == 0) dev_error(err_info, err);
    if (!valid) return;
    const int32_t o = order[k];
    ax[o] = fax;
    ay[o] = fay;
    az[o] = faz;
}

// ---------------------------------------------------------------- KDK (sim.go:302-343)

__global__ __launch_bounds__(kThreads) void k_kick(int64_t n, double h, double *vx, double *vy, double *vz,
                                                   const double *__restrict__ ax, const double *__restrict__ ay,
                                                   const double *__restrict__ az) {
    pdl_begin();
    int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    vx[i] += h * ax[i];
    vy[i] += h * ay[i];
    vz[i] += h * az[i];
}

// kick (sim.go:305-313) then drift (sim.go:315-343): x += dt u for c <= 0 (inv_c2 == 0), else
// x += dt u / sqrt(1 + u^2 / c^2) with the reference's 1 / c^2 factor inv_c2.
__global__ __launch_bounds__(kThreads) void k_kick_drift(int64_t n, double h, double dt, double inv_c2, double *px,
                                                         double *py, double *pz, double *vx, double *vy, double *vz,
                                                         const double *__restrict__ ax, const double *__restrict__ ay,
                                                         const double *__restrict__ az) {
    pdl_begin();
    int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double x = vx[i] + h * ax[i], y = vy[i] + h * ay[i], z = vz[i] + h * az[i];
    vx[i] = x;
    vy[i] = y;
    vz[i] = z;
    double f = dt;
    if (inv_c2 > 0) f = dt / sqrt(1 + (x * x + y * y + z * z) * inv_c2);
    px[i] += f * x;
    py[i] += f * y;
    pz[i] += f * z;
}

// ---------------------------------------------------------------- direct sum (direct.go:18-48)

// A sum of FP64 pair terms in the reference's order (ascending j) is a serial chain of adds, but
// the terms themselves are independent. A block takes T targets: its compute warps form the terms
// of T targets x J sources in shared memory (a thread keeps its source in registers and takes the
// targets in turn) while the add warps, one lane per target and axis, add the previous tile's
// terms in order, so every sum keeps its bits. One barrier a tile (two buffers). Skipped pairs
// leave a term of +0: the sums start at +0 and never become -0, so adding it changes nothing.
//
// The kernel is bound by the FP64 pipe (about 33 operations a pair, most of them the division and
// the square root), which needs every SM busy; one thread a target filled 32 of 152 SMs with
// 4,096 targets. T is chosen so that the blocks fill whole waves of two a SM: J = 64 sources a
// tile with up to 32 targets, or J = 256 with up to 8 (few targets: all compute threads still have
// a source). 4,096 targets of 131,072 bodies: 159 ms with a thread a target, 35.1 ms so (5.0e11 FP64
// operations/s of the 6.3e11 the pipe issues).
constexpr int kDirCompute = 256;  // compute threads; the add warps follow them
template <int kJ>
struct DirTile {
    static constexpr int kT = 2048 / kJ;                           // most targets of a block
    static constexpr int kStride = kJ + 1;                         // padded row: the add lanes hit all banks
    static constexpr int kRows = 3 * kT;
    static constexpr int kAdd = (kRows + 31) / 32 * 32;            // add threads
    static constexpr size_t kBytes = sizeof(double) * 2 * kRows * kStride;
};

template <int kJ>
__global__ __launch_bounds__(kDirCompute + DirTile<kJ>::kAdd) void k_direct_fp64(
    int64_t n, const double *__restrict__ px, const double *__restrict__ py, const double *__restrict__ pz,
    const double *__restrict__ mass, const uint8_t *__restrict__ kind, double eps2, int dm_off,
    const int64_t *__restrict__ targets, int64_t ntargets, int T, double *ax, double *ay, double *az) {
    using Tile = DirTile<kJ>;
    extern __shared__ double s_term[];  // [2][target][axis][kStride]
    __shared__ double s_x[Tile::kT], s_y[Tile::kT], s_z[Tile::kT];
    __shared__ int64_t s_i[Tile::kT];
    const int tid = threadIdx.x;
    const int64_t q0 = int64_t(blockIdx.x) * T;
    const int nt = ntargets - q0 < T ? int(ntargets - q0) : T;
    if (tid < nt) {
        const int64_t i = targets ? targets[q0 + tid] : q0 + tid;
        s_i[tid] = i;
        s_x[tid] = px[i];
        s_y[tid] = py[i];
        s_z[tid] = pz[i];
    }
    __syncthreads();
    const int64_t ntiles = (n + kJ - 1) / kJ;
    const bool adder = tid >= kDirCompute;
    const int a = tid - kDirCompute;  // add lane: target a / 3, axis a % 3
    const int jj = tid % kJ, g = tid / kJ;
    double x = 0, y = 0, z = 0, m = 0, sum = 0;
    bool skip = true;
    auto load = [&](int64_t tile) {
        const int64_t j = tile * kJ + jj;
        skip = j >= n;
        if (skip) return;
        const uint8_t kd = kind ? kind[j] : 0;
        skip = kd == GBH_BLACK_HOLE || (dm_off && kd == GBH_DARK_MATTER);
        x = px[j];
        y = py[j];
        z = pz[j];
        m = mass[j];
    };
    if (!adder) load(0);
    // tile t is formed while tile t - 1 is added
    for (int64_t t = 0; t <= ntiles; ++t) {
        if (!adder && t < ntiles) {
            const double xj = x, yj = y, zj = z, mj = m;
            const bool sk = skip;
            const int64_t j = t * kJ + jj;
            if (t + 1 < ntiles) load(t + 1);  // in flight during this tile's arithmetic
            double *row = s_term + size_t(t & 1) * Tile::kRows * Tile::kStride + jj;
            for (int k = g; k < nt; k += kDirCompute / kJ) {
                const double dx = xj - s_x[k], dy = yj - s_y[k], dz = zj - s_z[k];
                const double re2 = dx * dx + dy * dy + dz * dz + eps2;
                const double f = mj / (re2 * sqrt(re2));
                const bool off = sk || j == s_i[k];
                row[(3 * k) * Tile::kStride] = off ? 0.0 : f * dx;
                row[(3 * k + 1) * Tile::kStride] = off ? 0.0 : f * dy;
                row[(3 * k + 2) * Tile::kStride] = off ? 0.0 : f * dz;
            }
        } else if (adder && t > 0 && a < 3 * nt) {
            const double *row = s_term + (size_t((t - 1) & 1) * Tile::kRows + a) * Tile::kStride;
#pragma unroll 16
            for (int k = 0; k < kJ; ++k) sum += row[k];
        }
        __syncthreads();
    }
    if (!adder || a >= 3 * nt) return;
    const int64_t i = s_i[a / 3];
    if (kind && kind[i] == GBH_BLACK_HOLE) sum = 0;
    double *out = a % 3 == 0 ? ax : a % 3 == 1 ? ay : az;
    out[q0 + a / 3] = sum;
}

// ---------------------------------------------------------------- potential (potential.go:16-81)

__device__ __forceinline__ double schwarzschild(double m, double c) { return c <= 0 ? 0 : 2 * m / (c * c); }

__device__ __forceinline__ double pair_rs(uint8_t ki, double mi, uint8_t kj, double mj, double c) {
    bool hi = ki == GBH_BLACK_HOLE, hj = kj == GBH_BLACK_HOLE;
    if (c <= 0 || hi == hj) return 0;
    return hi ? schwarzschild(mi, c) : schwarzschild(mj, c);
}

__device__ __forceinline__ double pair_potential(double mi, double mj, double r2, double eps2, double rs) {
    double re = sqrt(r2 + eps2);
    if (rs == 0) return -mi * mj / re;
    if (re >= 1.5 * rs) return -mi * mj / (re - rs);
    return mi * mj * (-2 / rs + 4 / (rs * rs) * (re - 1.5 * rs));
}

// PotentialEnergyParallel (diag.go:42-64): row i of the exact pair sum, sum over j > i of the
// pair model's potential in ascending j, kinds and liveness as the reference reads them (all
// bodies). The rows are then added in ascending i (the reference adds its ParallelFor chunks
// in completion order, so only round-off may differ).
//
// As in k_direct_fp64, the compute threads form a tile's terms and one add lane a row adds them in
// order. Bound by the FP64 pipe (about 28 operations a pair). A block takes T rows, few enough
// that the blocks fill every SM several times over (the rows shorten, so the longest blocks are
// launched first and the short ones fill the end). 30,000 bodies: 44.8 ms with one thread a row
// and one thread adding the rows from global memory, 28.3 ms so, 25.8 without a radius to form and
// compare (kNewton: every pair, when there is no speed of light).
constexpr int kPotRows = 32, kPotJ = 64;
constexpr int kPotStride = kPotJ + 1;
template <bool kNewton>
__global__ __launch_bounds__(kDirCompute + 32) void k_pot_exact_rows(int64_t n, const double *__restrict__ px,
                                                                     const double *__restrict__ py,
                                                                     const double *__restrict__ pz,
                                                                     const double *__restrict__ mass,
                                                                     const uint8_t *__restrict__ kind, double eps2,
                                                                     double c, int dm_off, int T, double *rows) {
    __shared__ double s_term[2][kPotRows][kPotStride];
    __shared__ double s_x[kPotRows], s_y[kPotRows], s_z[kPotRows], s_m[kPotRows];
    __shared__ uint8_t s_k[kPotRows];
    const int tid = threadIdx.x;
    const int64_t i0 = int64_t(blockIdx.x) * T;
    const int nt = n - i0 < T ? int(n - i0) : T;
    if (tid < nt) {
        s_x[tid] = px[i0 + tid];
        s_y[tid] = py[i0 + tid];
        s_z[tid] = pz[i0 + tid];
        s_m[tid] = mass[i0 + tid];
        s_k[tid] = kind ? kind[i0 + tid] : 0;
    }
    __syncthreads();
    const int64_t ntiles = (n - i0 + kPotJ - 1) / kPotJ;
    const bool adder = tid >= kDirCompute;
    const int a = tid - kDirCompute;
    const int jj = tid % kPotJ, g = tid / kPotJ;
    double x = 0, y = 0, z = 0, m = 0, sum = 0;
    uint8_t kd = 0;
    auto load = [&](int64_t tile) {
        const int64_t j = i0 + tile * kPotJ + jj;
        if (j >= n) return;
        kd = kind ? kind[j] : 0;
        x = px[j];
        y = py[j];
        z = pz[j];
        m = mass[j];
    };
    if (!adder) load(0);
    for (int64_t t = 0; t <= ntiles; ++t) {
        if (!adder && t < ntiles) {
            const double xj = x, yj = y, zj = z, mj = m;
            const uint8_t kj = kd;
            const int64_t j = i0 + t * kPotJ + jj;
            if (t + 1 < ntiles) load(t + 1);
            const double smj = dm_off && kj == GBH_DARK_MATTER ? 0.0 : mj;
            for (int k = g; k < nt; k += kDirCompute / kPotJ) {
                const double dx = xj - s_x[k], dy = yj - s_y[k], dz = zj - s_z[k];
                const uint8_t ki = s_k[k];
                const double mi = s_m[k];
                const double smi = dm_off && ki == GBH_DARK_MATTER ? 0.0 : mi;
                const double r2 = dx * dx + dy * dy + dz * dz;
                const double v = kNewton ? -smi * smj / sqrt(r2 + eps2)
                                         : pair_potential(smi, smj, r2, eps2, pair_rs(ki, mi, kj, mj, c));
                s_term[t & 1][k][jj] = j < n && j > i0 + k ? v : 0.0;
            }
        } else if (adder && t > 0 && a < nt) {
            const double *row = s_term[(t - 1) & 1][a];
#pragma unroll 16
            for (int k = 0; k < kPotJ; ++k) sum += row[k];
        }
        __syncthreads();
    }
    if (adder && a < nt) rows[i0 + a] = sum;
}

// The rows added in ascending i by one thread, from tiles that the block stages in shared memory.
constexpr int kPotFinal = 2048;
__global__ __launch_bounds__(kThreads) void k_pot_exact_final(int64_t n, const double *__restrict__ rows, double *out) {
    __shared__ double s[2][kPotFinal];
    double sum = 0;
    const int64_t ntiles = (n + kPotFinal - 1) / kPotFinal;
    for (int64_t t = 0; t <= ntiles; ++t) {
        if (t < ntiles && threadIdx.x >= 32)
            for (int k = threadIdx.x - 32; k < kPotFinal; k += kThreads - 32)
                s[t & 1][k] = t * kPotFinal + k < n ? rows[t * kPotFinal + k] : 0.0;  // + 0: no change
        if (t > 0 && threadIdx.x == 0) {
#pragma unroll 16
            for (int k = 0; k < kPotFinal; ++k) sum += s[(t - 1) & 1][k];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = sum;
}

// holePotential, potential.go:84-96.
__device__ double hole_potential(int64_t i, const double *px, const double *py, const double *pz, const double *mass,
                                 const uint8_t *kind, const int32_t *holes, int32_t nholes, double eps2, double c,
                                 int dm_off) {
    double x = px[i], y = py[i], z = pz[i], u = 0;
    uint8_t ki = kind ? kind[i] : 0;
    double smi = (dm_off && ki == GBH_DARK_MATTER) ? 0.0 : mass[i];
    for (int32_t t = 0; t < nholes; ++t) {
        int32_t h = holes[t];
        if (h == i) continue;
        double dx = px[h] - x, dy = py[h] - y, dz = pz[h] - z;
        double rs = pair_rs(ki, mass[i], GBH_BLACK_HOLE, mass[h], c);
        u += pair_potential(smi, mass[h], dx * dx + dy * dy + dz * dz, eps2, rs);
    }
    return u;
}

// Per sorted star: sm[k] * walkPotential(k) - holePotential(order[k]); block partial sums.
__global__ __launch_bounds__(kThreads) void k_potential_walk(const DevInfo *info, const gbh_node *__restrict__ nodes,
                                                             const double *__restrict__ sx, const double *__restrict__ sy,
                                                             const double *__restrict__ sz, const double *__restrict__ sm,
                                                             const int32_t *__restrict__ order, const double *px,
                                                             const double *py, const double *pz, const double *mass,
                                                             const uint8_t *kind, const int32_t *holes, int32_t nholes,
                                                             double eps2, double c, int dm_off, int quad, double *part,
                                                             const int32_t *__restrict__ sid_sorted,
                                                             const SysGeo *__restrict__ geo, DevInfo *err_info) {
    int64_t k = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    int64_t ns = info->nstars, nn = info->nnodes;
    double v = 0, psi = 0;
    const bool valid = k < ns;
    const int32_t kk = valid ? int32_t(k) : 0;
    const double x = ns ? sx[kk] : 0, y = ns ? sy[kk] : 0, z = ns ? sz[kk] : 0;
    const int32_t root = ns && sid_sorted ? geo[sid_sorted[kk]].root : 0;
    const int err = walk_lockstep(
        nodes, nn, ns, valid, root, kk, x, y, z, 2, 2,
        [&](const gbh_node &nd, double dx, double dy, double dz, double d2) {
            double inv = 1 / (d2 + eps2);
            psi += nd.m * sqrt(inv);
            if (quad) {
                double dqd = nd.qxx * dx * dx + nd.qyy * dy * dy + nd.qzz * dz * dz +
                             2 * (nd.qxy * dx * dy + nd.qxz * dx * dz + nd.qyz * dy * dz);
                psi += 0.5 * dqd * inv * inv * sqrt(inv);
            }
        },
        [&](int32_t j) {
            double ddx = sx[j] - x, ddy = sy[j] - y, ddz = sz[j] - z;
            psi += sm[j] / sqrt(ddx * ddx + ddy * ddy + ddz * ddz + eps2);
        });
    if (err && (threadIdx.x & 31) == 0) dev_error(err_info, err);
    if (valid)
        v = sm[k] * psi - (nholes ? hole_potential(order[k], px, py, pz, mass, kind, holes, nholes, eps2, c, dm_off) : 0.0);
    // Deterministic block sum (tree order over threads).
    __shared__ double s[kThreads];
    s[threadIdx.x] = v;
    __syncthreads();
    for (int o = kThreads / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = s[0];
}

// Sum of the block parts plus the hole terms (potential.go:31-41); U = -sum / 2.
__global__ void k_potential_final(int64_t nparts, const double *part, const DevInfo *info,
                                  const double *__restrict__ sx, const double *__restrict__ sy,
                                  const double *__restrict__ sz, const double *__restrict__ sm, const double *px,
                                  const double *py, const double *pz, const double *mass, const uint8_t *kind,
                                  const int32_t *holes, int32_t nholes, double eps2, double c, int dm_off, double *u) {
    __shared__ double s[kThreads];
    double v = 0;
    for (int64_t b = threadIdx.x; b < nparts; b += blockDim.x) v += part[b];
    int64_t ns = info->nstars;
    for (int32_t t = 0; t < nholes; ++t) {
        int32_t i = holes[t];
        double x = px[i], y = py[i], z = pz[i];
        double rs = schwarzschild(mass[i], c);
        for (int64_t k = threadIdx.x; k < ns; k += blockDim.x) {
            double dx = sx[k] - x, dy = sy[k] - y, dz = sz[k] - z;
            v -= pair_potential(mass[i], sm[k], dx * dx + dy * dy + dz * dz, eps2, rs);
        }
        if (threadIdx.x == 0) v -= hole_potential(i, px, py, pz, mass, kind, holes, nholes, eps2, c, dm_off);
    }
    s[threadIdx.x] = v;
    __syncthreads();
    for (int o = kThreads / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) *u = -s[0] / 2;
}

}  // namespace

// ---------------------------------------------------------------- forests (many systems)

namespace {

// Each system's root (the pre-order index of its first star's chain) and its entries of the
// mixed walk's group table; a block a system.
__global__ __launch_bounds__(128) void k_sys_groups(int32_t gsize, const uint32_t *__restrict__ base, SysGeo *geo,
                                                    int4 *__restrict__ groups) {
    pdl_begin();
    SysGeo &g = geo[blockIdx.x];
    const int32_t lo = g.star_lo, hi = g.star_hi, glo = g.group_lo, ng = g.ngroups;
    const int32_t root = hi > lo ? int32_t(base[lo]) : -1;
    if (threadIdx.x == 0) g.root = root;
    for (int32_t q = threadIdx.x; q < ng; q += blockDim.x) {
        const int32_t start = lo + gsize * q;
        groups[glo + q] = make_int4(start, hi - start < gsize ? hi - start : gsize, root, 0);
    }
}

}  // namespace

void tree_free(TreeBufs &b) {
    void *ptrs[] = {b.pos4, b.bbox_part, b.keys, b.keys_alt, b.order, b.order_alt, b.lb_state, b.tile_len, b.hist, b.sx, b.sy, b.sz, b.sm,
                    b.st_hi, b.st_lo, b.st_off, b.chain_base, b.leaves, b.targets, b.geo, b.sid_sorted, b.groups, b.gcost, b.gperm, b.pre_parent, b.pre_info, b.child_base, b.pre_mask, b.pre_hi, b.pre_star, b.nodes,
                    b.n_parent, b.n_info, b.n_arrive, b.pnodes, b.mnodes, b.mrange, b.lnode, b.walk_ctr, b.next_part, b.info, b.part_acc};
    for (void *p : ptrs)
        if (p) cudaFree(p);
    b = TreeBufs{};
}

// Worst-case node count: at most n leaves, and at each of the 22 levels at most n/(leaf+1)
// cells hold more than leaf stars (only those have children).
static int64_t node_capacity(int64_t n, int leaf) { return n + 22 * (n / (leaf + 1) + 1) + 1; }

cudaError_t tree_alloc(TreeBufs &b, cudaStream_t stream, int64_t n, int leaf, int32_t nsys) {
    int64_t need_nodes = node_capacity(n, leaf);
    if (nsys < 1) nsys = 1;
    if (n <= b.cap_n && need_nodes <= b.cap_nodes && nsys <= b.cap_sys && n / 32 + nsys + 1 <= b.cap_groups) {
        b.nsys = nsys;
        return split_reserve(b, n);
    }
    if (nsys > b.cap_sys) b.cap_sys = 0;
    int64_t cn = n > b.cap_n ? n + n / 4 : b.cap_n;  // grow by 1.25x like gpuBuffers.ensure (gpu_darwin.go:164-177)
    int64_t cnodes = need_nodes > b.cap_nodes ? node_capacity(cn, leaf) : b.cap_nodes;
    if (cnodes < need_nodes) cnodes = need_nodes;
    const int64_t gen = b.generation + 1;
    tree_free(b);
    b.generation = gen;
    cn = cn < 1 ? 1 : cn;
    cudaError_t e = cudaSuccess;
#define GBH_ALLOC(ptr, count)                                                     \
    do {                                                                          \
        if (e == cudaSuccess) e = dev_alloc(&(ptr), sizeof(*(ptr)) * size_t(count)); \
    } while (0)
    GBH_ALLOC(b.pos4, cn);
    if (e == cudaSuccess) e = dev_alloc(&b.bbox_part, sort_part_bytes());
    GBH_ALLOC(b.keys, cn);
    GBH_ALLOC(b.keys_alt, cn);
    GBH_ALLOC(b.order, cn);
    GBH_ALLOC(b.order_alt, cn);
    GBH_ALLOC(b.sx, cn);
    GBH_ALLOC(b.sy, cn);
    GBH_ALLOC(b.sz, cn);
    GBH_ALLOC(b.sm, cn);
    GBH_ALLOC(b.st_hi, cn);
    GBH_ALLOC(b.st_lo, cn);
    GBH_ALLOC(b.st_off, cn);
    GBH_ALLOC(b.chain_base, cn);
    GBH_ALLOC(b.leaves, cn);
    GBH_ALLOC(b.targets, cn);
    const int32_t csys = nsys + nsys / 4 + 1;
    const int64_t cgroups = cn / 32 + csys + 1;  // groups of 32 or 64 stars
    GBH_ALLOC(b.geo, csys);
    GBH_ALLOC(b.sid_sorted, cn);
    GBH_ALLOC(b.groups, cgroups);
    GBH_ALLOC(b.gcost, cgroups);
    GBH_ALLOC(b.gperm, cgroups + 1);
    GBH_ALLOC(b.pre_parent, cnodes);
    GBH_ALLOC(b.pre_info, cnodes);
    GBH_ALLOC(b.child_base, cnodes);
    GBH_ALLOC(b.pre_mask, cnodes);
    GBH_ALLOC(b.pre_hi, cnodes);
    GBH_ALLOC(b.pre_star, cnodes);
    GBH_ALLOC(b.nodes, cnodes);
    GBH_ALLOC(b.n_parent, cnodes);
    GBH_ALLOC(b.n_info, cnodes);
    GBH_ALLOC(b.n_arrive, cnodes);
    GBH_ALLOC(b.pnodes, cnodes);
    GBH_ALLOC(b.mnodes, cnodes);
    GBH_ALLOC(b.mrange, cnodes);
    GBH_ALLOC(b.lnode, cnodes);
    GBH_ALLOC(b.walk_ctr, 16);
    // single-pass scans: the chain counts', the child counts', the active-star lists' and the large sort's
    b.lb_targets = lb_words_of(chain_tiles(cn)) + lb_words_of(child_tiles(cnodes));
    b.lb_sort = b.lb_targets + lb_words_of(target_tiles(cn));
    const int64_t lb_words = b.lb_sort + sort_lb_words(cn);
    GBH_ALLOC(b.lb_state, lb_words);
    const int64_t ctiles = cn / kSortTile + csys + 1;  // sort tiles never straddle systems
    GBH_ALLOC(b.tile_len, 2 * ctiles);
    GBH_ALLOC(b.hist, sort_hist_words(cn));
    GBH_ALLOC(b.next_part, kNextBlocks);
    GBH_ALLOC(b.info, 1);
#undef GBH_ALLOC
    if (e != cudaSuccess) {
        tree_free(b);
        return e;
    }
    b.cap_n = cn;
    b.cap_nodes = cnodes;
    b.lb_words = lb_words;
    b.cap_tiles = ctiles;
    b.cap_sys = csys;
    b.cap_groups = cgroups;
    b.nsys = nsys;
    // no launch order yet: gperm[cap_groups] = -1 matches no group count; bbox_done and next_done wrap
    // to 0 by themselves and must start there
    if ((e = cudaMemsetAsync(b.gperm, 0xff, sizeof(int32_t) * size_t(cgroups + 1), stream)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(b.info, 0, sizeof(DevInfo), stream)) != cudaSuccess) return e;
    return split_reserve(b, n);
}

#define GBH_LAUNCH_CHECK()                         \
    do {                                           \
        ++*L.count;                                \
        cudaError_t e_ = cudaGetLastError();       \
        if (e_ != cudaSuccess) return e_;          \
    } while (0)

cudaError_t tree_build(const Launch &L, TreeBufs &b, int64_t n, const double *px, const double *py, const double *pz,
                       const double *mass, const uint8_t *kind, const uint8_t *alive, double *ax, double *ay,
                       double *az, double theta, int leaf, int dm_off, bool exact, bool plain_records,
                       const ForestTiles *forest_tiles) {
    cudaStream_t s = L.stream;
    const bool forest = b.nsys > 1;
    if (forest && !forest_tiles) return cudaErrorInvalidValue;
    cudaError_t e = sort_stars(L, b, n, px, py, pz, mass, kind, alive, ax, ay, az, theta, dm_off, exact,
                               forest ? forest_tiles : nullptr);
    if (e != cudaSuccess) return e;
    // node set
    const int32_t *sid = forest ? b.sid_sorted : nullptr;
    GBH_LAUNCH_AFTER(L, k_chains, unsigned(chain_tiles(n)), kChainThreads, b.keys, b.info, sid, b.geo, leaf,
                     b.chain_base, b.pre_star, b.pre_info, b.pre_mask, b.lb_state, b.cap_nodes);
    const unsigned nbn = node_blocks(b.cap_nodes);
    GBH_LAUNCH_AFTER(L, k_topology, nbn, kThreads, b.keys, b.info, b.chain_base, b.pre_star, b.pre_info, b.pre_mask,
                     b.pre_parent, b.pre_hi, sid, b.geo, b.cap_nodes);
    GBH_LAUNCH_AFTER(L, k_child_scan, unsigned(child_tiles(b.cap_nodes)), kScanThreads, b.pre_mask, b.child_base,
                     b.cap_nodes, b.lb_state + lb_words_of(chain_tiles(b.cap_n)), b.info);
    GBH_LAUNCH_AFTER(L, k_emit_nodes, nbn, kThreads, b.info, b.chain_base, b.pre_star, b.pre_parent, b.pre_info,
                     b.pre_mask, b.pre_hi, b.child_base, b.nodes, b.n_parent, b.n_info, b.n_arrive, b.leaves, sid,
                     b.geo, b.cap_nodes);
    if (forest) {
        GBH_LAUNCH_AFTER(L, k_sys_groups, unsigned(b.nsys), 128, b.group == 32 ? 32 : 64, b.chain_base, b.geo,
                         b.groups);
    }
    b.moments_exact = exact;
    if (!exact) return upsweep_fast(L, b, plain_records);
    k_upsweep<<<blocks_for(n, kThreads), kThreads, 0, s>>>(b.keys, b.info, b.leaves, b.sx, b.sy, b.sz, b.sm, b.nodes,
                                                           b.n_parent, b.n_info, b.n_arrive, b.pnodes, b.mnodes,
                                                           b.mrange, sid, b.geo, b.info);
    GBH_LAUNCH_CHECK();
    return cudaSuccess;
}

namespace {
__global__ __launch_bounds__(kThreads) void k_fault_link(const DevInfo *info, gbh_node *nodes, PNode *pnodes,
                                                         MNode *mnodes, LNode *lnode, int64_t cap) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= info->nnodes || i >= cap) return;
    if (nodes[i].next != -1 || nodes[i].first != -1) return;
    nodes[i].next = 0;
    pnodes[i].links.y = 0;
    mnodes[i].d.w = __int_as_float(0);
    lnode[i].a.w = fabsf(lnode[i].a.w);  // the list walk: the leaf becomes an inner node whose child is node 0
    lnode[i].b.w = __int_as_float(0);
}
}  // namespace

cudaError_t fault_link(const Launch &L, TreeBufs &b) {
    k_fault_link<<<blocks_for(b.cap_nodes, kThreads), kThreads, 0, L.stream>>>(b.info, b.nodes, b.pnodes, b.mnodes,
                                                                               b.lnode, b.cap_nodes);
    GBH_LAUNCH_CHECK();
    return cudaSuccess;
}

cudaError_t walk_fp64(const Launch &L, const TreeBufs &b, int64_t n, double eps2, int quad, double *ax, double *ay,
                      double *az, bool targets) {
    // Stars a warp: 32, fewer while every warp still has an FP64 pipe of its own (four an SM). Fewer
    // stars share a shorter walk, but an instruction costs the pipe the same for 4 lanes as for 32.
    // Walks with 32, 16, 8 and 4 stars a warp: 1,000 stars (theta 0.9) 1.13, 1.09, 1.03, 0.95 ms; 4,096
    // (theta 0.5) 4.68, 4.22, 3.99, 4.93; 16,384 8.39, 9.92, 15.7, 25.8.
    const int pipes = 4 * (L.num_sms > 0 ? L.num_sms : 152);
    const int per = n <= 4 * pipes ? 4 : n <= 8 * pipes ? 8 : n <= 16 * pipes ? 16 : kFp64Threads;
    k_walk_fp64<<<blocks_for(b.cap_n, per), kFp64Threads, 0, L.stream>>>(
        b.info, b.nodes, b.sx, b.sy, b.sz, b.sm, b.order, eps2, quad, per, ax, ay, az, targets ? b.targets : nullptr,
        b.nsys > 1 ? b.sid_sorted : nullptr, b.geo, b.info);
    GBH_LAUNCH_CHECK();
    return cudaSuccess;
}

cudaError_t kick(const Launch &L, int64_t n, double h, double *vx, double *vy, double *vz, const double *ax,
                 const double *ay, const double *az) {
    if (n == 0) return cudaSuccess;
    GBH_LAUNCH_AFTER(L, k_kick, blocks_for(n, kThreads), kThreads, n, h, vx, vy, vz, ax, ay, az);
    return cudaSuccess;
}

cudaError_t kick_drift(const Launch &L, int64_t n, double h, double dt, double c, double *px, double *py, double *pz,
                       double *vx, double *vy, double *vz, const double *ax, const double *ay, const double *az) {
    if (n == 0) return cudaSuccess;
    const double inv_c2 = c > 0 ? 1 / (c * c) : 0.0;  // sim.go:335 (invC2)
    GBH_LAUNCH_AFTER(L, k_kick_drift, blocks_for(n, kThreads), kThreads, n, h, dt, inv_c2, px, py, pz, vx, vy, vz, ax, ay,
                     az);
    return cudaSuccess;
}

template <int kJ>
static cudaError_t launch_direct(const Launch &L, int64_t n, const double *px, const double *py, const double *pz,
                                 const double *mass, const uint8_t *kind, double eps2, int dm_off,
                                 const int64_t *targets, int64_t ntargets, int T, double *ax, double *ay, double *az) {
    using Tile = DirTile<kJ>;
    // set on every call: the attribute belongs to the current device
    cudaError_t e = cudaFuncSetAttribute(k_direct_fp64<kJ>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(Tile::kBytes));
    if (e != cudaSuccess) return e;
    k_direct_fp64<kJ><<<blocks_for(ntargets, T), kDirCompute + Tile::kAdd, Tile::kBytes, L.stream>>>(
        n, px, py, pz, mass, kind, eps2, dm_off, targets, ntargets, T, ax, ay, az);
    GBH_LAUNCH_CHECK();
    return cudaSuccess;
}

cudaError_t direct_fp64(const Launch &L, int64_t n, const double *px, const double *py, const double *pz,
                        const double *mass, const uint8_t *kind, double eps2, int dm_off, const int64_t *targets,
                        int64_t ntargets, double *ax, double *ay, double *az) {
    if (ntargets == 0 || n == 0) return cudaSuccess;
    // two blocks a SM are resident: as few targets a block as fill whole waves of them
    const int64_t wave = 2 * int64_t(L.num_sms > 0 ? L.num_sms : 152);
    const int64_t waves = (ntargets + wave * DirTile<64>::kT - 1) / (wave * DirTile<64>::kT);
    const int T = int((ntargets + waves * wave - 1) / (waves * wave));
    if (T <= DirTile<256>::kT)
        return launch_direct<256>(L, n, px, py, pz, mass, kind, eps2, dm_off, targets, ntargets, T, ax, ay, az);
    return launch_direct<64>(L, n, px, py, pz, mass, kind, eps2, dm_off, targets, ntargets, T, ax, ay, az);
}

// Potential from the mixed walk's psi (sorted order): the block sums of m_k psi_k minus each
// star's hole pairs, as k_potential_walk forms them from the FP64 walk.
__global__ __launch_bounds__(kThreads) void k_potential_parts_psi(const DevInfo *info, const int32_t *__restrict__ order,
                                                                  const double *__restrict__ psi, const double *px,
                                                                  const double *py, const double *pz,
                                                                  const double *mass, const uint8_t *kind,
                                                                  const int32_t *holes, int32_t nholes, double eps2,
                                                                  double c, int dm_off, double *part) {
    int64_t k = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    double v = 0;
    if (k < info->nstars) {
        int32_t i = order[k];
        double smi = (dm_off && kind && kind[i] == GBH_DARK_MATTER) ? 0.0 : mass[i];
        v = smi * psi[k] - (nholes ? hole_potential(i, px, py, pz, mass, kind, holes, nholes, eps2, c, dm_off) : 0.0);
    }
    __shared__ double s[kThreads];
    s[threadIdx.x] = v;
    __syncthreads();
    for (int o = kThreads / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = s[0];
}

// U = -(parts - hole pairs) / 2, the hole-star pairs taken over the alive non-hole bodies in
// state order (k_potential_final takes them over the sorted copies).
__global__ void k_potential_final_state(int64_t nparts, const double *part, int64_t n, const double *px,
                                        const double *py, const double *pz, const double *mass, const uint8_t *kind,
                                        const uint8_t *alive, const int32_t *holes, int32_t nholes, double eps2,
                                        double c, int dm_off, double *u) {
    __shared__ double s[kThreads];
    double v = 0;
    for (int64_t b = threadIdx.x; b < nparts; b += blockDim.x) v += part[b];
    for (int32_t t = 0; t < nholes; ++t) {
        int32_t i = holes[t];
        double x = px[i], y = py[i], z = pz[i];
        double rs = schwarzschild(mass[i], c);
        for (int64_t j = threadIdx.x; j < n; j += blockDim.x) {
            uint8_t kj = kind ? kind[j] : 0;
            if (kj == GBH_BLACK_HOLE || (alive && !alive[j])) continue;
            double smj = (dm_off && kj == GBH_DARK_MATTER) ? 0.0 : mass[j];
            double dx = px[j] - x, dy = py[j] - y, dz = pz[j] - z;
            v -= pair_potential(mass[i], smj, dx * dx + dy * dy + dz * dz, eps2, rs);
        }
        if (threadIdx.x == 0) v -= hole_potential(i, px, py, pz, mass, kind, holes, nholes, eps2, c, dm_off);
    }
    s[threadIdx.x] = v;
    __syncthreads();
    for (int o = kThreads / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) *u = -s[0] / 2;
}

cudaError_t potential_exact_fp64(const Launch &L, int64_t n, const double *px, const double *py, const double *pz,
                                 const double *mass, const uint8_t *kind, double eps2, double c, int dm_off,
                                 double *rows, double *u_dev) {
    // about four blocks a SM or more
    const int64_t per = n / (4 * int64_t(L.num_sms > 0 ? L.num_sms : 152));
    const int T = int(per < 1 ? 1 : per > kPotRows ? kPotRows : per);
    // without a speed of light every pair is Newtonian (pair.go:14-23): no radius to form and compare
    auto *kernel = c <= 0 ? k_pot_exact_rows<true> : k_pot_exact_rows<false>;
    kernel<<<blocks_for(n, T), kDirCompute + 32, 0, L.stream>>>(n, px, py, pz, mass, kind, eps2, c, dm_off, T, rows);
    GBH_LAUNCH_CHECK();
    k_pot_exact_final<<<1, kThreads, 0, L.stream>>>(n, rows, u_dev);
    GBH_LAUNCH_CHECK();
    return cudaSuccess;
}

cudaError_t potential_mixed(const Launch &L, const TreeBufs &b, int64_t n, const double *px, const double *py,
                            const double *pz, const double *mass, const uint8_t *kind, const uint8_t *alive,
                            const int32_t *holes, int32_t nholes, double eps2, double c, int dm_off, int quad,
                            double *psi, double *part, double *u_dev) {
    cudaError_t e = walk_mixed_potential(L, b, b.cap_n, float(eps2), quad, psi);
    if (e != cudaSuccess) return e;
    unsigned nb = blocks_for(b.cap_n, kThreads);
    k_potential_parts_psi<<<nb, kThreads, 0, L.stream>>>(b.info, b.order, psi, px, py, pz, mass, kind, holes, nholes,
                                                         eps2, c, dm_off, part);
    GBH_LAUNCH_CHECK();
    k_potential_final_state<<<1, kThreads, 0, L.stream>>>(nb, part, n, px, py, pz, mass, kind, alive, holes, nholes,
                                                          eps2, c, dm_off, u_dev);
    GBH_LAUNCH_CHECK();
    return cudaSuccess;
}

cudaError_t potential_fp64(const Launch &L, const TreeBufs &b, int64_t n, const double *px, const double *py,
                           const double *pz, const double *mass, const uint8_t *kind, const uint8_t *alive,
                           const int32_t *holes, int32_t nholes, double eps2, double c, int dm_off, int quad,
                           double *part, double *u_dev) {
    (void)n;
    (void)alive;
    unsigned nb = blocks_for(b.cap_n, kThreads);
    k_potential_walk<<<nb, kThreads, 0, L.stream>>>(b.info, b.nodes, b.sx, b.sy, b.sz, b.sm, b.order, px, py, pz, mass,
                                                    kind, holes, nholes, eps2, c, dm_off, quad, part,
                                                    b.nsys > 1 ? b.sid_sorted : nullptr, b.geo, b.info);
    GBH_LAUNCH_CHECK();
    k_potential_final<<<1, kThreads, 0, L.stream>>>(nb, part, b.info, b.sx, b.sy, b.sz, b.sm, px, py, pz, mass, kind,
                                                    holes, nholes, eps2, c, dm_off, u_dev);
    GBH_LAUNCH_CHECK();
    return cudaSuccess;
}

}  // namespace gbh

namespace gbh {

// ---------------------------------------------------------------- diagnostics (diag.go:31-135)

namespace {

constexpr int kDiagBlocksMax = 1024;
constexpr int kDiagSums = 11;  // kinetic, p(3), L(3), m x (3), m

// Per-block sums over bodies i (all bodies, as Momentum/AngularMomentum/CenterOfMass iterate
// s.Len(); kinetic over the bodies that gravitate, sourceKinetic diag.go:66-76).
__global__ __launch_bounds__(kThreads) void k_diag_partial(int64_t n, const double *__restrict__ px,
                                                           const double *__restrict__ py, const double *__restrict__ pz,
                                                           const double *__restrict__ vx, const double *__restrict__ vy,
                                                           const double *__restrict__ vz,
                                                           const double *__restrict__ mass,
                                                           const uint8_t *__restrict__ kind, double c, int dm_off,
                                                           double *__restrict__ part) {
    double acc[kDiagSums] = {};
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
        double m = mass[i], x = px[i], y = py[i], z = pz[i], ux = vx[i], uy = vy[i], uz = vz[i];
        uint8_t kd = kind ? kind[i] : 0;
        bool source = !(dm_off && kd == GBH_DARK_MATTER);
        double u2 = ux * ux + uy * uy + uz * uz;
        double g = c <= 0 ? 1.0 : sqrt(1 + u2 / (c * c));  // gamma, relativity.go:15-20
        if (source) acc[0] += m * u2 / (g + 1);           // kinetic, relativity.go:22-26
        acc[1] += m * ux;
        acc[2] += m * uy;
        acc[3] += m * uz;
        acc[4] += m * (y * uz - z * uy);
        acc[5] += m * (z * ux - x * uz);
        acc[6] += m * (x * uy - y * ux);
        acc[7] += m * x;
        acc[8] += m * y;
        acc[9] += m * z;
        acc[10] += m;
    }
    __shared__ double s[kThreads];
    for (int q = 0; q < kDiagSums; ++q) {
        s[threadIdx.x] = acc[q];
        __syncthreads();
        for (int o = kThreads / 2; o > 0; o >>= 1) {
            if (threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
            __syncthreads();
        }
        if (threadIdx.x == 0) part[blockIdx.x * kDiagSums + q] = s[0];
        __syncthreads();
    }
}

// Each sum's block parts in block order: staged in shared memory by the whole block, added by one
// lane a sum (1,024 parts: 11 threads reading them from global memory took 40 us).
__global__ __launch_bounds__(kThreads) void k_diag_final(int nparts, const double *__restrict__ part, double *out) {
    constexpr int kTile = 128;  // parts a tile
    __shared__ double s[kTile * kDiagSums];
    double v = 0;
    for (int b0 = 0; b0 < nparts; b0 += kTile) {
        const int cnt = nparts - b0 < kTile ? nparts - b0 : kTile;
        for (int k = threadIdx.x; k < cnt * kDiagSums; k += kThreads) s[k] = part[b0 * kDiagSums + k];
        __syncthreads();
        if (threadIdx.x < kDiagSums) {
#pragma unroll 8
            for (int b = 0; b < cnt; ++b) v += s[b * kDiagSums + threadIdx.x];
        }
        __syncthreads();
    }
    if (threadIdx.x < kDiagSums) out[threadIdx.x] = v;
}

}  // namespace

int diag_parts() { return kDiagBlocksMax; }

cudaError_t diagnostics(const Launch &L, int64_t n, const double *px, const double *py, const double *pz,
                        const double *vx, const double *vy, const double *vz, const double *mass, const uint8_t *kind,
                        double c, int dm_off, double *part, double *out) {
    unsigned nb = blocks_for(n, kThreads);
    if (nb > unsigned(kDiagBlocksMax)) nb = kDiagBlocksMax;
    k_diag_partial<<<nb, kThreads, 0, L.stream>>>(n, px, py, pz, vx, vy, vz, mass, kind, c, dm_off, part);
    GBH_LAUNCH_CHECK();
    k_diag_final<<<1, kThreads, 0, L.stream>>>(int(nb), part, out);
    GBH_LAUNCH_CHECK();
    return cudaSuccess;
}

}  // namespace gbh

namespace gbh {

// ---------------------------------------------------------------- active-star lists (block steps)

namespace {

// The active stars' sorted positions in order, in one launch: flags ranked by ballots, tiles by
// look-back. A block takes the next tile of 1,024 positions.
__global__ __launch_bounds__(kTargetThreads) void k_targets(DevInfo *info, const int32_t *__restrict__ order,
                                                            const int32_t *__restrict__ end, int32_t tick,
                                                            int32_t *__restrict__ targets, uint32_t *lb) {
    pdl_begin();
    __shared__ uint32_t s_warp[kTargetThreads / 32 + 1];
    __shared__ uint32_t s_tile, s_prefix;
    if (threadIdx.x == 0) s_tile = atomicAdd(lb, 1u);
    __syncthreads();
    const uint32_t tile = s_tile;
    const int64_t ns = info->nstars;
    const int64_t k0 = int64_t(tile) * kTargetTile + int64_t(threadIdx.x) * kTargetItems;
    if (int64_t(tile) * kTargetTile >= ns) return;  // uniform
    uint32_t on = 0, total;
#pragma unroll
    for (int q = 0; q < kTargetItems; ++q)
        if (k0 + q < ns && end[order[k0 + q]] == tick) on |= 1u << q;
    const uint32_t cnt = __popc(on);
    uint32_t at = block_excl_scan<kTargetThreads>(cnt, s_warp, total);
    if (threadIdx.x < 32) {
        const unsigned long long e = look_back(reinterpret_cast<unsigned long long *>(lb + 2), tile, total, info);
        if (threadIdx.x == 0) {
            s_prefix = uint32_t(e);
            if ((int64_t(tile) + 1) * kTargetTile >= ns) info->ntargets = uint32_t(e) + total;
        }
    }
    __syncthreads();
    at += s_prefix;
#pragma unroll
    for (int q = 0; q < kTargetItems; ++q)
        if (on >> q & 1u) targets[at++] = int32_t(k0) + q;
}

}  // namespace

cudaError_t select_targets(const Launch &L, TreeBufs &b, int64_t n, const int32_t *end, int32_t tick) {
    GBH_LAUNCH_AFTER(L, k_targets, unsigned(target_tiles(n)), kTargetThreads, b.info, b.order, end, tick, b.targets,
                     b.lb_state + b.lb_targets);
    return cudaSuccess;
}

}  // namespace gbh

namespace gbh {

// ---------------------------------------------------------------- block time steps
//
// Gravity has no block steps in the reference; these follow its gas block steps
// (internal/sim/blockstep.go:22-90): a global step T is split into 2^(levels-1) ticks, a body
// on rung r steps T / 2^r, its rung is the smallest r with T / 2^r <= dt_i (rungFor,
// blockstep.go:38-45) capped at levels - 1, with dt_i = eta sqrt(eps / |a_i|), and a step may
// start only at a multiple of its length (blockstep.go:84-86). Kick-drift-kick per body: an
// opening half kick when its step starts, all bodies drift together from event to event, and
// at the end of its step a body gets its new acceleration, the closing half kick, a new rung
// and the next opening kick. With one level this is exactly the global KDK of sim.go.

namespace {

__device__ __forceinline__ int rung_for(double dt, double T, int rmax) {
    int r = 0;
    double x = T;
    while (x > dt && r < rmax) {
        x *= 0.5;
        ++r;
    }
    return r;
}

__device__ __forceinline__ double body_dt(double ax, double ay, double az, double eta, double eps) {
    double a = sqrt(ax * ax + ay * ay + az * az);
    return a > 0 ? eta * sqrt(eps / a) : INFINITY;
}

// The earliest step end over all bodies, and the bodies that end there (the host sizes that event's
// walk by them): every thread's (tick, bodies) over its bodies, reduced by block, and by the last
// block to finish over the blocks' parts (a counter that wraps to 0 by itself). A tick of INT_MAX
// holds no bodies.
__device__ __forceinline__ unsigned long long next_join(unsigned long long a, unsigned long long b) {
    const uint32_t ta = uint32_t(a >> 32), tb = uint32_t(b >> 32);
    return ta < tb ? a : tb < ta ? b : a + uint32_t(b);
}
__device__ __forceinline__ void reduce_next(int32_t tick, uint32_t bodies, unsigned long long *part, DevInfo *info) {
    __shared__ unsigned long long s_w[kThreads / 32];
    __shared__ bool s_last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto block_join = [&](unsigned long long v) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = next_join(v, __shfl_xor_sync(0xffffffffu, v, o));
        __syncthreads();
        if (lane == 0) s_w[warp] = v;
        __syncthreads();
        v = s_w[0];
        for (int w = 1; w < kThreads / 32; ++w) v = next_join(v, s_w[w]);
        return v;
    };
    unsigned long long v = block_join(static_cast<unsigned long long>(uint32_t(tick)) << 32 | bodies);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = v;
        __threadfence();
        s_last = atomicInc(&info->next_done, gridDim.x - 1) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    v = static_cast<unsigned long long>(uint32_t(INT_MAX)) << 32;
    for (unsigned b = threadIdx.x; b < gridDim.x; b += kThreads) v = next_join(v, __ldcg(part + b));
    v = block_join(v);
    if (threadIdx.x == 0) {
        info->next_tick = int32_t(v >> 32);
        info->next_count = uint32_t(v);
    }
}
// Adds a body that ends at e to a thread's (tick, bodies).
__device__ __forceinline__ void add_end(int32_t e, int32_t &tick, uint32_t &bodies) {
    if (e < tick) {
        tick = e;
        bodies = 1;
    } else if (e == tick) {
        ++bodies;
    }
}

// Tick 0 of a global step: every body starts a step (rung from its acceleration) with the
// opening half kick.
__global__ __launch_bounds__(kThreads) void k_block_open(int64_t n, double T, int32_t ticks, int levels, double eta,
                                                         double eps, const double *__restrict__ ax,
                                                         const double *__restrict__ ay, const double *__restrict__ az,
                                                         double *vx, double *vy, double *vz, uint8_t *rung,
                                                         int32_t *end, unsigned long long *part, DevInfo *info) {
    pdl_begin();
    int32_t tick = INT_MAX;
    uint32_t bodies = 0;
    for (int64_t i = int64_t(blockIdx.x) * kThreads + threadIdx.x; i < n; i += int64_t(gridDim.x) * kThreads) {
        double a0 = ax[i], a1 = ay[i], a2 = az[i];
        int r = rung_for(body_dt(a0, a1, a2, eta, eps), T, levels - 1);
        rung[i] = uint8_t(r);
        int32_t e = ticks >> r;
        end[i] = e;
        double h = 0.5 * (T / double(1 << r));
        vx[i] += h * a0;
        vy[i] += h * a1;
        vz[i] += h * a2;
        add_end(e, tick, bodies);
    }
    reduce_next(tick, bodies, part, info);
}

// driftOne (sim.go:345-350) of every body from tick t to the next event's tick: x += dt u / gamma(u, c),
// gamma = 1 for c <= 0 (relativity.go:15-20).
__global__ __launch_bounds__(kThreads) void k_block_drift(int64_t n, int32_t t, double tick_len, double c, double *px,
                                                          double *py, double *pz, const double *__restrict__ vx,
                                                          const double *__restrict__ vy, const double *__restrict__ vz,
                                                          const DevInfo *info) {
    pdl_begin();
    int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double dt = double(info->next_tick - t) * tick_len;
    double ux = vx[i], uy = vy[i], uz = vz[i];
    double f = dt / (c <= 0 ? 1.0 : sqrt(1 + (ux * ux + uy * uy + uz * uz) / (c * c)));
    px[i] += f * ux;
    py[i] += f * uy;
    pz[i] += f * uz;
}

// Bodies whose step ends at tick: closing half kick with the new acceleration, then (before
// the end of the global step) a new rung aligned to tick and the opening half kick.
__global__ __launch_bounds__(kThreads) void k_block_close(int64_t n, int32_t tick, int32_t ticks, double T, int levels,
                                                          double eta, double eps, const double *__restrict__ ax,
                                                          const double *__restrict__ ay, const double *__restrict__ az,
                                                          double *vx, double *vy, double *vz, uint8_t *rung,
                                                          int32_t *end, unsigned long long *part, DevInfo *info) {
    pdl_begin();
    int32_t next = INT_MAX;
    uint32_t bodies = 0;
    for (int64_t i = int64_t(blockIdx.x) * kThreads + threadIdx.x; i < n; i += int64_t(gridDim.x) * kThreads) {
        int32_t e = end[i];
        if (e == tick) {
            double a0 = ax[i], a1 = ay[i], a2 = az[i];
            double h = 0.5 * (T / double(1 << rung[i]));
            double u = vx[i] + h * a0, v = vy[i] + h * a1, w = vz[i] + h * a2;
            if (tick < ticks) {
                int r = rung_for(body_dt(a0, a1, a2, eta, eps), T, levels - 1);
                while (tick % (ticks >> r) != 0) ++r;
                rung[i] = uint8_t(r);
                e = tick + (ticks >> r);
                end[i] = e;
                double h2 = 0.5 * (T / double(1 << r));
                u += h2 * a0;
                v += h2 * a1;
                w += h2 * a2;
            }
            vx[i] = u;
            vy[i] = v;
            vz[i] = w;
        }
        add_end(e, next, bodies);
    }
    reduce_next(next, bodies, part, info);
}

inline unsigned next_blocks(int64_t n) {
    const unsigned nb = blocks_for(n, kThreads);
    return nb < unsigned(kNextBlocks) ? nb : unsigned(kNextBlocks);
}

}  // namespace

cudaError_t block_open(const Launch &L, const TreeBufs &b, int64_t n, double T, int levels, double eta, double eps,
                       const double *ax, const double *ay, const double *az, double *vx, double *vy, double *vz,
                       uint8_t *rung, int32_t *end) {
    GBH_LAUNCH_AFTER(L, k_block_open, next_blocks(n), kThreads, n, T, 1 << (levels - 1), levels, eta, eps, ax, ay, az, vx,
                     vy, vz, rung, end, b.next_part, b.info);
    return cudaSuccess;
}

cudaError_t block_drift(const Launch &L, const TreeBufs &b, int64_t n, int32_t t, double tick_len, double c, double *px,
                        double *py, double *pz, const double *vx, const double *vy, const double *vz) {
    GBH_LAUNCH_AFTER(L, k_block_drift, blocks_for(n, kThreads), kThreads, n, t, tick_len, c, px, py, pz, vx, vy, vz,
                     b.info);
    return cudaSuccess;
}

cudaError_t block_close(const Launch &L, const TreeBufs &b, int64_t n, int32_t tick, double T, int levels, double eta,
                        double eps, const double *ax, const double *ay, const double *az, double *vx, double *vy,
                        double *vz, uint8_t *rung, int32_t *end) {
    GBH_LAUNCH_AFTER(L, k_block_close, next_blocks(n), kThreads, n, tick, 1 << (levels - 1), T, levels, eta, eps, ax, ay, az,
                     vx, vy, vz, rung, end, b.next_part, b.info);
    return cudaSuccess;
}

}  // namespace gbh
