// split.cu — the hole-aware step of internal/sim/split.go (stepSplit) without gas, instant gravity
// and no spins: star-star forces from the tree once per step (api.cu), every force involving an
// alive black hole summed here directly (O(N x holes), the pair model of pair.go: Paczynski-Wiita
// star-hole pairs for c > 0), and the stars near a hole plus the holes themselves advanced in
// power-of-two substeps, every drift by u / gamma (relativity.go). Built with -fmad=false: the pair terms, kicks and drifts
// round like the FP64 restatement (orc_split_kdk), so the FP64 walk's trajectories match it bit
// for bit. A hole's pull from the far stars is summed in 256-body chunks (sequential inside a
// chunk, chunks in index order), the fixed order the restatement uses.
#include <cuda_runtime.h>

#include <algorithm>

#include "gbh_internal.cuh"
#include "lookback.cuh"

namespace gbh {
namespace {

constexpr int kEw = 256;
constexpr int kHoleChunk = 256;

inline unsigned ew_blocks(int64_t n) { return unsigned(std::max<int64_t>(1, (n + kEw - 1) / kEw)); }

// pair.go:26-35 (PairForce): f such that the acceleration is f d; capped inside 1.5 rs.
__device__ __forceinline__ double pair_force(double m, double r2, double eps2, double rs) {
    double re2 = r2 + eps2;
    double re = sqrt(re2);
    if (rs == 0) return m / (re2 * re);
    double den = fmax(re - rs, rs / 2);
    return m / (den * den * re);
}

__device__ __forceinline__ double schwarzschild(double m, double c) { return c <= 0 ? 0 : 2 * m / (c * c); }

// PairRS (pair.go:14-23) of body i with hole h: the hole's radius unless i is a hole too.
__device__ __forceinline__ double hole_rs(int64_t i, int32_t h, const double *mass, const uint8_t *kind, double c) {
    return kind[i] == GBH_BLACK_HOLE ? 0.0 : schwarzschild(mass[h], c);
}

// dt / gamma (relativity.go:15-20, driftIdx / driftFar split.go:226-250).
__device__ __forceinline__ double drift_factor(double dt, double ux, double uy, double uz, double c) {
    return dt / (c <= 0 ? 1.0 : sqrt(1 + (ux * ux + uy * uy + uz * uz) / (c * c)));
}

// split.go:27-36 (holeTimescale): sqrt(r_eps / a) of body i in the field of hole h.
__device__ __forceinline__ double timescale(int64_t i, int64_t h, const double *px, const double *py,
                                            const double *pz, const double *mass, const uint8_t *kind, double eps2,
                                            double c) {
    double dx = px[i] - px[h], dy = py[i] - py[h], dz = pz[i] - pz[h];
    double r2 = dx * dx + dy * dy + dz * dz;
    double a = pair_force(mass[h], r2, eps2, hole_rs(i, int32_t(h), mass, kind, c)) * sqrt(r2);
    if (a == 0) return __longlong_as_double(0x7ff0000000000000LL);
    return sqrt(sqrt(r2 + eps2) / a);
}

// split.go:119-137 (holePull): the pull of every hole but i itself on body i, holes in order.
__device__ __forceinline__ void hole_pull(int64_t i, const int32_t *__restrict__ holes, int32_t nh,
                                          const double *px, const double *py, const double *pz,
                                          const double *mass, const uint8_t *kind, double eps2, double c, double &fx,
                                          double &fy, double &fz) {
    double x = px[i], y = py[i], z = pz[i];
    fx = fy = fz = 0;
    for (int32_t k = 0; k < nh; ++k) {
        int32_t h = holes[k];
        if (h == i) continue;
        double dx = px[h] - x, dy = py[h] - y, dz = pz[h] - z;
        double f = pair_force(mass[h], dx * dx + dy * dy + dz * dz, eps2, hole_rs(i, h, mass, kind, c));
        fx += f * dx;
        fy += f * dy;
        fz += f * dz;
    }
}

__device__ __forceinline__ double source_mass(int64_t i, const double *mass, const uint8_t *kind, int dm_off) {
    return dm_off && kind[i] == GBH_DARK_MATTER ? 0.0 : mass[i];  // Params.SourceMass, sim.go:93-98
}

// classify (split.go:39-85): near flags, the near stars' list in index order, and the minimum
// timescale over near stars and hole pairs (a positive double orders like its bits; their complement
// is kept, so that the scalars start at 0). Blocks take tiles of 256 bodies in counter order and rank
// their near stars by look-back. 20,002-body step of 4 substeps with the list scanned and written by
// four more launches 434 us, 420 so.
__global__ __launch_bounds__(kEw) void k_classify(int64_t n, const double *__restrict__ px,
                                                  const double *__restrict__ py, const double *__restrict__ pz,
                                                  const double *__restrict__ mass, const uint8_t *__restrict__ kind,
                                                  const int32_t *__restrict__ holes, int32_t nh, double eps2, double c,
                                                  double limit, uint8_t *near8, int32_t *near, SplitScalars *out,
                                                  unsigned long long *lb) {
    pdl_begin();
    __shared__ double smin[kEw / 32];
    __shared__ uint32_t s_warp[kEw / 32 + 1], s_tile, s_prefix;
    if (threadIdx.x == 0) s_tile = atomicAdd(reinterpret_cast<uint32_t *>(lb), 1u);
    __syncthreads();
    const uint32_t tile = s_tile;
    const int64_t i = int64_t(tile) * kEw + threadIdx.x;
    double local = __longlong_as_double(0x7ff0000000000000LL);
    bool nr = false;
    if (i < n) {
        if (kind[i] != GBH_BLACK_HOLE)
            for (int32_t k = 0; k < nh; ++k) {
                double tau = timescale(i, holes[k], px, py, pz, mass, kind, eps2, c);
                if (tau < limit) {
                    nr = true;
                    local = fmin(local, tau);
                }
            }
        near8[i] = nr;
    }
    for (int o = 16; o > 0; o >>= 1) local = fmin(local, __shfl_xor_sync(0xffffffffu, local, o));
    if ((threadIdx.x & 31) == 0) smin[threadIdx.x >> 5] = local;
    uint32_t total;
    const uint32_t at = block_excl_scan<kEw>(nr, s_warp, total);  // its barriers order smin too
    if (threadIdx.x < 32) {
        const unsigned long long before = look_back(lb + 1, tile, total, &out->info);
        if (threadIdx.x == 0) {
            s_prefix = uint32_t(before);
            if ((int64_t(tile) + 1) * kEw >= n) out->nnear = before + total;
        }
    }
    __syncthreads();
    if (nr) near[s_prefix + at] = int32_t(i);
    if (threadIdx.x == 0) {
        for (int w = 1; w < kEw / 32; ++w) local = fmin(local, smin[w]);
        if (tile == 0)  // hole pairs: each with the mass of the later one (split.go:64-70)
            for (int32_t a = 0; a < nh; ++a)
                for (int32_t b = a + 1; b < nh; ++b) {
                    double tau = timescale(holes[a], holes[b], px, py, pz, mass, kind, eps2, c);
                    if (tau < limit) local = fmin(local, tau);
                }
        atomicMax(&out->tau_inv, ~static_cast<unsigned long long>(__double_as_longlong(local)));
    }
}

// outerHoleForces (split.go:83-116) of one 256-body chunk. Each body: far stars feel every hole;
// near stars and holes get 0 here (the holes' sums are added by k_kick_outer). Each hole: the
// chunk's far stars pull on it, summed in index order.
//
// A hole's sum is a serial chain of FP64 adds (72 cycles each), but its terms are independent:
// every thread forms its own body's terms for up to kHoleBatch holes in shared memory (+0 for a
// skipped body: the sums start at +0 and never become -0, so it changes nothing), and one lane per
// hole and axis adds them in order. 20,000 bodies and 2 holes: 290 us with one thread a hole
// running through the chunk's square roots and divisions, 24 us so (with the far bodies' own pulls).
constexpr int kHoleBatch = 7;  // 43 KB of terms
constexpr int kTermStride = kHoleChunk + 1;
__global__ __launch_bounds__(kHoleChunk) void k_far_part(int64_t n, const double *__restrict__ px,
                                                         const double *__restrict__ py, const double *__restrict__ pz,
                                                         const double *__restrict__ mass,
                                                         const uint8_t *__restrict__ kind,
                                                         const uint8_t *__restrict__ near8, int dm_off,
                                                         const int32_t *__restrict__ holes, int32_t nh, double eps2,
                                                         double c, double *fx, double *fy, double *fz, double *part) {
    pdl_begin();
    __shared__ double s_term[3 * kHoleBatch][kTermStride];
    const int64_t i = int64_t(blockIdx.x) * kHoleChunk + threadIdx.x;
    const bool far = i < n && kind[i] != GBH_BLACK_HOLE && !near8[i];
    double x = 0, y = 0, z = 0, sm = 0;
    if (far) {
        hole_pull(i, holes, nh, px, py, pz, mass, kind, eps2, c, x, y, z);
        sm = source_mass(i, mass, kind, dm_off);
    }
    if (i < n) {
        fx[i] = x;
        fy[i] = y;
        fz[i] = z;
    }
    if (far) {
        x = px[i];
        y = py[i];
        z = pz[i];
    }
    for (int32_t k0 = 0; k0 < nh; k0 += kHoleBatch) {
        const int cnt = nh - k0 < kHoleBatch ? nh - k0 : kHoleBatch;
        for (int k = 0; k < cnt; ++k) {
            double tx = 0, ty = 0, tz = 0;
            if (far) {
                const int32_t h = holes[k0 + k];
                const double dx = x - px[h], dy = y - py[h], dz = z - pz[h];
                const double f = pair_force(sm, dx * dx + dy * dy + dz * dz, eps2, schwarzschild(mass[h], c));
                tx = f * dx;
                ty = f * dy;
                tz = f * dz;
            }
            s_term[3 * k][threadIdx.x] = tx;
            s_term[3 * k + 1][threadIdx.x] = ty;
            s_term[3 * k + 2][threadIdx.x] = tz;
        }
        __syncthreads();
        if (threadIdx.x < 3 * cnt) {
            double a = 0;
#pragma unroll 16
            for (int q = 0; q < kHoleChunk; ++q) a += s_term[threadIdx.x][q];
            part[(int64_t(blockIdx.x) * nh + k0) * 3 + threadIdx.x] = a;
        }
        __syncthreads();
    }
}

// kickOuter (split.go:206-213): every body, v += h (a + far), and with `drift` the drift by dt of
// the far bodies (driftFar, split.go:236-250, no gas: neither a hole nor near) right after their
// kick: the substeps between the two read and move only near stars and holes. The last nh blocks
// take a hole each: its chunk partials added in chunk order to 0, then its kick.
__global__ __launch_bounds__(kEw) void k_kick_outer(int64_t n, double h, bool drift, double dt, double c,
                                                    const uint8_t *__restrict__ kind,
                                                    const uint8_t *__restrict__ near8, double *px, double *py,
                                                    double *pz, double *vx, double *vy, double *vz,
                                                    const double *__restrict__ ax, const double *__restrict__ ay,
                                                    const double *__restrict__ az, const double *__restrict__ fx,
                                                    const double *__restrict__ fy, const double *__restrict__ fz,
                                                    const int32_t *__restrict__ holes, int32_t nh, int64_t nchunks,
                                                    const double *__restrict__ part) {
    pdl_begin();
    const int64_t nb = int64_t(gridDim.x) - nh;
    if (int64_t(blockIdx.x) >= nb) {
        __shared__ double s[3][kEw + 1];
        const int32_t k = int32_t(blockIdx.x - nb);
        double a = 0;
        for (int64_t c0 = 0; c0 < nchunks; c0 += kEw) {
            const int64_t q = c0 + threadIdx.x;
            for (int e = 0; e < 3; ++e) s[e][threadIdx.x] = q < nchunks ? part[(q * nh + k) * 3 + e] : 0.0;
            __syncthreads();
            const int cnt = nchunks - c0 < kEw ? int(nchunks - c0) : kEw;
            if (threadIdx.x < 3) {
#pragma unroll 8
                for (int t = 0; t < cnt; ++t) a += s[threadIdx.x][t];
            }
            __syncthreads();
        }
        if (threadIdx.x < 3) {
            const int32_t i = holes[k];
            double *v = threadIdx.x == 0 ? vx : threadIdx.x == 1 ? vy : vz;
            const double *ac = threadIdx.x == 0 ? ax : threadIdx.x == 1 ? ay : az;
            v[i] = v[i] + h * (ac[i] + a);
        }
        return;
    }
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const bool hole = kind[i] == GBH_BLACK_HOLE;
    if (hole)  // an alive hole is kicked by its own block; a dead one is not in the list (its far force is 0)
        for (int32_t k = 0; k < nh; ++k)
            if (holes[k] == i) return;
    const double u = vx[i] + h * (ax[i] + fx[i]), v = vy[i] + h * (ay[i] + fy[i]), w = vz[i] + h * (az[i] + fz[i]);
    vx[i] = u;
    vy[i] = v;
    vz[i] = w;
    if (drift && !hole && !near8[i]) {
        const double f = drift_factor(dt, u, v, w, c);
        px[i] = px[i] + f * u;
        py[i] = py[i] + f * v;
        pz[i] = pz[i] + f * w;
    }
}

// fastForces (split.go:142-158) and, with `kick`, the closing half kick h of a substep (kickFast,
// split.go:215-224). Near stars: the pull of every hole, a thread each. Holes, a block each: the
// pulls of the other holes, then of the near stars in index order; the compute threads form a
// tile's terms and three lanes add the previous tile's in order, as k_far_part does. 400 near
// stars: 500 us with a thread a hole, 21 us so.
constexpr int kFastThreads = kEw + 32;  // the last warp adds
__global__ __launch_bounds__(kFastThreads) void k_fast(int32_t nnear, const int32_t *__restrict__ near,
                                                       const double *__restrict__ px, const double *__restrict__ py,
                                                       const double *__restrict__ pz, const double *__restrict__ mass,
                                                       const uint8_t *__restrict__ kind, int dm_off,
                                                       const int32_t *__restrict__ holes, int32_t nh, double eps2,
                                                       double c, bool kick, double h, double *vx, double *vy,
                                                       double *vz, double *fx, double *fy, double *fz) {
    pdl_begin();
    if (int32_t(blockIdx.x) >= nh) {
        const int32_t q = (int32_t(blockIdx.x) - nh) * kFastThreads + threadIdx.x;
        if (q >= nnear) return;
        const int32_t i = near[q];
        double x, y, z;
        hole_pull(i, holes, nh, px, py, pz, mass, kind, eps2, c, x, y, z);
        fx[i] = x;
        fy[i] = y;
        fz[i] = z;
        if (kick) {
            vx[i] = vx[i] + h * x;
            vy[i] = vy[i] + h * y;
            vz[i] = vz[i] + h * z;
        }
        return;
    }
    __shared__ double s_term[2][3][kEw + 1];
    const int tid = threadIdx.x;
    const int32_t hole = holes[blockIdx.x];
    const double x = px[hole], y = py[hole], z = pz[hole];
    const double rs = schwarzschild(mass[hole], c);
    const int32_t total = nh + nnear;
    const int32_t ntiles = (total + kEw - 1) / kEw;
    double sum = 0;
    for (int32_t t = 0; t <= ntiles; ++t) {
        if (tid < kEw && t < ntiles) {
            const int32_t q = t * kEw + tid;
            double tx = 0, ty = 0, tz = 0;
            if (q < total) {
                const int32_t i = q < nh ? holes[q] : near[q - nh];
                if (i != hole) {
                    const double dx = px[i] - x, dy = py[i] - y, dz = pz[i] - z;
                    // hole pairs are Newtonian (PairRS) and always pull
                    const double m = q < nh ? mass[i] : source_mass(i, mass, kind, dm_off);
                    const double f = pair_force(m, dx * dx + dy * dy + dz * dz, eps2, q < nh ? 0.0 : rs);
                    tx = f * dx;
                    ty = f * dy;
                    tz = f * dz;
                }
            }
            s_term[t & 1][0][tid] = tx;
            s_term[t & 1][1][tid] = ty;
            s_term[t & 1][2][tid] = tz;
        } else if (t > 0 && tid >= kEw && tid < kEw + 3) {
            const int cnt = total - (t - 1) * kEw < kEw ? total - (t - 1) * kEw : kEw;
#pragma unroll 8
            for (int k = 0; k < cnt; ++k) sum += s_term[(t - 1) & 1][tid - kEw][k];
        }
        __syncthreads();
    }
    if (tid >= kEw && tid < kEw + 3) {
        double *f = tid == kEw ? fx : tid == kEw + 1 ? fy : fz;
        f[hole] = sum;
        if (kick) {
            double *v = tid == kEw ? vx : tid == kEw + 1 ? vy : vz;
            v[hole] = v[hole] + h * sum;
        }
    }
}

// The opening half kick of a substep (kickFast, split.go:215-224) and its drift (driftIdx,
// split.go:226-234) over the near stars, then the holes: entry q < nnear is near[q], the rest are
// the holes.
__global__ void k_fast_open(int32_t nnear, const int32_t *__restrict__ near, const int32_t *__restrict__ holes,
                            int32_t nh, double h, double dt, double c, double *px, double *py, double *pz, double *vx,
                            double *vy, double *vz, const double *__restrict__ fx, const double *__restrict__ fy,
                            const double *__restrict__ fz) {
    pdl_begin();
    int32_t q = int32_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (q >= nnear + nh) return;
    int32_t i = q < nnear ? near[q] : holes[q - nnear];
    const double u = vx[i] + h * fx[i], v = vy[i] + h * fy[i], w = vz[i] + h * fz[i];
    vx[i] = u;
    vy[i] = v;
    vz[i] = w;
    const double f = drift_factor(dt, u, v, w, c);
    px[i] = px[i] + f * u;
    py[i] = py[i] + f * v;
    pz[i] = pz[i] + f * w;
}

}  // namespace

void split_free(SplitBufs &s) {
    void *ptrs[] = {s.holes, s.near8, s.near, s.far, s.fast, s.part, s.scalars};
    for (void *p : ptrs)
        if (p) cudaFree(p);
    if (s.host) cudaFreeHost(s.host);
    s = SplitBufs{};
}

cudaError_t split_reserve(SplitBufs &s, int64_t n, const std::vector<int32_t> &holes) {
    cudaError_t e = cudaSuccess;
    const int32_t nh = int32_t(holes.size());
    if (n > s.cap_n) {
        void *ptrs[] = {s.near8, s.near, s.far, s.fast, s.scalars};
        for (void *p : ptrs)
            if (p) cudaFree(p);
        s.near8 = nullptr;
        s.near = nullptr;
        s.scalars = nullptr;
        s.far = s.fast = nullptr;
        s.cap_n = 0;
        int64_t cap = n + n / 4;
        s.scalar_bytes = sizeof(SplitScalars) + sizeof(unsigned long long) * (1 + size_t(ew_blocks(cap)));
        if (e == cudaSuccess) e = dev_alloc(&s.near8, size_t(cap));
        if (e == cudaSuccess) e = dev_alloc(&s.near, sizeof(int32_t) * size_t(cap));
        if (e == cudaSuccess) e = dev_alloc(&s.scalars, s.scalar_bytes);
        if (e == cudaSuccess) e = dev_alloc(&s.far, sizeof(double) * 3 * size_t(cap));
        if (e == cudaSuccess) e = dev_alloc(&s.fast, sizeof(double) * 3 * size_t(cap));
        if (e != cudaSuccess) return e;
        s.cap_n = cap;
    }
    int64_t need_part = ((n + kHoleChunk - 1) / kHoleChunk) * std::max(nh, 1) * 3;
    if (need_part > s.cap_part) {
        if (s.part) cudaFree(s.part);
        s.part = nullptr;
        s.cap_part = 0;
        if ((e = dev_alloc(&s.part, sizeof(double) * size_t(need_part + need_part / 4)))) return e;
        s.cap_part = need_part + need_part / 4;
    }
    if (nh > s.cap_holes) {
        if (s.holes) cudaFree(s.holes);
        s.holes = nullptr;
        s.cap_holes = 0;
        if ((e = dev_alloc(&s.holes, sizeof(int32_t) * size_t(nh)))) return e;
        s.cap_holes = nh;
    }
    if (!s.host && (e = cudaMallocHost(&s.host, sizeof(SplitScalars)))) return e;
    s.nholes = nh;
    return cudaSuccess;
}

cudaError_t split_classify(const Launch &L, SplitBufs &s, int64_t n, const double *px, const double *py,
                           const double *pz, const double *mass, const uint8_t *kind, double eps2, double c,
                           double limit) {
    cudaError_t e = cudaMemsetAsync(s.scalars, 0, s.scalar_bytes, L.stream);
    if (e != cudaSuccess) return e;
    GBH_LAUNCH_AFTER(L, k_classify, ew_blocks(n), kEw, n, px, py, pz, mass, kind, s.holes, s.nholes, eps2, c, limit,
                     s.near8, s.near, s.scalars, reinterpret_cast<unsigned long long *>(s.scalars + 1));
    return cudaMemcpyAsync(s.host, s.scalars, sizeof(SplitScalars), cudaMemcpyDeviceToHost, L.stream);
}

cudaError_t split_outer(const Launch &L, SplitBufs &s, int64_t n, const double *px, const double *py,
                        const double *pz, const double *mass, const uint8_t *kind, int dm_off, double eps2, double c) {
    GBH_LAUNCH_AFTER(L, k_far_part, unsigned((n + kHoleChunk - 1) / kHoleChunk), kHoleChunk, n, px, py, pz, mass, kind,
                     s.near8, dm_off, s.holes, s.nholes, eps2, c, s.far, s.far + n, s.far + 2 * n, s.part);
    return cudaSuccess;
}

cudaError_t split_kick_outer(const Launch &L, SplitBufs &s, int64_t n, double h, bool drift, double dt, double c,
                             const uint8_t *kind, double *px, double *py, double *pz, double *vx, double *vy,
                             double *vz, const double *ax, const double *ay, const double *az) {
    GBH_LAUNCH_AFTER(L, k_kick_outer, ew_blocks(n) + unsigned(s.nholes), kEw, n, h, drift, dt, c, kind, s.near8, px,
                     py, pz, vx, vy, vz, ax, ay, az, s.far, s.far + n, s.far + 2 * n, s.holes, s.nholes, (n +
                     kHoleChunk - 1) / kHoleChunk, s.part);
    return cudaSuccess;
}

cudaError_t split_fast(const Launch &L, SplitBufs &s, int64_t n, int32_t nnear, bool kick, double h, const double *px,
                       const double *py, const double *pz, double *vx, double *vy, double *vz, const double *mass,
                       const uint8_t *kind, int dm_off, double eps2, double c) {
    const unsigned nb = unsigned(s.nholes) + unsigned((nnear + kFastThreads - 1) / kFastThreads);
    GBH_LAUNCH_AFTER(L, k_fast, nb, kFastThreads, nnear, s.near, px, py, pz, mass, kind, dm_off, s.holes, s.nholes,
                     eps2, c, kick, h, vx, vy, vz, s.fast, s.fast + n, s.fast + 2 * n);
    return cudaSuccess;
}

cudaError_t split_fast_open(const Launch &L, SplitBufs &s, int64_t n, int32_t nnear, double h, double dt, double c,
                            double *px, double *py, double *pz, double *vx, double *vy, double *vz) {
    GBH_LAUNCH_AFTER(L, k_fast_open, ew_blocks(int64_t(nnear) + s.nholes), kEw, nnear, s.near, s.holes, s.nholes, h,
                     dt, c, px, py, pz, vx, vy, vz, s.fast, s.fast + n, s.fast + 2 * n);
    return cudaSuccess;
}

}  // namespace gbh
