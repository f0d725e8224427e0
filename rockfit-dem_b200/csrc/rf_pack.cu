// Seeded polydisperse specimen generator: random positions in a cylindrical container,
// overlaps removed by FIRE with a repulsive (frictionless, undamped) Hertz contact, radii
// grown in stages from a loose start to their targets. FP64 throughout (a one-time
// generator, not the hot path). Neighbour search: a cell grid rebuilt every iteration. A
// small specimen's iteration is a chain of launches and memory latencies, so it is as few
// kernels as the grid's dependencies allow, captured in batches in a CUDA graph: scan of the
// cell counts, scatter, per-cell order with the positions gathered into it, forces with the
// FIRE decision by the last block, and the FIRE update with the next grid's cell counts.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>
#include "rf_common.cuh"

namespace rf {
namespace pack {

struct Scal {
    double dt, alpha, fdotv, ff, vv, maxov;
    double scale;          // current radius scale g
    unsigned long long npos, iters;
    uint32_t counter, arrived;
};

struct Par {
    uint32_t N, cells, nx, ny, nz;
    double ox, oy, oz, inv_h;       // grid origin and 1 / cell edge
    double Rc, Hh;                  // container radius and half height
    double dtmax, dtmin, finc, fdec, alpha0, falpha;
    uint32_t ndelay;
};

struct Dev {
    double4* x;       // x, y, z, target radius
    double4* v;       // velocity (w unused)
    double4* f;       // force (w unused)
    double4* xs;      // x in cell order
    uint32_t *key, *count, *start, *sorted, *bsum;
    double4* part;    // per-block (F.v, |F|^2, |v|^2, max overlap)
    Scal* s;
};

__device__ __forceinline__ uint32_t cell_of(const double4 p, const Par& c) {
    long ix = (long)floor((p.x - c.ox) * c.inv_h), iy = (long)floor((p.y - c.oy) * c.inv_h),
         iz = (long)floor((p.z - c.oz) * c.inv_h);
    ix = ix < 0 ? 0 : (ix >= (long)c.nx ? c.nx - 1 : ix);
    iy = iy < 0 ? 0 : (iy >= (long)c.ny ? c.ny - 1 : iy);
    iz = iz < 0 ? 0 : (iz >= (long)c.nz ? c.nz - 1 : iz);
    return (uint32_t)(ix + c.nx * (iy + c.ny * iz));
}

__global__ void k_bin(Dev d, Par c) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < c.N; i += gridDim.x * blockDim.x) {
        const uint32_t k = cell_of(d.x[i], c);
        d.key[i] = k;
        atomicAdd(&d.count[k], 1u);
    }
}
// Exclusive scan of the cell counts into cell starts (start[cells] = N), SCAN_CHUNK cells per
// block. Up to SCAN_SELF chunks each block adds up the counts before its chunk itself, one
// kernel instead of three; beyond that the chunk sums and their scan are kernels of their own.
constexpr uint32_t SCAN_CHUNK = 4096;
constexpr uint32_t SCAN_SELF = 32;

__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t* wsum, uint32_t* total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t incl = v;
    for (int o = 1; o < 32; o <<= 1) { const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += y; }
    if (lane == 31) wsum[w] = incl;
    __syncthreads();
    if (w == 0) {
        const uint32_t t = lane < (int)(blockDim.x >> 5) ? wsum[lane] : 0;
        uint32_t ti = t;
        for (int o = 1; o < 32; o <<= 1) { const uint32_t y = __shfl_up_sync(0xffffffffu, ti, o); if (lane >= o) ti += y; }
        wsum[lane] = ti - t;
        if (lane == 31) *total = ti;
    }
    __syncthreads();
    const uint32_t r = wsum[w] + incl - v;
    __syncthreads();
    return r;
}

__global__ void k_scan_sums(Dev d, Par c) {
    __shared__ uint32_t sh[32];
    const size_t base = (size_t)blockIdx.x * SCAN_CHUNK;
    uint32_t s = 0;
    for (uint32_t t = threadIdx.x; t < SCAN_CHUNK; t += blockDim.x)
        if (base + t < c.cells) s += d.count[base + t];
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        uint32_t v = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : 0;
        for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (threadIdx.x == 0) d.bsum[blockIdx.x] = v;
    }
}

// one block: exclusive scan of the nb chunk sums, in place
__global__ void k_scan_chunks(Dev d, uint32_t nb) {
    __shared__ uint32_t wsum[32];
    __shared__ uint32_t total;
    uint32_t carry = 0;
    for (uint32_t base = 0; base < nb; base += blockDim.x) {
        const uint32_t q = base + threadIdx.x;
        const uint32_t v = q < nb ? d.bsum[q] : 0;
        const uint32_t ex = block_excl_scan(v, wsum, &total);
        if (q < nb) d.bsum[q] = carry + ex;
        carry += total;
        __syncthreads();
    }
}

__global__ void k_scan_apply(Dev d, Par c, int self) {
    __shared__ uint32_t wsum[32];
    __shared__ uint32_t total;
    const size_t base = (size_t)blockIdx.x * SCAN_CHUNK;
    uint32_t carry = 0;
    if (self) {
        uint32_t v = 0;
        const uint4* c4 = reinterpret_cast<const uint4*>(d.count);
#pragma unroll 4
        for (size_t q = threadIdx.x; q < base / 4; q += blockDim.x) { const uint4 u = c4[q]; v += (u.x + u.y) + (u.z + u.w); }
        block_excl_scan(v, wsum, &total);
        carry = total;
        __syncthreads();
    } else {
        carry = d.bsum[blockIdx.x];
    }
    const size_t q = base + 4 * threadIdx.x;             // (SCAN_CHUNK: four cells a thread)
    uint32_t v[4], sum = 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) { v[u] = q + u < c.cells ? d.count[q + u] : 0u; sum += v[u]; }
    uint32_t run = carry + block_excl_scan(sum, wsum, &total);
#pragma unroll
    for (int u = 0; u < 4; ++u) { if (q + u < c.cells) d.start[q + u] = run; run += v[u]; }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) d.start[c.cells] = carry + total;
}
// The counts run back to zero as the cells fill: the update counts the next grid into them.
__global__ void k_scatter(Dev d, Par c) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < c.N; i += gridDim.x * blockDim.x) {
        const uint32_t k = d.key[i];
        d.sorted[d.start[k] + atomicSub(&d.count[k], 1u) - 1u] = i;
    }
}

// The positions in cell order, a cell's occupants in id order (the scatter's atomics leave them in
// arrival order), so the force sums below, and with them the whole packing, are deterministic,
// and the forces read the cells' runs straight through. A thread a particle finds its place among
// its cell's occupants (a thread a cell sorted them one load after another: 11 us a launch at 20k
// particles, cold, against 4.4).
__global__ void k_cellsort(Dev d, Par c) {
    for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < c.N; q += gridDim.x * blockDim.x) {
        const uint32_t i = d.sorted[q], k = d.key[i];
        const double4 x = d.x[i];
        const uint32_t s0 = d.start[k], s1 = d.start[k + 1];
        uint32_t at = s0;
#pragma unroll 4
        for (uint32_t u = s0; u < s1; ++u) at += d.sorted[u] < i ? 1u : 0u;
        d.xs[at] = x;
    }
}

// Forces: repulsive Hertz between overlapping spheres and against the container wall,
// f = 4/3 sqrt(R*) delta^1.5 (unit modulus, unit masses). Partials of F.v, |F|^2,
// |v|^2 and the largest overlap (relative to the smaller radius); the last block to finish
// makes the FIRE decision.
// The candidates of a particle are the occupants of nine runs of cells (three x-neighbouring cells
// are one run of the cell order). Eight lanes a particle test them and list the overlapping ones in
// run order; the warp's listed pairs are then evaluated a lane a pair (about one tested pair in six
// overlaps, and one evaluation is some 300 instructions of FP64 roots and quotients), and the
// particle's first lane adds its pairs' forces in list order, the order of a plain loop. A thread
// a particle ran a chain of some 40 candidates, on 79 CTAs for 20k particles: 43 us a launch
// (cold), 25 us so; the packing of 3k particles 185 -> 80 ms, of 20k 178 -> 105 ms. Two and four
// lanes were slower at every size (20k: 125 ms); one lane was 7 % faster at 1M only.
#define PACK_LANES 8
#define PACK_HITS 32                         // listed pairs of a particle before they are evaluated
__device__ __forceinline__ void fire_decide(Dev d, Par c, int nblocks);
__global__ void __launch_bounds__(256) k_force(Dev d, Par c) {
    constexpr uint32_t LANES = PACK_LANES, G = 32 / LANES, CAP = PACK_HITS;     // G: particles of a warp
    __shared__ uint32_t s_hit[8][G][CAP], s_run[8][G][9], s_off[8][G][9];
    __shared__ uint16_t s_pair[8][G * CAP];
    __shared__ double s_res[8][3][32];
    const uint32_t FULL = 0xffffffffu;
    const uint32_t wp = threadIdx.x >> 5, lane = threadIdx.x & 31u, sub = lane % LANES, grp = lane / LANES;
    const uint32_t lower = (1u << sub) - 1u;
    const double g = d.s->scale;
    double fv = 0, ff = 0, vv = 0, mo = 0;
    for (uint32_t i0 = (blockIdx.x * 8u + wp) * G; i0 < c.N; i0 += gridDim.x * 8u * G) {
        const uint32_t i = i0 + grp;
        const bool in = i < c.N;
        double4 xi = make_double4(0, 0, 0, 0);
        double fx = 0, fy = 0, fz = 0;
        if (in) xi = d.x[i];
        const double ri = g * xi.w;
        const uint32_t key = in ? d.key[i] : 0u;
        const int ix = key % c.nx, iy = (key / c.nx) % c.ny, iz = key / (c.nx * c.ny);
        const uint32_t xa = ix > 0 ? ix - 1 : 0, xb = ix + 1 < (int)c.nx ? ix + 1 : ix;
        auto run_of = [&](int r, uint32_t& s0) -> uint32_t {         // occupants of run r
            const int z = iz + r / 3 - 1, y = iy + r % 3 - 1;
            s0 = 0;
            if (!in || z < 0 || z >= (int)c.nz || y < 0 || y >= (int)c.ny) return 0u;
            const uint32_t line = c.nx * (y + c.ny * z);
            s0 = d.start[line + xa];
            return d.start[line + xb + 1] - s0;
        };
        auto pair = [&](double rx, double ry, double rz, double ra, double rb) -> double3 {
            const double r2 = rx * rx + ry * ry + rz * rz, sr = ra + rb;
            const double r = sqrt(r2), dl = sr - r;
            const double Rs = ra * rb / sr;
            const double fn = (4.0 / 3.0) * sqrt(Rs) * dl * sqrt(dl);
            mo = fmax(mo, dl / fmin(ra, rb));
            return make_double3(fn * rx / r, fn * ry / r, fn * rz / r);
        };
        uint32_t cnt = 0;                                // the particle's listed pairs
        // evaluates the warp's listed pairs and adds them up
        auto flush = [&]() {
            uint32_t all = sub == 0 ? cnt : 0u;
#pragma unroll
            for (uint32_t o = LANES; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(FULL, all, o);
                if (lane >= o) all += y;
            }
            const uint32_t first = __shfl_sync(FULL, all, grp * LANES) - cnt;
            all = __shfl_sync(FULL, all, 32 - LANES);
            for (uint32_t t = sub; t < cnt; t += LANES) s_pair[wp][first + t] = (uint16_t)(grp | (t << 5));
            __syncwarp();
            uint32_t added = 0;
            for (uint32_t b = 0; b < all; b += 32u) {
                const uint32_t x = b + lane, e = x < all ? s_pair[wp][x] : 0u, u = e & 31u;
                const double px = __shfl_sync(FULL, xi.x, u * LANES), py = __shfl_sync(FULL, xi.y, u * LANES),
                             pz = __shfl_sync(FULL, xi.z, u * LANES), pr = __shfl_sync(FULL, ri, u * LANES);
                if (x < all) {
                    const double4 xj = d.xs[s_hit[wp][u][e >> 5]];
                    const double3 t = pair(xj.x - px, xj.y - py, xj.z - pz, pr, g * xj.w);
                    s_res[wp][0][lane] = t.x; s_res[wp][1][lane] = t.y; s_res[wp][2][lane] = t.z;
                }
                __syncwarp();
                if (sub == 0)
                    for (; added < cnt && first + added < b + 32u; ++added) {
                        const uint32_t k = first + added - b;
                        fx -= s_res[wp][0][k]; fy -= s_res[wp][1][k]; fz -= s_res[wp][2][k];
                    }
                __syncwarp();
            }
            cnt = 0;
        };
        auto overlaps = [&](uint32_t q) -> bool {
            const double4 xj = d.xs[q];
            const double rx = xj.x - xi.x, ry = xj.y - xi.y, rz = xj.z - xi.z;
            const double rj = g * xj.w;
            const double r2 = rx * rx + ry * ry + rz * rz, sr = ri + rj;
            return !(r2 >= sr * sr || r2 <= 0);          // (the particle itself: r2 = 0)
        };
        uint32_t total = 0;
#pragma unroll
        for (uint32_t t = 0; t < (9 + LANES - 1) / LANES; ++t) {      // runs sub, sub + LANES, ...
            const int r = (int)(sub + LANES * t);
            uint32_t s0 = 0;
            const uint32_t n = r < 9 ? run_of(r, s0) : 0u;
            uint32_t at = n;
#pragma unroll
            for (uint32_t o = 1; o < LANES; o <<= 1) {
                const uint32_t v = __shfl_up_sync(FULL, at, o, LANES);
                if (sub >= o) at += v;
            }
            if (r < 9) { s_run[wp][grp][r] = s0; s_off[wp][grp][r] = total + at - n; }   // candidates before run r
            total += __shfl_sync(FULL, at, LANES - 1, LANES);
        }
        __syncwarp();
        const uint32_t most = __reduce_max_sync(FULL, total);
        for (uint32_t base = 0; base < most; base += LANES) {
            const uint32_t f = base + sub;
            bool hit = false;
            uint32_t q = 0;
            if (f < total) {
                uint32_t r = 0;
#pragma unroll
                for (uint32_t t = 1; t < 9; ++t) r = f >= s_off[wp][grp][t] ? t : r;
                q = s_run[wp][grp][r] + (f - s_off[wp][grp][r]);
                hit = overlaps(q);
            }
            const uint32_t bal = (__ballot_sync(FULL, hit) >> (grp * LANES)) & ((1u << LANES) - 1u);
            if (hit) s_hit[wp][grp][cnt + __popc(bal & lower)] = q;
            cnt += __popc(bal);
            if (__any_sync(FULL, cnt > CAP - LANES) || base + LANES >= most) { __syncwarp(); flush(); }
        }
        __syncwarp();
        if (!in || sub != 0) continue;
        // container wall (cylinder side and end caps)
        const double rho = sqrt(xi.x * xi.x + xi.y * xi.y);
        const double dw = rho + ri - c.Rc;
        if (dw > 0 && rho > 0) {
            const double fn = (4.0 / 3.0) * sqrt(ri) * dw * sqrt(dw);
            fx -= fn * xi.x / rho; fy -= fn * xi.y / rho;
            mo = fmax(mo, dw / ri);
        }
        const double dtop = xi.z + ri - c.Hh, dbot = -xi.z + ri - c.Hh;
        if (dtop > 0) { fz -= (4.0 / 3.0) * sqrt(ri) * dtop * sqrt(dtop); mo = fmax(mo, dtop / ri); }
        if (dbot > 0) { fz += (4.0 / 3.0) * sqrt(ri) * dbot * sqrt(dbot); mo = fmax(mo, dbot / ri); }
        const double4 vi = d.v[i];
        d.f[i] = make_double4(fx, fy, fz, 0.0);
        fv += fx * vi.x + fy * vi.y + fz * vi.z;
        ff += fx * fx + fy * fy + fz * fz;
        vv += vi.x * vi.x + vi.y * vi.y + vi.z * vi.z;
    }
    __shared__ double sh[4][32];
    __shared__ bool s_last;
    for (int o = 16; o; o >>= 1) {
        fv += __shfl_xor_sync(0xffffffffu, fv, o);
        ff += __shfl_xor_sync(0xffffffffu, ff, o);
        vv += __shfl_xor_sync(0xffffffffu, vv, o);
        mo = fmax(mo, __shfl_xor_sync(0xffffffffu, mo, o));
    }
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) { sh[0][w] = fv; sh[1][w] = ff; sh[2][w] = vv; sh[3][w] = mo; }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0, b = 0, e = 0, m = 0;
        for (int q = 0; q < (int)(blockDim.x >> 5); ++q) { a += sh[0][q]; b += sh[1][q]; e += sh[2][q]; m = fmax(m, sh[3][q]); }
        d.part[blockIdx.x] = make_double4(a, b, e, m);
        __threadfence();
        s_last = atomicAdd(&d.s->arrived, 1u) == gridDim.x - 1u;
    }
    __syncthreads();
    if (s_last) { __threadfence(); fire_decide(d, c, (int)gridDim.x); }
}

// FIRE step decision (256 threads): sums of the block partials in a fixed order -- 1024
// strided shares, four a thread, then a fixed tree over their 32 groups -- then power, time
// step and mixing factor on thread 0.
__device__ __forceinline__ void fire_decide(Dev d, Par c, int nblocks) {
    __shared__ double sh[4][32];
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        double fv = 0, ff = 0, vv = 0, mo = 0;
        for (int b = threadIdx.x + 256 * u; b < nblocks; b += 1024) {
            const double2 p = __ldcg(reinterpret_cast<const double2*>(&d.part[b]));
            const double2 q = __ldcg(reinterpret_cast<const double2*>(&d.part[b]) + 1);
            fv += p.x; ff += p.y; vv += q.x; mo = fmax(mo, q.y);
        }
        for (int o = 16; o; o >>= 1) {
            fv += __shfl_xor_sync(0xffffffffu, fv, o);
            ff += __shfl_xor_sync(0xffffffffu, ff, o);
            vv += __shfl_xor_sync(0xffffffffu, vv, o);
            mo = fmax(mo, __shfl_xor_sync(0xffffffffu, mo, o));
        }
        if (l == 0) { sh[0][w + 8 * u] = fv; sh[1][w + 8 * u] = ff; sh[2][w + 8 * u] = vv; sh[3][w + 8 * u] = mo; }
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    double fv = 0, ff = 0, vv = 0, mo = 0;
    for (int q = 0; q < 32; ++q) { fv += sh[0][q]; ff += sh[1][q]; vv += sh[2][q]; mo = fmax(mo, sh[3][q]); }
    Scal* s = d.s;
    s->arrived = 0;
    s->fdotv = fv; s->ff = ff; s->vv = vv; s->maxov = mo;
    if (fv > 0) {
        s->npos += 1;
        if (s->npos > c.ndelay) { s->dt = fmin(s->dt * c.finc, c.dtmax); s->alpha *= c.falpha; }
        s->counter = 0;
    } else {
        s->npos = 0;
        s->dt = fmax(s->dt * c.fdec, c.dtmin);
        s->alpha = c.alpha0;
        s->counter = 1;                     // velocity reset this iteration
    }
    s->iters += 1;
}

// FIRE update: back off half a step and stop on uphill power, then semi-implicit Euler
// and the velocity mixing v = (1 - a) v + a |v| F / |F| (per particle).
__global__ void k_fire_update(Dev d, Par c) {
    const Scal s = *d.s;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < c.N; i += gridDim.x * blockDim.x) {
        double4 x = d.x[i], v = d.v[i];
        const double4 f = d.f[i];
        if (s.counter) {
            x.x -= 0.5 * s.dt * v.x; x.y -= 0.5 * s.dt * v.y; x.z -= 0.5 * s.dt * v.z;
            v = make_double4(0, 0, 0, 0);
        }
        v.x += f.x * s.dt; v.y += f.y * s.dt; v.z += f.z * s.dt;
        const double vn = sqrt(v.x * v.x + v.y * v.y + v.z * v.z), fn = sqrt(f.x * f.x + f.y * f.y + f.z * f.z);
        if (fn > 0) {
            const double a = s.alpha, k = a * vn / fn;
            v.x = (1 - a) * v.x + k * f.x; v.y = (1 - a) * v.y + k * f.y; v.z = (1 - a) * v.z + k * f.z;
        }
        x.x += v.x * s.dt; x.y += v.y * s.dt; x.z += v.z * s.dt;
        d.x[i] = x; d.v[i] = v;
        const uint32_t k = cell_of(x, c);        // the next iteration's grid
        d.key[i] = k;
        atomicAdd(&d.count[k], 1u);
    }
}

inline uint64_t splitmix64(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
inline double unif(uint64_t seed, uint64_t k) {
    return (double)(splitmix64(seed * 0x2545F4914F6CDD1Dull + k) >> 11) * (1.0 / 9007199254740992.0);
}

}  // namespace pack
}  // namespace rf

using namespace rf;
using namespace rf::pack;

extern "C" rf_status rf_pack_cylinder(uint64_t seed, uint64_t N, double r0, double rmin, double rmax, double aspect,
                                      double phi, const double center[3], double* R, double* radius,
                                      double* diameter, double* height, double* max_overlap) {
    return rf_pack_cylinder_dist(seed, N, r0, rmin, rmax, RF_RADII_UNIFORM, aspect, phi, center, R, radius, diameter,
                                 height, max_overlap);
}

extern "C" rf_status rf_pack_cylinder_dist(uint64_t seed, uint64_t N, double r0, double rmin, double rmax, int dist,
                                           double aspect, double phi, const double center[3], double* R,
                                           double* radius, double* diameter, double* height, double* max_overlap) {
    if (N < 2 || !(r0 > 0) || !(rmin > 0) || !(rmax >= rmin) || !(aspect > 0) || !(phi > 0.05 && phi < 0.7) || !R ||
        !radius || !center || (dist != RF_RADII_UNIFORM && dist != RF_RADII_LOG_UNIFORM)) {
        set_error("rf_pack_cylinder: bad arguments");
        return RF_ERR_INVALID;
    }
    // work in units of r0; container sized for the target packing fraction
    std::vector<double4> hx(N);
    double vol = 0.0;
    for (uint64_t i = 0; i < N; ++i) {
        const double u = unif(seed, 4 * i + 3);
        const double r = dist == RF_RADII_LOG_UNIFORM ? rmin * std::pow(rmax / rmin, u) : rmin + (rmax - rmin) * u;
        hx[i].w = r;
        vol += 4.0 / 3.0 * M_PI * r * r * r;
    }
    const double Vc = vol / phi;
    const double D = std::cbrt(4.0 * Vc / (M_PI * aspect)), H = aspect * D;
    const double Rc = 0.5 * D, Hh = 0.5 * H;
    for (uint64_t i = 0; i < N; ++i) {      // uniform in the container (rejection on the disc)
        double x, y;
        uint64_t k = 0;
        do {
            x = (2.0 * unif(seed, 4 * i + 0 + 4 * N * k) - 1.0) * Rc;
            y = (2.0 * unif(seed, 4 * i + 1 + 4 * N * k) - 1.0) * Rc;
            ++k;
        } while (x * x + y * y > (Rc - hx[i].w) * (Rc - hx[i].w) && k < 64);
        hx[i].x = x; hx[i].y = y;
        hx[i].z = (2.0 * unif(seed, 4 * i + 2) - 1.0) * (Hh - hx[i].w);
    }
    double rmx = rmax;
    Par c{};
    c.N = (uint32_t)N;
    const double hcell = 2.0 * rmx * 1.0001;
    c.inv_h = 1.0 / hcell;
    c.ox = -Rc - hcell; c.oy = -Rc - hcell; c.oz = -Hh - hcell;
    c.nx = (uint32_t)std::ceil((2 * Rc + 2 * hcell) / hcell) + 1; c.ny = c.nx;
    c.nz = (uint32_t)std::ceil((2 * Hh + 2 * hcell) / hcell) + 1;
    c.cells = c.nx * c.ny * c.nz;
    c.Rc = Rc; c.Hh = Hh;
    c.dtmax = 1.0; c.dtmin = 1e-4; c.finc = 1.1; c.fdec = 0.5; c.alpha0 = 0.1; c.falpha = 0.99; c.ndelay = 5;
    Dev d{};
    std::vector<void*> allocs;
    auto al = [&](void** p, size_t bytes) { cudaError_t e = cudaMalloc(p, bytes); if (!e) allocs.push_back(*p); return e; };
    const int nb = (int)((N + 255) / 256) < 148 * 8 ? (int)((N + 255) / 256) : 148 * 8;
    const int per = 256 / PACK_LANES, nbf = (int)((N + per - 1) / per) < 148 * 8 ? (int)((N + per - 1) / per) : 148 * 8;
    cudaError_t e = cudaSuccess;
    if (!e) e = al((void**)&d.x, N * sizeof(double4));
    if (!e) e = al((void**)&d.v, N * sizeof(double4));
    if (!e) e = al((void**)&d.f, N * sizeof(double4));
    if (!e) e = al((void**)&d.key, N * 4);
    if (!e) e = al((void**)&d.sorted, N * 4);
    if (!e) e = al((void**)&d.count, (size_t)c.cells * 4);
    if (!e) e = al((void**)&d.start, ((size_t)c.cells + 1) * 4);
    if (!e) e = al((void**)&d.xs, N * sizeof(double4));
    if (!e) e = al((void**)&d.part, nbf * sizeof(double4));
    const uint32_t nchunks = (c.cells + SCAN_CHUNK - 1) / SCAN_CHUNK;
    if (!e) e = al((void**)&d.bsum, (size_t)nchunks * sizeof(uint32_t));
    if (!e) e = al((void**)&d.s, sizeof(Scal));
    cudaStream_t st = nullptr;
    if (!e) e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    Scal hs{};
    hs.dt = 0.1; hs.alpha = c.alpha0; hs.scale = 0.5;
    if (!e) e = cudaMemcpyAsync(d.x, hx.data(), N * sizeof(double4), cudaMemcpyHostToDevice, st);
    if (!e) e = cudaMemsetAsync(d.v, 0, N * sizeof(double4), st);
    if (!e) e = cudaMemcpyAsync(d.s, &hs, sizeof(hs), cudaMemcpyHostToDevice, st);
    // the first iteration's grid; every update counts the next one's
    if (!e) e = cudaMemsetAsync(d.count, 0, (size_t)c.cells * 4, st);
    if (!e) { k_bin<<<nb, 256, 0, st>>>(d, c); e = cudaGetLastError(); }
    // one batch of FIRE iterations, captured once and relaunched
    const int BATCH = 50;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    if (!e) e = cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal);
    if (!e) {
        for (int it = 0; it < BATCH; ++it) {
            if (nchunks <= SCAN_SELF) {
                k_scan_apply<<<nchunks, 1024, 0, st>>>(d, c, 1);
            } else {
                k_scan_sums<<<nchunks, 256, 0, st>>>(d, c);
                k_scan_chunks<<<1, 1024, 0, st>>>(d, nchunks);
                k_scan_apply<<<nchunks, 1024, 0, st>>>(d, c, 0);
            }
            k_scatter<<<nb, 256, 0, st>>>(d, c);
            k_cellsort<<<(c.N + 127) / 128, 128, 0, st>>>(d, c);
            k_force<<<nbf, 256, 0, st>>>(d, c);
            k_fire_update<<<nb, 256, 0, st>>>(d, c);
        }
        e = cudaStreamEndCapture(st, &graph);
    }
    if (!e) e = cudaGraphInstantiate(&exec, graph, 0);
    // radius growth: g from 0.5 to 1, relaxing each stage to a small overlap
    double g = 0.5, mo = 0.0;
    const int max_batches_per_stage = 200;
    for (int stage = 0; !e && stage < 400; ++stage) {
        const double tol = (g >= 1.0) ? 2e-4 : 5e-3;
        int b = 0;
        for (; b < max_batches_per_stage && !e; ++b) {
            e = cudaGraphLaunch(exec, st);
            if (!e) e = cudaMemcpyAsync(&hs, d.s, sizeof(hs), cudaMemcpyDeviceToHost, st);
            if (!e) e = cudaStreamSynchronize(st);
            if (hs.maxov < tol) break;
        }
        mo = hs.maxov;
        if (g >= 1.0) break;
        g = std::min(1.0, g * 1.02);
        hs.scale = g;
        // keep dt/alpha, restart the positive-power count
        hs.npos = 0;
        if (!e) e = cudaMemcpyAsync(d.s, &hs, sizeof(hs), cudaMemcpyHostToDevice, st);
        (void)b;
    }
    if (!e) e = cudaMemcpyAsync(hx.data(), d.x, N * sizeof(double4), cudaMemcpyDeviceToHost, st);
    if (!e) e = cudaStreamSynchronize(st);
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    if (st) cudaStreamDestroy(st);
    for (void* p : allocs) cudaFree(p);
    if (e) return cuda_status(e, "rf_pack_cylinder");
    // number the particles in spatial order (cells of 6 r0, x fastest, then y, then z;
    // packing order within a cell), so that a particle's neighbours sit close to it in
    // memory and the step kernels' neighbour gathers hit the caches
    std::vector<uint64_t> key(N), order(N);
    {
        const double h = 6.0;
        const double x0 = -Rc, y0 = -Rc, z0 = -Hh;
        const uint64_t nx = (uint64_t)std::ceil(2.0 * Rc / h) + 2, ny = nx;
        for (uint64_t i = 0; i < N; ++i) {
            const double fx = std::floor((hx[i].x - x0) / h), fy = std::floor((hx[i].y - y0) / h),
                         fz = std::floor((hx[i].z - z0) / h);
            const uint64_t cx = fx < 0 ? 0 : (uint64_t)fx, cy = fy < 0 ? 0 : (uint64_t)fy, cz = fz < 0 ? 0 : (uint64_t)fz;
            key[i] = cx + nx * (cy + ny * cz);
            order[i] = i;
        }
        std::stable_sort(order.begin(), order.end(), [&](uint64_t a, uint64_t b) { return key[a] < key[b]; });
    }
    for (uint64_t q = 0; q < N; ++q) {
        const double4& p = hx[order[q]];
        R[q] = center[0] + r0 * p.x;
        R[q + N] = center[1] + r0 * p.y;
        R[q + 2 * N] = center[2] + r0 * p.z;
        radius[q] = r0 * p.w;
    }
    if (diameter) *diameter = r0 * D;
    if (height) *height = r0 * H;
    if (max_overlap) *max_overlap = mo;
    return RF_OK;
}
