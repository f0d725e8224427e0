// md_* drop-in kernels: the RockFit-DEM hot-path step operations on buffers in the
// reference's own layout (md_data_types.h), in place, on a caller stream.
//
// Rows are read by warps, a lane a slot: the reference's row-major layout (8-byte ids,
// 12-byte slot state) is then read in whole lines, where one thread a row touches a line
// of its own with every load. A slot's force and moment terms are kept apart and added by
// the particle's lane in slot order, as the reference's row loops run, so the sums round
// the same way. Cell binning replaces cub's radix sort with a
// counting sort (histogram, scan, scatter, per-cell id order), whose output is
// the same stable (cell, id) order.
#include <cstdio>
#include <mutex>
#include "rf_physics.cuh"

namespace rf {

typedef uint_fast32_t mid_t;   // the reference's id type at this boundary
static_assert(sizeof(mid_t) == 8 || sizeof(mid_t) == 4, "unexpected uint_fast32_t width");

__device__ __forceinline__ f3 ld3p(const float* P, size_t N, size_t i) {   // planar x|y|z
    return mk3(P[i], P[i + N], P[i + 2 * N]);
}
__device__ __forceinline__ f3 ld3(const rf_float3* p, size_t k) { return mk3(p[k].x, p[k].y, p[k].z); }
__device__ __forceinline__ void st3(rf_float3* p, size_t k, f3 v) { p[k].x = v.x; p[k].y = v.y; p[k].z = v.z; }

static inline int grid_for(size_t n, int block) {
    size_t g = (n + block - 1) / block;
    if (g < 1) g = 1;
    if (g > 148 * 16) g = 148 * 16;
    return (int)g;
}

static inline unsigned row_grid(size_t N, int per_cta) { return (unsigned)((N + per_cta - 1) / per_cta); }

// ---------------------------------------------------------------------------
// Cells
// ---------------------------------------------------------------------------
__global__ void k_cell_index(const float* __restrict__ R, size_t N, mid_t* __restrict__ CI, RefGrid g,
                             uint32_t* __restrict__ counts, uint32_t* err) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x) {
        uint32_t cx, cy, cz;
        const uint32_t c = ref_cell(ld3p(R, N, i), g, &cx, &cy, &cz);
        CI[i] = (mid_t)c;
        if (cx > g.nx - 1 || cy > g.ny - 1 || cz > g.nz - 1 || (uint64_t)c >= g.CN)
            raise_status(err, RF_ERR_CELL_RANGE);
        // binned by the key, as the sort orders it: a key past the grid goes to the tail
        // bin; an out-of-range cell coordinate whose linear key still lands inside the grid
        // (it wraps into another row) is binned under that key, as the scatter files it
        if (counts) atomicAdd(&counts[(uint64_t)c < g.CN ? (uint64_t)c : g.CN], 1u);
    }
}

// Exclusive scan, three passes: per-block totals, scan of totals, add back.
__global__ void k_scan_block_sums(const uint32_t* __restrict__ in, size_t n, uint32_t* __restrict__ bsum) {
    __shared__ uint32_t sh[32];
    const size_t base = (size_t)blockIdx.x * 4096;
    uint32_t s = 0;
    for (int t = threadIdx.x; t < 4096; t += blockDim.x)
        if (base + t < n) s += in[base + t];
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        uint32_t v = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : 0;
        for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (threadIdx.x == 0) bsum[blockIdx.x] = v;
    }
}
__global__ void k_scan_totals(uint32_t* __restrict__ bsum, size_t nb) {
    const int lane = threadIdx.x;                // one warp
    uint32_t acc = 0;
    for (size_t b0 = 0; b0 < nb; b0 += 32) {
        const uint32_t v = b0 + lane < nb ? bsum[b0 + lane] : 0;
        uint32_t incl = v;
        for (int o = 1; o < 32; o <<= 1) { const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += y; }
        if (b0 + lane < nb) bsum[b0 + lane] = acc + incl - v;
        acc += __shfl_sync(0xffffffffu, incl, 31);
    }
}
// 1024 threads x 4 items per block of 4096
__global__ void k_scan_apply(const uint32_t* __restrict__ in, size_t n, const uint32_t* __restrict__ boff,
                             uint32_t* __restrict__ out) {
    __shared__ uint32_t wsum[32];
    const size_t base = (size_t)blockIdx.x * 4096 + (size_t)threadIdx.x * 4;
    uint32_t v[4], t = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) { v[q] = (base + q < n) ? in[base + q] : 0; t += v[q]; }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t incl = t;
    for (int o = 1; o < 32; o <<= 1) { uint32_t y = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += y; }
    if (lane == 31) wsum[w] = incl;
    __syncthreads();
    if (w == 0) {
        uint32_t s = lane < (int)(blockDim.x >> 5) ? wsum[lane] : 0, si = s;
        for (int o = 1; o < 32; o <<= 1) { uint32_t y = __shfl_up_sync(0xffffffffu, si, o); if (lane >= o) si += y; }
        wsum[lane] = si - s;
    }
    __syncthreads();
    uint32_t run = boff[blockIdx.x] + wsum[w] + incl - t;
#pragma unroll
    for (int q = 0; q < 4; ++q) { if (base + q < n) out[base + q] = run; run += v[q]; }
}

__global__ void k_cell_scatter(const mid_t* __restrict__ CI, size_t N, uint64_t CN, const uint32_t* __restrict__ start,
                               uint32_t* __restrict__ fill, mid_t* __restrict__ CIs) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x) {
        const uint64_t c = (uint64_t)CI[i];
        const uint64_t b = c < CN ? c : CN;
        const uint32_t p = start[b] + atomicAdd(&fill[b], 1u);
        CIs[N + p] = (mid_t)i;
    }
}

// Order each cell's ids ascending (the stable sort's tie order), write the sorted keys and
// pnC. A warp takes 32 cells: their counts and pnC in whole lines, then the occupied ones
// one after another, a lane an occupant (its place is the number of smaller ids). Cells of
// more than 32, and the tail bin (ordered by key, then id), are sorted by one lane.
__device__ __noinline__ void sort_run(const mid_t* CI, mid_t* ids, uint32_t n, bool tail) {
    for (uint32_t a = 1; a < n; ++a) {
        mid_t v = ids[a];
        uint64_t kv = tail ? (uint64_t)CI[v] : 0;
        uint32_t b = a;
        while (b > 0) {
            mid_t u = ids[b - 1];
            uint64_t ku = tail ? (uint64_t)CI[u] : 0;
            if (ku < kv || (ku == kv && u < v)) break;
            ids[b] = u;
            --b;
        }
        ids[b] = v;
    }
}
__global__ void __launch_bounds__(128) k_cell_finish(const mid_t* __restrict__ CI, size_t N, uint64_t CN,
                                                     const uint32_t* __restrict__ counts, const uint32_t* __restrict__ start,
                                                     mid_t* CIs, mid_t* __restrict__ pnC) {
    const uint32_t FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const uint64_t c = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x);
    uint32_t cn = 0, cs = 0;
    if (c <= CN) { cn = counts[c]; cs = start[c]; }
    if (c < CN) {
        pnC[c] = cn ? (mid_t)cs : (mid_t)0;
        pnC[c + CN] = (mid_t)cn;
    }
    uint32_t occupied = __ballot_sync(FULL, cn != 0);
    while (occupied) {
        const int l = __ffs(occupied) - 1;
        occupied &= occupied - 1;
        const uint32_t n = __shfl_sync(FULL, cn, l), s = __shfl_sync(FULL, cs, l);
        const uint64_t cell = c - lane + l;
        mid_t* ids = CIs + N + s;
        if (n <= 32 && cell < CN) {
            const mid_t v = (uint32_t)lane < n ? ids[lane] : empty_id<mid_t>();
            uint32_t rank = 0;
            for (uint32_t q = 0; q < n; ++q) rank += __shfl_sync(FULL, v, q) < v ? 1u : 0u;
            __syncwarp();
            if ((uint32_t)lane < n) {
                ids[rank] = v;
                CIs[s + lane] = (mid_t)cell;
            }
        } else {
            if (lane == 0) sort_run(CI, ids, n, cell >= CN);
            __syncwarp();
            for (uint32_t q = lane; q < n; q += 32) CIs[s + q] = cell < CN ? (mid_t)cell : CI[ids[q]];
        }
    }
}

// d_DetermineCellPointer's run scan continues past N into the id half of CIs
// (md_calculate_cell.cu:72): the last run's count grows by one when CIs[N] equals
// its key. Reproduced so pnC matches the reference bit for bit.
__global__ void k_cell_last_run(size_t N, uint64_t CN, mid_t* __restrict__ CIs, mid_t* __restrict__ pnC) {
    if (threadIdx.x == 0 && blockIdx.x == 0 && N > 0) {
        const mid_t last = CIs[N - 1];
        if ((uint64_t)last < CN && CIs[N] == last) pnC[last + CN] += 1;
    }
}

// ---------------------------------------------------------------------------
// Rows
// ---------------------------------------------------------------------------
// Eight lanes per particle, one per octant cell: a lane walks its own cell's occupants.
constexpr int LIST_GROUP = 8;            // lanes a particle
constexpr int LIST_PARTICLES = 16;       // particles a 128-thread CTA

// First occupant and count of a cell's run; out-of-grid cells are empty and reported.
__device__ __forceinline__ void cell_run(const mid_t* pnC, uint64_t CN, int64_t cell, uint64_t& s, uint64_t& n,
                                         uint32_t* err) {
    s = 0; n = 0;
    if (cell < 0 || (uint64_t)cell >= CN) { raise_status(err, RF_ERR_CELL_RANGE); return; }
    s = (uint64_t)pnC[cell]; n = (uint64_t)pnC[cell + CN];
}

// A lane counts the pairs of its cell, the group's prefix sums give each cell's place in the
// row, and a second walk (its positions are in the caches by then) writes them in order.
__global__ void __launch_bounds__(128) k_list_construct(const float* __restrict__ R, size_t N, const mid_t* __restrict__ CIs,
                                                        const mid_t* __restrict__ pnC, mid_t* __restrict__ IL, uint32_t K,
                                                        RefGrid g, float aacut, uint32_t* err) {
    const int sub = threadIdx.x % LIST_GROUP;
    const size_t i = (size_t)blockIdx.x * LIST_PARTICLES + threadIdx.x / LIST_GROUP;
    const bool valid = i < N;
    f3 xi = mk3(0.f, 0.f, 0.f);
    uint64_t s = 0, cnt = 0;
    if (valid) {
        xi = ld3p(R, N, i);
        cell_run(pnC, g.CN, octant_cell(octant_of(xi, g), sub), s, cnt, err);
        if (s > N) s = N;
        if (cnt > N - s) cnt = N - s;
    }
    auto hit = [&](uint64_t m, mid_t& j) {
        j = CIs[s + m + N];
        return (size_t)j < N && dist2_rn(xi, ld3p(R, N, j)) < aacut && (size_t)j != i;
    };
    uint32_t n = 0;
    mid_t j;
    for (uint64_t m = 0; m < cnt; ++m) n += hit(m, j) ? 1u : 0u;
    uint32_t at = n;
    for (int o = 1; o < LIST_GROUP; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, at, o, LIST_GROUP);
        if (sub >= o) at += y;
    }
    at -= n;
    if (n && (uint64_t)at + n > K) raise_status(err, RF_ERR_ROW_OVERFLOW);
    for (uint64_t m = 0; n && m < cnt; ++m)
        if (hit(m, j)) {
            if (at < K) IL[i * K + at] = j;
            ++at; --n;
        }
}

// InteractionListReConstructBPM of one particle by one thread: candidates in cell order, the
// row scanned for each (addnewlinkbpm, md_interaction_list_reconstructbpm.cu:25-41; slot 0
// of particle 0 reads as "none found").
__device__ __noinline__ void reconstruct_row(const float* R, size_t N, size_t i, const mid_t* CIs, const mid_t* pnC,
                                             mid_t* IL, uint8_t* ILtype, uint32_t K, const RefGrid& g, float aacut,
                                             uint32_t* err) {
    const mid_t E = empty_id<mid_t>();
    const f3 xi = ld3p(R, N, i);
    const Octant oc = octant_of(xi, g);
    mid_t* row = IL + i * K;
    for (int c = 0; c < 8; ++c) {
        uint64_t s, cnt;
        cell_run(pnC, g.CN, octant_cell(oc, c), s, cnt, err);
        for (uint64_t m = 0; m < cnt; ++m) {
            if (s + m >= N) break;
            const mid_t j = CIs[s + m + N];
            if ((size_t)j >= N) continue;
            const float rr = dist2_rn(xi, ld3p(R, N, j));
            if (!(rr < aacut && (double)rr > 1e-10)) continue;
            uint64_t kfree = 0;
            bool any_free = false, found = false;
            for (uint32_t q = 0; q < K; ++q) {
                const mid_t kj = row[q];
                if (kj == E) {
                    any_free = true;
                    if (kfree == 0) kfree = i * K + q;
                }
                if (kj == j) { found = true; break; }
            }
            if (found) continue;
            // A full row: the reference writes IL[0] here; the row is left unchanged instead.
            if (!any_free) { raise_status(err, RF_ERR_ROW_OVERFLOW); continue; }
            IL[kfree] = j;
            ILtype[kfree] = 0;
        }
    }
}

// Almost every candidate of a step is in the row already. The group's lanes first mark the
// candidates of their cells within the cutoff (32 at a time), then look those up in the row,
// staged in shared memory as 32-bit ids (marking first: a look-up in the same loop would be
// run by the whole warp for each of its lanes' hits in turn). A particle with one that is
// missing is taken again in the reference's order by one lane. Rows too long to stage
// (K > LIST_STAGE_K) go there at once. Bound by the instructions of the candidate walk (24 a
// cell and lane): 198k particles 281 us with one thread a particle that scans the row
// for every hit, 144 us so; the lanes of a group side by side in one cell took longer.
constexpr uint32_t LIST_STAGE_K = 512;
__global__ void __launch_bounds__(128) k_list_reconstruct_bpm(const float* __restrict__ R, size_t N,
                                                              const mid_t* __restrict__ CIs, const mid_t* __restrict__ pnC,
                                                              mid_t* __restrict__ IL, uint8_t* __restrict__ ILtype,
                                                              uint32_t K, RefGrid g, float aacut, uint32_t* err) {
    extern __shared__ uint4 s_rows[];
    const int sub = threadIdx.x % LIST_GROUP, p = threadIdx.x / LIST_GROUP;
    const size_t i = (size_t)blockIdx.x * LIST_PARTICLES + p;
    const bool valid = i < N;
    bool missing = false;
    if (K <= LIST_STAGE_K) {
        const uint32_t quads = (K + 3) / 4;
        uint4* row = s_rows + (size_t)p * (quads | 1u);       // (odd: groups start in different banks)
        uint32_t* row1 = reinterpret_cast<uint32_t*>(row);
        if (valid)
            for (uint32_t q = sub; q < 4 * quads; q += LIST_GROUP) row1[q] = q < K ? (uint32_t)IL[i * K + q] : EMPTY32;
        __syncwarp();
        if (valid) {
            const float *X = R, *Y = R + N, *Z = R + 2 * N;
            const f3 xi = mk3(X[i], Y[i], Z[i]);
            uint64_t s, cnt;
            cell_run(pnC, g.CN, octant_cell(octant_of(xi, g), sub), s, cnt, err);
            if (s > N) s = N;
            if (cnt > N - s) cnt = N - s;
            const mid_t* ids = CIs + N + s;
            for (uint32_t left = (uint32_t)cnt; left;) {
                const uint32_t n = left < 32u ? left : 32u;
                uint32_t hits = 0;
#pragma unroll 4
                for (uint32_t m = 0; m < n; ++m) {
                    const mid_t j = ids[m];
                    if ((size_t)j >= N) continue;
                    const float rr = dist2_rn(xi, mk3(X[(uint32_t)j], Y[(uint32_t)j], Z[(uint32_t)j]));
                    if (rr < aacut && above_1em10(rr)) hits |= 1u << m;
                }
                while (hits) {
                    const uint32_t j = (uint32_t)ids[__ffs(hits) - 1];
                    hits &= hits - 1;
                    bool found = false;
#pragma unroll 8
                    for (uint32_t q = 0; q < quads; ++q) {
                        const uint4 e = row[q];
                        found |= e.x == j || e.y == j || e.z == j || e.w == j;
                    }
                    missing |= !found;
                }
                ids += n;
                left -= n;
            }
        }
    } else {
        missing = valid;
    }
    const uint32_t any = __ballot_sync(0xffffffffu, missing);
    if (sub == 0 && ((any >> (threadIdx.x & 24)) & 0xFFu))
        reconstruct_row(R, N, i, CIs, pnC, IL, ILtype, K, g, aacut, err);
}

// ---------------------------------------------------------------------------
// Row kernels: a warp takes ROWS consecutive rows, a lane a slot (32 slots at a time)
// ---------------------------------------------------------------------------
constexpr int ROWS = 8;
constexpr int ROW_CTA = 4 * ROWS;        // rows of a 128-thread CTA

__global__ void __launch_bounds__(128) k_delete_far_links(const float* __restrict__ R, size_t N, mid_t* __restrict__ IL,
                                                          uint8_t* __restrict__ ILtype, rf_float3* Rij, rf_float3* Oijt,
                                                          rf_float3* Fijn, rf_float3* Fijt, rf_float3* Mijn,
                                                          rf_float3* Mijt, rf_float3* Mijadd, uint32_t K, float aacut) {
    const mid_t E = empty_id<mid_t>();
    const f3 z = mk3(0.f, 0.f, 0.f);
    const int lane = threadIdx.x & 31;
    const size_t base = ((size_t)blockIdx.x * 4 + (threadIdx.x >> 5)) * ROWS;
    for (uint32_t c0 = 0; c0 < K; c0 += 32) {
        const uint32_t q = c0 + lane;
        mid_t id[ROWS];
        uint32_t far = 0;
#pragma unroll
        for (int r = 0; r < ROWS; ++r) id[r] = (q < K && base + r < N) ? IL[(base + r) * K + q] : E;
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            if (id[r] == E || (size_t)id[r] >= N) continue;
            const float rr = dist2_rn(ld3p(R, N, base + r), ld3p(R, N, id[r]));
            if (rr > aacut || below_1em10(rr)) far |= 1u << r;
        }
        while (far) {                            // few: links drift out one at a time
            const int r = __ffs(far) - 1;
            far &= far - 1;
            const size_t k = (base + r) * K + q;
            IL[k] = E;
            ILtype[k] = 0;
            // 1/L0 is left as it was: the reference's "_1d_iL = 0;" clears its own pointer.
            st3(Rij, k, z); st3(Oijt, k, z); st3(Fijn, k, z); st3(Fijt, k, z);
            st3(Mijn, k, z); st3(Mijt, k, z); st3(Mijadd, k, z);
        }
    }
}

__global__ void __launch_bounds__(128) k_construct_bonds(const float* __restrict__ R, size_t N, const mid_t* __restrict__ IL,
                                                         uint8_t* __restrict__ ILtype, float* __restrict__ iL,
                                                         rf_float3* Rij, rf_float3* Oijt, rf_float3* Fijn, rf_float3* Fijt,
                                                         rf_float3* Mijn, rf_float3* Mijt, rf_float3* Mijadd, uint32_t K,
                                                         float aa_create) {
    const mid_t E = empty_id<mid_t>();
    const f3 z = mk3(0.f, 0.f, 0.f);
    const int lane = threadIdx.x & 31;
    const size_t base = ((size_t)blockIdx.x * 4 + (threadIdx.x >> 5)) * ROWS;
    for (int r = 0; r < ROWS && base + r < N; ++r) {
        const size_t i = base + r;
        const f3 xi = ld3p(R, N, i);
        for (uint32_t q = lane; q < K; q += 32) {
            const size_t k = i * K + q;
            const mid_t j = IL[k];
            if (j == E || (size_t)j >= N) continue;
            const f3 xj = ld3p(R, N, j);
            const float rx = xj.x - xi.x, ry = xj.y - xi.y, rz = xj.z - xi.z;
            const float rm2 = rm2_bond(rx, ry, rz);
            if (rm2 < aa_create && (double)rm2 > 1e-18) {
                iL[k] = __frsqrt_rn(rm2);
                ILtype[k] = 1;
            } else {
                ILtype[k] = 0;
            }
            st3(Rij, k, z); st3(Oijt, k, z); st3(Fijn, k, z); st3(Fijt, k, z);
            st3(Mijn, k, z); st3(Mijt, k, z); st3(Mijadd, k, z);
        }
    }
}

// ---------------------------------------------------------------------------
// Forces
// ---------------------------------------------------------------------------
// d_CalculateForcesDEM_22 (BOND) and _21 over the rows. The lanes of a warp first look at a
// row's slots (coalesced ids and types); the slots with work -- intact bonds, or overlapping
// type-0 pairs -- go into a list in row and slot order, and whenever it holds 32 every lane
// evaluates one. The terms wait in shared memory for the particle's lane (lane r of the warp
// adds row r's, in slot order). Bound by the row and state traffic (32-byte sectors of
// 12-byte state): 198k particles, K = 32, bonds 177 -> 113 us and contacts 181 -> 84 us against
// one thread a row.
template <bool BOND, class Par>
__global__ void __launch_bounds__(128, 6) k_row_forces(const float* __restrict__ R, const float* __restrict__ V,
                                                    const float* __restrict__ W, const mid_t* __restrict__ IL,
                                                    uint8_t* __restrict__ ILtype, const float* __restrict__ iL,
                                                    rf_float3* __restrict__ Rij, rf_float3* __restrict__ Oijt,
                                                    rf_float3* __restrict__ Mijn, rf_float3* __restrict__ Mijt,
                                                    float* __restrict__ F, float* __restrict__ M, size_t N, uint32_t K,
                                                    Par p) {
    constexpr int NF = 2, NM = BOND ? 3 : 2, NT = 3 * (NF + NM);
    __shared__ uint32_t s_id[4][64], s_at[4][64];       // list: neighbour, slot (row in the warp * K + slot)
    __shared__ float s_t[4][NT][32];                    // the terms of a round
    __shared__ uint8_t s_nm[4][32];                     // moment terms of an entry, 0x80: then clear
    __shared__ float s_own[4][ROWS][9];                 // the rows' positions, velocities, spins
    const mid_t E = empty_id<mid_t>();
    const uint32_t FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const size_t base = ((size_t)blockIdx.x * 4 + wp) * ROWS;
    if (base >= N) return;
    const int rows = N - base < (size_t)ROWS ? (int)(N - base) : ROWS;
    for (int q = lane; q < ROWS * 9; q += 32) {
        const int c = q / ROWS, r = q % ROWS;
        const float* a = c < 3 ? R : c < 6 ? V : W;
        s_own[wp][r][c] = r < rows ? a[base + r + (size_t)(c % 3) * N] : 0.f;
    }
    __syncwarp();
    f3 fs = mk3(0.f, 0.f, 0.f), ms = fs;                // lane r: the sums of row r
    float rP = 0.f;
    if constexpr (!BOND) rP = p.rP;
    uint32_t head = 0, cnt = 0;
    auto round = [&](uint32_t n) {
        int row = -1;
        if ((uint32_t)lane < n) {
            const uint32_t e = (head + lane) & 63u;
            const size_t j = s_id[wp][e];
            const uint32_t at = s_at[wp][e];
            row = (int)(at / K);
            const size_t k = base * K + at;
            const float* o = s_own[wp][row];
            const f3 xi = mk3(o[0], o[1], o[2]), vi = mk3(o[3], o[4], o[5]), wi = mk3(o[6], o[7], o[8]);
            const f3 xj = ld3p(R, N, j);
            const f3 r = mk3(xj.x - xi.x, xj.y - xi.y, xj.z - xi.z);
            KeepTerms t;
            if constexpr (BOND) {
                f3 rij = ld3(Rij, k), oijt = ld3(Oijt, k), mijn = ld3(Mijn, k), mijt = ld3(Mijt, k);
                const bool broke = bond_slot(p, r, vi, ld3p(V, N, j), wi, ld3p(W, N, j), iL[k], rij, oijt, mijn, mijt, t);
                st3(Rij, k, rij); st3(Oijt, k, oijt); st3(Mijn, k, mijn); st3(Mijt, k, mijt);
                if (broke) ILtype[k] = 0;
            } else {
                f3 oijt = ld3(Oijt, k);
                contact_pair(p, r, norm3(r.x, r.y, r.z), vi, ld3p(V, N, j), wi, ld3p(W, N, j), oijt, t);
                st3(Oijt, k, oijt);
                s_nm[wp][lane] = t.clear ? 0x80 : 0;
                if (t.clear) t.mt[1] = mk3(0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int q = 0; q < NF; ++q) {
                s_t[wp][3 * q][lane] = t.ft[q].x; s_t[wp][3 * q + 1][lane] = t.ft[q].y; s_t[wp][3 * q + 2][lane] = t.ft[q].z;
            }
#pragma unroll
            for (int q = 0; q < NM; ++q) {
                const int b = 3 * (NF + q);
                s_t[wp][b][lane] = t.mt[q].x; s_t[wp][b + 1][lane] = t.mt[q].y; s_t[wp][b + 2][lane] = t.mt[q].z;
            }
        }
        uint32_t mine = 0;
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            const uint32_t b = __ballot_sync(FULL, row == r);
            if (lane == r) mine = b;
        }
        __syncwarp();
        while (mine) {
            const int e = __ffs(mine) - 1;
            mine &= mine - 1;
#pragma unroll
            for (int q = 0; q < NF; ++q) {
                fs.x += s_t[wp][3 * q][e]; fs.y += s_t[wp][3 * q + 1][e]; fs.z += s_t[wp][3 * q + 2][e];
            }
            if (!BOND && s_nm[wp][e]) { ms = mk3(0.f, 0.f, 0.f); continue; }
#pragma unroll
            for (int q = 0; q < NM; ++q) {
                const int b = 3 * (NF + q);
                ms.x += s_t[wp][b][e]; ms.y += s_t[wp][b + 1][e]; ms.z += s_t[wp][b + 2][e];
            }
        }
        __syncwarp();
        head += n; cnt -= n;
    };
    for (uint32_t c0 = 0; c0 < K; c0 += 32) {
        const uint32_t q = c0 + lane;
        mid_t id[ROWS];
        uint8_t ty[ROWS];
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            const bool in = q < K && r < rows;
            id[r] = in ? IL[(base + r) * K + q] : E;
            ty[r] = in ? ILtype[(base + r) * K + q] : 1;
        }
        uint32_t todo = 0, zero = 0;                    // rows whose slot of this lane has work, has no overlap
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            if (BOND) {
                if (id[r] != E && ty[r] == 1) todo |= 1u << r;
            } else if (id[r] == E) {
                zero |= 1u << r;                        // empty and open slots keep no overlap
            } else if (ty[r] == 0) {
                const float* o = s_own[wp][r];
                const f3 xj = ld3p(R, N, (size_t)id[r]);
                const bool touch = norm3(xj.x - o[0], xj.y - o[1], xj.z - o[2]) < 2.0f * rP;
                (touch ? todo : zero) |= 1u << r;
            }
        }
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            if (r >= rows) break;                       // (uniform)
            const bool work = (todo >> r) & 1u;
            if (!BOND) {
                const uint32_t zm = __ballot_sync(FULL, ((zero >> r) & 1u) && q < K);
                float* oz = (float*)(Oijt + (base + r) * K + c0);
#pragma unroll
                for (int f = lane; f < 96; f += 32)
                    if ((zm >> (f / 3)) & 1u) oz[f] = 0.f;
            }
            const uint32_t bal = __ballot_sync(FULL, work);
            if (work) {
                const uint32_t e = (head + cnt + __popc(bal & ((1u << lane) - 1u))) & 63u;
                s_id[wp][e] = (uint32_t)id[r];
                s_at[wp][e] = (uint32_t)r * K + q;
            }
            cnt += __popc(bal);
            __syncwarp();
            if (cnt >= 32) round(32);
        }
    }
    if (cnt) round(cnt);
    if (lane < rows) {
        const size_t i = base + lane;
        F[i] += fs.x; F[i + N] += fs.y; F[i + 2 * N] += fs.z;
        M[i] += ms.x; M[i + N] += ms.y; M[i + 2 * N] += ms.z;
    }
}

__global__ void k_increments(const float* __restrict__ F, float* __restrict__ V, float* __restrict__ R,
                             const float* __restrict__ M, float* __restrict__ W, size_t N, float dtm, float dt, float dtI) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x)
        for (int c = 0; c < 3; ++c) {
            const size_t q = i + c * N;
            V[q] += __fmul_rn(F[q], dtm);
            R[q] += __fmul_rn(V[q], dt);
            W[q] += __fmul_rn(M[q], dtI);
        }
}

// Block-wide sum of two doubles (deterministic tree).
__device__ __forceinline__ void block_sum2(double& a, double& b) {
    __shared__ double sa[32], sb[32];
    for (int o = 16; o; o >>= 1) { a += __shfl_xor_sync(0xffffffffu, a, o); b += __shfl_xor_sync(0xffffffffu, b, o); }
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) { sa[w] = a; sb[w] = b; }
    __syncthreads();
    if (w == 0) {
        a = l < (int)(blockDim.x >> 5) ? sa[l] : 0.0;
        b = l < (int)(blockDim.x >> 5) ? sb[l] : 0.0;
        for (int o = 16; o; o >>= 1) { a += __shfl_xor_sync(0xffffffffu, a, o); b += __shfl_xor_sync(0xffffffffu, b, o); }
    }
}

__global__ void k_brazil(float* R, float* V, float* F, float* FL, size_t N, rf_float3 c, float RR, float Yt, float Yb,
                         float Ytr, float Ybr, float vt, float Zcut, uint64_t nblocks) {
    double sfb = 0.0, sft = 0.0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x)
        brazil_particle(R[i], R[i + N], R[i + 2 * N], V[i], V[i + N], V[i + 2 * N], F[i], F[i + N], F[i + 2 * N], c,
                        RR, Yt, Yb, Ytr, Ybr, vt, Zcut, sfb, sft);
    block_sum2(sfb, sft);
    if (threadIdx.x == 0) { FL[blockIdx.x] = (float)sfb; FL[nblocks + blockIdx.x] = (float)sft; }
}

__global__ void k_uniaxial(float* R, float* V, float* F, float* FL, size_t N, rf_float3 c, float RR, float Zt, float Zb,
                           float Ztr, float Zbr, float vt, float Zcut, uint64_t nblocks) {
    double sfb = 0.0, sft = 0.0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x)
        uniaxial_particle(R[i], R[i + N], R[i + 2 * N], V[i + 2 * N], F[i + 2 * N], c, RR, Zt, Zb, Ztr, Zbr, vt, Zcut,
                          sfb, sft);
    block_sum2(sfb, sft);
    if (threadIdx.x == 0) { FL[blockIdx.x] = (float)sfb; FL[nblocks + blockIdx.x] = (float)sft; }
}

__global__ void k_cut(float* R, float* V, float* F, size_t N, rf_float3 c, rf_float3 h, rf_float3 hp) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x) {
        if (outside_box(R[i], R[i + N], R[i + 2 * N], c, h)) {
            R[i] = hp.x; R[i + N] = hp.y; R[i + 2 * N] = hp.z;
            V[i] = 0.f; V[i + N] = 0.f; V[i + 2 * N] = 0.f;
            F[i] = 0.f; F[i + N] = 0.f; F[i + 2 * N] = 0.f;
        }
    }
}

// d_CalculateIncrementsFIRE (md_firerelaxation.cu:18-56)
__global__ void k_fire_inc(const float* __restrict__ F, float* __restrict__ V, float* __restrict__ R, size_t N, float dtm,
                           float dt, float a) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x) {
        const float Fx = F[i], Fy = F[i + N], Fz = F[i + 2 * N];
        float vx = __fmul_rn(Fx, dtm), vy = __fmul_rn(Fy, dtm), vz = __fmul_rn(Fz, dtm);
        const float vv = vx * vx + vy * vy + vz * vz;
        const float f = Fx * Fx + Fy * Fy + Fz * Fz;
        float vdf;
        if (f > 1e-12f) vdf = a * __fsqrt_rn(vv * __frcp_rn(f));
        else vdf = a * __fsqrt_rn(vv) * 1e6f;
        vx = (1.0f - a) * vx + vdf * Fx;
        vy = (1.0f - a) * vy + vdf * Fy;
        vz = (1.0f - a) * vz + vdf * Fz;
        V[i] = vx; V[i + N] = vy; V[i + 2 * N] = vz;
        R[i] += __fmul_rn(vx, dt); R[i + N] += __fmul_rn(vy, dt); R[i + 2 * N] += __fmul_rn(vz, dt);
    }
}
__global__ void k_fire_half(const float* __restrict__ V, float* __restrict__ R, size_t N, float dt2) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < 3 * N; i += (size_t)gridDim.x * blockDim.x)
        R[i] -= __fmul_rn(V[i], dt2);
}
__global__ void k_fdotv(const float* __restrict__ V, const float* __restrict__ F, size_t N, double* __restrict__ partial) {
    double s = 0.0, dummy = 0.0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < 3 * N; i += (size_t)gridDim.x * blockDim.x)
        s += (double)F[i] * (double)V[i];
    block_sum2(s, dummy);
    if (threadIdx.x == 0) partial[blockIdx.x] = s;
}
// Identity of the CUDA context current on the calling thread, unique within the process
// (cuCtxGetId). A cudaDeviceReset destroys the device's primary context together with
// every device address taken in it; the next runtime call makes a new context with a
// new id, so an address cached with the id of the context it came from is known to be
// stale when the ids differ. cudaSetDevice makes the device's primary context current
// (creating it if needed) and allocates nothing. The driver functions come through
// cudaGetDriverEntryPoint, so the library keeps linking against the runtime only.
static rf_status current_context_id(int dev, unsigned long long* id) {
    typedef int (*ctx_get_current_t)(void**);
    typedef int (*ctx_get_id_t)(void*, unsigned long long*);
    static ctx_get_current_t get_current = nullptr;
    static ctx_get_id_t get_id = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_current = (ctx_get_current_t)f;
        f = nullptr;
        if (cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_id = (ctx_get_id_t)f;
    });
    if (!get_current || !get_id) { set_error("driver entry points cuCtxGetCurrent / cuCtxGetId unavailable"); return RF_ERR_CUDA; }
    RF_CUDA(cudaSetDevice(dev));
    void* ctx = nullptr;
    if (get_current(&ctx) != 0 || !ctx || get_id(ctx, id) != 0) {
        set_error("no CUDA context current on device %d", dev);
        return RF_ERR_CUDA;
    }
    return RF_OK;
}

// Status word of the md_* launches of one host thread on the current device (one per
// device, re-made when the device's context was reset). nullptr if it cannot be had.
static uint32_t* status_word() {
    const int kMaxDev = 64;
    static thread_local uint32_t* w[kMaxDev] = {nullptr};
    static thread_local unsigned long long ctx[kMaxDev] = {0};
    int dev = 0;
    unsigned long long id = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDev) return nullptr;
    if (current_context_id(dev, &id) != RF_OK) return nullptr;
    if (!w[dev] || ctx[dev] != id) {
        // a word of an earlier context went away with it; a word of this one is kept
        w[dev] = nullptr;
        uint32_t* p = nullptr;
        if (cudaMalloc(&p, sizeof(uint32_t)) != cudaSuccess) return nullptr;
        if (cudaMemset(p, 0, sizeof(uint32_t)) != cudaSuccess) { cudaFree(p); return nullptr; }
        w[dev] = p;
        ctx[dev] = id;
    }
    return w[dev];
}

// Read and clear the status word after a launch sequence (synchronises the stream).
static rf_status take_status(cudaStream_t s) {
    uint32_t* w = status_word();
    if (!w) { set_error("md_* status word unavailable on the current device"); return RF_ERR_CUDA; }
    uint32_t h = 0;
    RF_CUDA(cudaMemcpyAsync(&h, w, sizeof(h), cudaMemcpyDeviceToHost, s));
    RF_CUDA(cudaStreamSynchronize(s));
    if (h) {
        RF_CUDA(cudaMemsetAsync(w, 0, sizeof(uint32_t), s));
        RF_CUDA(cudaStreamSynchronize(s));
        set_error("device status %u", h);
        return (rf_status)h;
    }
    return RF_OK;
}

}  // namespace rf

using namespace rf;

static inline cudaStream_t S(rf_stream s) { return (cudaStream_t)s; }
static inline RefGrid make_grid(float a, float inv_a, rf_uint3 cN, uint64_t CN) {
    RefGrid g;
    g.a = a; g.inv_a = inv_a; g.nx = cN.x; g.ny = cN.y; g.nz = cN.z; g.CN = CN;
    return g;
}

extern "C" {

rf_status md_CalculateCellIndex(const float* R, uint_fast32_t N, uint_fast32_t* CI, float _1d_a, rf_uint3 cN,
                                rf_stream stream) {
    if (!R || !CI || N == 0) { set_error("md_CalculateCellIndex: bad arguments"); return RF_ERR_INVALID; }
    RefGrid g = make_grid(0.f, _1d_a, cN, (uint64_t)cN.x * cN.y * cN.z);
    k_cell_index<<<grid_for(N, 256), 256, 0, S(stream)>>>(R, N, CI, g, nullptr, status_word());
    RF_CHECK_LAUNCH("k_cell_index");
    return take_status(S(stream));
}

size_t md_CellDistributionScratchBytes(uint_fast32_t N, uint_fast32_t CN) {
    (void)N;
    const size_t cells = (size_t)CN + 1;                 // + tail bin for out-of-grid keys
    const size_t nb = (cells + 4095) / 4096;
    return (3 * cells + nb) * sizeof(uint32_t) + 256;
}

rf_status md_CellDistribution(const float* R, uint_fast32_t N, uint_fast32_t* CI, uint_fast32_t* CIs,
                              uint_fast32_t* pnC, uint_fast32_t CN, float _1d_a, rf_uint3 cN, void* scratch,
                              size_t scratch_bytes, rf_stream stream) {
    if (!R || !CI || !CIs || !pnC || N == 0 || CN == 0 || !scratch) {
        set_error("md_CellDistribution: bad arguments");
        return RF_ERR_INVALID;
    }
    if (scratch_bytes < md_CellDistributionScratchBytes(N, CN)) {
        set_error("md_CellDistribution: scratch too small (%zu < %zu)", scratch_bytes,
                  md_CellDistributionScratchBytes(N, CN));
        return RF_ERR_INVALID;
    }
    if ((uint64_t)cN.x * cN.y * cN.z != (uint64_t)CN) { set_error("md_CellDistribution: CN != Nr.x*Nr.y*Nr.z"); return RF_ERR_INVALID; }
    cudaStream_t s = S(stream);
    const size_t cells = (size_t)CN + 1, nb = (cells + 4095) / 4096;
    uint32_t* counts = (uint32_t*)scratch;
    uint32_t* start = counts + cells;
    uint32_t* fill = start + cells;
    uint32_t* bsum = fill + cells;
    RefGrid g = make_grid(0.f, _1d_a, cN, CN);
    RF_CUDA(cudaMemsetAsync(counts, 0, cells * sizeof(uint32_t), s));
    RF_CUDA(cudaMemsetAsync(fill, 0, cells * sizeof(uint32_t), s));
    k_cell_index<<<grid_for(N, 256), 256, 0, s>>>(R, N, CI, g, counts, status_word());
    k_scan_block_sums<<<(unsigned)nb, 1024, 0, s>>>(counts, cells, bsum);
    k_scan_totals<<<1, 32, 0, s>>>(bsum, nb);
    k_scan_apply<<<(unsigned)nb, 1024, 0, s>>>(counts, cells, bsum, start);
    k_cell_scatter<<<grid_for(N, 256), 256, 0, s>>>(CI, N, CN, start, fill, CIs);
    k_cell_finish<<<row_grid(cells, 128), 128, 0, s>>>(CI, N, CN, counts, start, CIs, pnC);
    k_cell_last_run<<<1, 32, 0, s>>>(N, CN, CIs, pnC);
    RF_CHECK_LAUNCH("md_CellDistribution");
    return take_status(s);
}

rf_status md_InteractionListConstruct(const float* R, uint_fast32_t N, const uint_fast32_t* CIs,
                                      const uint_fast32_t* pnC, uint_fast32_t* IL, uint_fast32_t K, float a,
                                      float _1d_a, float aacut, rf_uint3 cN, uint_fast32_t CN, rf_stream stream) {
    if (!R || !CIs || !pnC || !IL || N == 0 || K == 0) { set_error("md_InteractionListConstruct: bad arguments"); return RF_ERR_INVALID; }
    cudaStream_t s = S(stream);
    RF_CUDA(cudaMemsetAsync(IL, 0xFF, (size_t)N * K * sizeof(uint_fast32_t), s));
    k_list_construct<<<row_grid(N, LIST_PARTICLES), 128, 0, s>>>(R, N, CIs, pnC, IL, (uint32_t)K, make_grid(a, _1d_a, cN, CN),
                                                     aacut, status_word());
    RF_CHECK_LAUNCH("k_list_construct");
    return take_status(s);
}

rf_status md_InteractionListReConstructBPM(const float* R, uint_fast32_t N, const uint_fast32_t* CIs,
                                           const uint_fast32_t* pnC, uint_fast32_t* IL, uint8_t* ILtype,
                                           uint_fast32_t K, float a, float _1d_a, float aacut, rf_uint3 cN,
                                           uint_fast32_t CN, rf_stream stream) {
    if (!R || !CIs || !pnC || !IL || !ILtype || N == 0 || K == 0) {
        set_error("md_InteractionListReConstructBPM: bad arguments");
        return RF_ERR_INVALID;
    }
    cudaStream_t s = S(stream);
    const size_t stage = K <= LIST_STAGE_K ? (size_t)LIST_PARTICLES * (((K + 3) / 4) | 1u) * sizeof(uint4) : 0;
    k_list_reconstruct_bpm<<<row_grid(N, LIST_PARTICLES), 128, stage, s>>>(R, N, CIs, pnC, IL, ILtype, (uint32_t)K,
                                                            make_grid(a, _1d_a, cN, CN), aacut, status_word());
    RF_CHECK_LAUNCH("k_list_reconstruct_bpm");
    return take_status(s);
}

rf_status md_DeleteFarLinks(const float* R, uint_fast32_t N, uint_fast32_t* IL, uint8_t* ILtype, float* _1d_iL,
                            rf_float3* Rij, rf_float3* Oijt, rf_float3* Fijn, rf_float3* Fijt, rf_float3* Mijn,
                            rf_float3* Mijt, rf_float3* Mijadd, uint_fast32_t K, float aacut, rf_stream stream) {
    (void)_1d_iL;
    if (!R || !IL || !ILtype || !Rij || !Oijt || !Fijn || !Fijt || !Mijn || !Mijt || !Mijadd || N == 0 || K == 0) {
        set_error("md_DeleteFarLinks: bad arguments");
        return RF_ERR_INVALID;
    }
    k_delete_far_links<<<row_grid(N, ROW_CTA), 128, 0, S(stream)>>>(R, N, IL, ILtype, Rij, Oijt, Fijn, Fijt, Mijn, Mijt,
                                                               Mijadd, (uint32_t)K, aacut);
    RF_CHECK_LAUNCH("k_delete_far_links");
    return RF_OK;
}

rf_status md_ConstructBoundInteractions(const float* R, const float* V, const float* W, const uint_fast32_t* IL,
                                        uint8_t* ILtype, float* _1d_iL, rf_float3* Rij, rf_float3* Oijt,
                                        rf_float3* Fijn, rf_float3* Fijt, rf_float3* Mijn, rf_float3* Mijt,
                                        rf_float3* Mijadd, uint_fast32_t N, uint_fast32_t K, float aa_create,
                                        float b_r, rf_stream stream) {
    (void)V; (void)W; (void)b_r;
    if (!R || !IL || !ILtype || !_1d_iL || !Rij || !Oijt || !Fijn || !Fijt || !Mijn || !Mijt || !Mijadd || N == 0 || K == 0) {
        set_error("md_ConstructBoundInteractions: bad arguments");
        return RF_ERR_INVALID;
    }
    k_construct_bonds<<<row_grid(N, ROW_CTA), 128, 0, S(stream)>>>(R, N, IL, ILtype, _1d_iL, Rij, Oijt, Fijn, Fijt, Mijn,
                                                              Mijt, Mijadd, (uint32_t)K, aa_create);
    RF_CHECK_LAUNCH("k_construct_bonds");
    return RF_OK;
}

rf_status md_CalculateForcesDEM_22(const float* R, const float* V, const float* W, const uint_fast32_t* IL,
                                   uint8_t* ILtype, const float* _1d_iL, rf_float3* Rij, rf_float3* Oijt,
                                   rf_float3* Mijn, rf_float3* Mijt, float* F, float* M, uint_fast32_t N,
                                   uint_fast32_t K, float dt, float m_E, float m_G, float b_r, float m_Gcritn,
                                   float m_Gcritt, rf_stream stream) {
    if (!R || !V || !W || !IL || !ILtype || !_1d_iL || !Rij || !Oijt || !Mijn || !Mijt || !F || !M || N == 0 || K == 0) {
        set_error("md_CalculateForcesDEM_22: bad arguments");
        return RF_ERR_INVALID;
    }
    BondParams p{dt, m_E, m_G, b_r, m_Gcritn, m_Gcritt};
    k_row_forces<true><<<row_grid(N, ROW_CTA), 128, 0, S(stream)>>>(R, V, W, IL, ILtype, _1d_iL, Rij, Oijt, Mijn, Mijt, F, M,
                                                                    N, (uint32_t)K, p);
    RF_CHECK_LAUNCH("k_row_forces (bonds)");
    return RF_OK;
}

rf_status md_CalculateForcesDEM_21(const float* R, const float* V, const float* W, const uint_fast32_t* IL,
                                   uint8_t* ILtype, const float* _1d_iL, rf_float3* Rij, rf_float3* Oijt, float* F,
                                   float* M, uint_fast32_t N, uint_fast32_t K, float dt, float m_E, float m_G,
                                   float p_A, float m_mu, float m_muroll, float mP, float rP, rf_stream stream) {
    (void)_1d_iL; (void)Rij;
    if (!R || !V || !W || !IL || !ILtype || !Oijt || !F || !M || N == 0 || K == 0) {
        set_error("md_CalculateForcesDEM_21: bad arguments");
        return RF_ERR_INVALID;
    }
    ContactParams p{dt, m_E, m_G, p_A, m_mu, m_muroll, mP, rP};
    k_row_forces<false><<<row_grid(N, ROW_CTA), 128, 0, S(stream)>>>(R, V, W, IL, (uint8_t*)ILtype, nullptr, nullptr, Oijt,
                                                                     nullptr, nullptr, F, M, N, (uint32_t)K, p);
    RF_CHECK_LAUNCH("k_row_forces (contacts)");
    return RF_OK;
}

rf_status md_CalculateIncrementsDEM(const float* F, float* V, float* R, const float* M, float* W, uint_fast32_t N,
                                    float _1d_Mass_m_dt, float dt, float _1d_I_m_dt, rf_stream stream) {
    if (!F || !V || !R || !M || !W || N == 0) { set_error("md_CalculateIncrementsDEM: bad arguments"); return RF_ERR_INVALID; }
    k_increments<<<grid_for(N, 256), 256, 0, S(stream)>>>(F, V, R, M, W, N, _1d_Mass_m_dt, dt, _1d_I_m_dt);
    RF_CHECK_LAUNCH("k_increments");
    return RF_OK;
}

rf_status md_braziltest_simple2(float* R, float* V, float* F, float* FL, uint_fast32_t N, rf_float3 c, float RR,
                                float Yt, float Yb, float Ytr, float Ybr, float vt, float Zcut, uint64_t nblocks,
                                rf_stream stream) {
    if (!R || !V || !F || !FL || N == 0 || nblocks == 0) { set_error("md_braziltest_simple2: bad arguments"); return RF_ERR_INVALID; }
    cudaStream_t s = S(stream);
    const int g = (int)(nblocks < 148 * 4 ? nblocks : 148 * 4);
    RF_CUDA(cudaMemsetAsync(FL, 0, 2 * nblocks * sizeof(float), s));
    k_brazil<<<g, 256, 0, s>>>(R, V, F, FL, N, c, RR, Yt, Yb, Ytr, Ybr, vt, Zcut, nblocks);
    RF_CHECK_LAUNCH("k_brazil");
    return RF_OK;
}

rf_status md_UniaxialCompression3_simple(float* R, float* V, float* F, float* FL, uint_fast32_t N, rf_float3 c,
                                         float RR, float Zt, float Zb, float Ztr, float Zbr, float vt, float Zcut,
                                         uint64_t nblocks, rf_stream stream) {
    if (!R || !V || !F || !FL || N == 0 || nblocks == 0) {
        set_error("md_UniaxialCompression3_simple: bad arguments");
        return RF_ERR_INVALID;
    }
    cudaStream_t s = S(stream);
    const int g = (int)(nblocks < 148 * 4 ? nblocks : 148 * 4);
    RF_CUDA(cudaMemsetAsync(FL, 0, 2 * nblocks * sizeof(float), s));
    k_uniaxial<<<g, 256, 0, s>>>(R, V, F, FL, N, c, RR, Zt, Zb, Ztr, Zbr, vt, Zcut, nblocks);
    RF_CHECK_LAUNCH("k_uniaxial");
    return RF_OK;
}

rf_status md_ParallelepipedCutRestriction(float* R, float* V, float* F, uint_fast32_t N, rf_float3 center,
                                          rf_float3 sized2, rf_float3 hp, rf_stream stream) {
    if (!R || !V || !F || N == 0) { set_error("md_ParallelepipedCutRestriction: bad arguments"); return RF_ERR_INVALID; }
    k_cut<<<grid_for(N, 256), 256, 0, S(stream)>>>(R, V, F, N, center, sized2, hp);
    RF_CHECK_LAUNCH("k_cut");
    return RF_OK;
}

rf_status md_CalculateIncrementsFIRE(const float* F, float* V, float* R, uint_fast32_t N, float _1d_Mass_m_dt, float dt,
                                     float F_alpha, rf_stream stream) {
    if (!F || !V || !R || N == 0) { set_error("md_CalculateIncrementsFIRE: bad arguments"); return RF_ERR_INVALID; }
    k_fire_inc<<<grid_for(N, 256), 256, 0, S(stream)>>>(F, V, R, N, _1d_Mass_m_dt, dt, F_alpha);
    RF_CHECK_LAUNCH("k_fire_inc");
    return RF_OK;
}

rf_status md_CalculateDecrementsHalfStepFIRE(const float* V, float* R, uint_fast32_t N, float dt_d2, rf_stream stream) {
    if (!V || !R || N == 0) { set_error("md_CalculateDecrementsHalfStepFIRE: bad arguments"); return RF_ERR_INVALID; }
    k_fire_half<<<grid_for(3 * (size_t)N, 256), 256, 0, S(stream)>>>(V, R, N, dt_d2);
    RF_CHECK_LAUNCH("k_fire_half");
    return RF_OK;
}

rf_status md_FdotVEntire(const float* V, const float* F, double* FdotV, uint64_t nblocks, uint_fast32_t N,
                         rf_stream stream) {
    if (!V || !F || !FdotV || N == 0 || nblocks == 0) { set_error("md_FdotVEntire: bad arguments"); return RF_ERR_INVALID; }
    const int g = (int)(nblocks < 148 * 8 ? nblocks : 148 * 8);
    cudaStream_t s = S(stream);
    RF_CUDA(cudaMemsetAsync(FdotV, 0, nblocks * sizeof(double), s));
    k_fdotv<<<g, 256, 0, s>>>(V, F, N, FdotV);
    RF_CHECK_LAUNCH("k_fdotv");
    return RF_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Cell binning without any allocation.
//
// Some callers cannot allocate device memory at the point where they bin: a host
// framework that owns every device byte through its own allocator and forbids other
// allocations, or a plugin handed only its input and output buffers.
// md_CellDistribution needs caller-provided scratch; md_CellDistributionNoAlloc
// instead uses the file-scope device array below as its scratch, so it allocates
// nothing. The array is fixed in size (cell grids of up to RF_NOALLOC_MAX_CELLS - 1
// cells, about 6.3 MB) and every GPU that loads this library holds it until the
// process exits. Like the other md_* entry points, a call returns only once its work
// on the stream has finished: it reads the device status word back.
// ---------------------------------------------------------------------------
#define RF_NOALLOC_MAX_CELLS (1u << 19)   /* cells + the out-of-grid tail bin */
#define RF_NOALLOC_WORDS (3u * RF_NOALLOC_MAX_CELLS + 256u)
static __device__ __align__(256) uint32_t g_noalloc_scratch[RF_NOALLOC_WORDS];

namespace rf {
namespace {
// Device address of g_noalloc_scratch per device. In host code the symbol name is
// only a host-side stand-in, so the address comes from cudaGetSymbolAddress, once
// per device, with that device current. The address belongs to the context it was
// taken in: after a cudaDeviceReset the array lives at a new address in the new
// context, so the lookup is redone when the context id differs from the cached one.
const int kMaxDevices = 64;
uint32_t* g_noalloc_ptr[kMaxDevices] = {nullptr};
unsigned long long g_noalloc_ctx[kMaxDevices] = {0};
std::mutex g_noalloc_mu;

rf_status noalloc_scratch(uint32_t** out) {
    int dev = 0;
    RF_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) { set_error("md_CellDistributionNoAlloc: device %d out of range", dev); return RF_ERR_INVALID; }
    unsigned long long id = 0;
    rf_status st = current_context_id(dev, &id);
    if (st) return st;
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (!g_noalloc_ptr[dev] || g_noalloc_ctx[dev] != id) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) return cuda_status(e, "md_CellDistributionNoAlloc: cudaGetSymbolAddress");
        g_noalloc_ptr[dev] = (uint32_t*)p;
        g_noalloc_ctx[dev] = id;
    }
    *out = g_noalloc_ptr[dev];
    return RF_OK;
}
}  // namespace
}  // namespace rf

extern "C" rf_status md_CellDistributionNoAlloc(const float* R, uint_fast32_t N, uint_fast32_t* CI,
                                                uint_fast32_t* CIs, uint_fast32_t* pnC, uint_fast32_t CN,
                                                float _1d_a, rf_uint3 cN, rf_stream stream) {
    if (!R || !CI || !CIs || !pnC || N == 0 || CN == 0) {
        set_error("md_CellDistributionNoAlloc: bad arguments");
        return RF_ERR_INVALID;
    }
    if ((uint64_t)cN.x * cN.y * cN.z != (uint64_t)CN) {
        set_error("md_CellDistributionNoAlloc: CN != Nr.x*Nr.y*Nr.z");
        return RF_ERR_INVALID;
    }
    if ((uint64_t)CN + 1 > RF_NOALLOC_MAX_CELLS) {
        set_error("md_CellDistributionNoAlloc: %llu cells exceed the fixed scratch limit of %u cells; "
                  "use md_CellDistribution with caller scratch", (unsigned long long)CN, RF_NOALLOC_MAX_CELLS - 1);
        return RF_ERR_INVALID;
    }
    uint32_t* base = nullptr;
    rf_status st = noalloc_scratch(&base);
    if (st) return st;
    cudaStream_t s = (cudaStream_t)stream;
    const size_t cells = (size_t)CN + 1, nb = (cells + 4095) / 4096;
    uint32_t* counts = base;
    uint32_t* start = counts + cells;
    uint32_t* fill = start + cells;
    uint32_t* bsum = fill + cells;
    uint32_t* status = base + RF_NOALLOC_WORDS - 1;
    RefGrid g = make_grid(0.f, _1d_a, cN, CN);
    // The array keeps the previous call's contents: counters and status start at zero.
    RF_CUDA(cudaMemsetAsync(counts, 0, cells * sizeof(uint32_t), s));
    RF_CUDA(cudaMemsetAsync(fill, 0, cells * sizeof(uint32_t), s));
    RF_CUDA(cudaMemsetAsync(status, 0, sizeof(uint32_t), s));
    k_cell_index<<<grid_for(N, 256), 256, 0, s>>>(R, N, CI, g, counts, status);
    k_scan_block_sums<<<(unsigned)nb, 1024, 0, s>>>(counts, cells, bsum);
    k_scan_totals<<<1, 32, 0, s>>>(bsum, nb);
    k_scan_apply<<<(unsigned)nb, 1024, 0, s>>>(counts, cells, bsum, start);
    k_cell_scatter<<<grid_for(N, 256), 256, 0, s>>>(CI, N, CN, start, fill, CIs);
    k_cell_finish<<<row_grid(cells, 128), 128, 0, s>>>(CI, N, CN, counts, start, CIs, pnC);
    k_cell_last_run<<<1, 32, 0, s>>>(N, CN, CIs, pnC);
    RF_CHECK_LAUNCH("md_CellDistributionNoAlloc");
    uint32_t h = 0;
    RF_CUDA(cudaMemcpyAsync(&h, status, sizeof(h), cudaMemcpyDeviceToHost, s));
    RF_CUDA(cudaStreamSynchronize(s));
    if (h) {
        set_error("md_CellDistributionNoAlloc: device status %u", h);
        return (rf_status)h;
    }
    return RF_OK;
}
