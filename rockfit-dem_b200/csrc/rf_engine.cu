// Fused B200 engine for the explicit BPM test loop.
//
// One explicit step of the reference (md_calculationbraziltest.cu:170-190:
// CellDistribution, InteractionListReConstructBPM, F=M=0, _22, _21, platen,
// SumForcesULoading, increments, cut, DeleteFarLinks, CompressB/U) is ONE kernel
// here, a warp taking 32 particles, or fewer where they would not fill the GPU:
//
//   delete  -- DeleteFarLinks of the previous step, with this step's positions
//              (the reference runs it at the end of the previous step on the same
//              positions, so the result is identical);
//   add     -- new neighbours inside a_farcut, taken from a Verlet candidate list
//              (cutoff a_farcut + skin, rebuilt only when some particle has moved
//              more than 0.3*skin since the last build) instead of re-binning every
//              step. New links are inserted in the order the reference would insert
//              them: by (octant-cell rank, id), computed from the same float cell
//              arithmetic, into the first free slot;
//   bonds   -- bond slots in slot order (same sums, same rounding as _22);
//   contacts-- contact slots in slot order (as _21), F = (0 + F_bond) + F_contact;
//   platen, increments, cut -- per particle, into the other position buffer;
//   load    -- per-block FP64 partial sums, the last block finishes the scalar
//              step (SumForcesULoading, CompressB/U, fracture, load curve) on device.
//
// Layout in HBM: positions as float4 (x, y, z, 0) or double4 (x, y, z, radius), velocity and
// spin together as one 32-byte record, both double-buffered; row ids row-major [N][K]; the
// bonds' state as 64-byte records, ordinal-major [QB][N], so that lanes taking the q-th bond
// of consecutive particles read consecutive whole sectors; per-particle 32-bit masks for
// occupied slots, bond slots and contacts with non-zero tangential overlap (so empty and
// idle slots cost no state reads).
//
// The step loop is a CUDA graph: WHILE(continue) { IF(rebuild) {bin, scan,
// scatter, candidates}; step }, with both conditions set on device by the step
// kernel, so one graph launch advances many steps without host round trips.
#include <cstdio>
#include <cstring>
#include <fstream>
#include <vector>
#include <algorithm>
#include <utility>
#include <cuda_bf16.h>
#include "rf_physics.cuh"

#ifndef RF_STEP_MIN_BLOCKS
#define RF_STEP_MIN_BLOCKS 6      // resident 128-thread CTAs per SM the step kernel is compiled for
#endif

#ifndef RF_GRAPH_UNROLL
#define RF_GRAPH_UNROLL 8         // explicit steps per iteration of the graph's WHILE loop
#endif
// outcome of one bond record, handed by the lane that evaluated it to its particle's lane
// (bits 8-12: the record's row slot)
// margin buckets of the candidate lists: a candidate's margin (distance - list cutoff at
// the build) below RF_CB1, RF_CB2, RF_CB3 skins, or above
#define RF_CB1 0.05f
#define RF_CB2 0.15f
#define RF_CB3 0.3f
#define RF_REC_DELETE 1u          // beyond the bond's keep distance: the slot is deleted
#define RF_REC_BROKE 2u           // the bond broke this step
#define RF_REC_PARALLEL 4u        // the pair overlaps: the slot's contact was taken with the bond
#define RF_REC_CLEAR 8u           // that contact's zero-spin rule cleared the particle's moment sum
#ifndef RF_REBUILD_EACH_STEP_N
#define RF_REBUILD_EACH_STEP_N (1u << 20)   // from this many particles the rebuild condition is evaluated every step
#endif

namespace rf {

// Scalar state of the run, device resident (compression_data + result bookkeeping).
struct DevScalars {
    double V, VLoad, Top, Bottom, TopR, BottomR, FractureStress, FractureStrain, MinStress, ZeroStress, Stress,
        Strain, MaxStrain, Size0;
    double size_d[3], center_d[3];
    double sz0;
    double keep_frac;       // post-peak stop: fracture once Stress < keep_frac * peak (0: off)
    float center[3], size[3], sized2[3];
    float RR, _1d_Area, Hd2;
    int32_t Loading, Fracture;
    unsigned long long steps, target, rebuilds, curve_n, broken;
    uint32_t done, err, rebuild, moved, block_counter, spec_counter;
    // largest displacement since the last candidate build of the positions a step reads
    // (FP32 bits of its square, accumulated by the step writing them), for skipping scans
    uint32_t d2max_next;
    float dmax;
    // FIRE relaxation of a quasi-static load increment (extended model)
    double fdt, falpha, fdt0, fdtmax, fdtmin, finc, fdec, falpha0, fshrink, ftol;
    double fresidual, fmean, fpower, fcv, fcf, fcm;
    unsigned long long fiter, fmax_iter, fnpos, fiter_total;
    uint32_t fndelay, fuphill, fconverged, fstop, fcounter, fwarm;
};

struct Consts {
    uint32_t N, K, KC;
    int kind;
    double dt_d, p_r_d;
    BondParams bp;
    ContactParams cp;
    float dtm, dt, dtI;
    float aacut, aa_farcut;
    RefGrid g;
    float zcut;
    rf_float3 box_c, box_h, hp;
    // candidate grid
    float cg_inv_h;
    float cg_ox, cg_oy, cg_oz;
    uint32_t cg_nx, cg_ny, cg_nz, cg_cells;
    float rc2, disp2, hard2;   // rebuild trigger and the displacement the candidate lists cover
    float acut_f;              // sqrt(aacut)
    unsigned long long curve_cap;
    cudaGraphConditionalHandle h_loop, h_rebuild;
    int use_graph;
    int fire_skip;             // FIRE loop: the kernels of the body's later iterations leave if a rebuild is due
    // extended model (ext != 0): FP64 positions with radii, per-bond strengths
    int ext;
    ExtParams ep;
    float kn, ks, br_lambda, cmass;     // bond stiffness per area, bond radius / min(r_i, r_j), mass = cmass r^3
    double aa_farcut_d, aacut_d;
    // list rule: lgap_d == 0 lists pairs within a_farcut (add test on the float aacut,
    // delete test on aa_farcut, as the reference); lgap_d > 0 within min(a_farcut, r_i + r_j + g)
    double a_farcut_d, lgap_d;
    float lgap_f, skin_f;
    // reference constants in the extended model (rf_ext_params.ref_mode): per-bond stiffness
    // E/L0, G/L0 from the record's 1/L0, bond radius b_r, the Q1 bending factor, platen
    // coordinates rounded to float as the reference's drivers pass them
    int ref_mode;
    float refE, refG, ref_br;
};

// Per-specimen geometry of a batch (constant during a run): the platen's cut height, the
// cut box and its hidden point, the specimen's particle range.
struct SpecGeom {
    float zcut;
    rf_float3 box_c, box_h, hp;
    uint32_t p0, p1;
};

struct __align__(32) F8 { float4 a, b; };
struct __align__(32) Rec { float4 s0, s1, s2, k; };     // k: (L0 as a double, tensile, shear strength) or (1/L0, 0, 0, 0)

struct Dev {
    // batch of specimens (one specimen: spec == sc, geom[0], blk_spec == nullptr)
    DevScalars* spec;           // [nspec] per-specimen platen / result scalars
    const SpecGeom* geom;       // [nspec]
    const uint16_t* blk_spec;   // [N / 128] specimen of the first of every 128 particles
    double2* partial2;          // [CTAs] load partials of a CTA's second specimen
    uint32_t *nz, *nz2;         // [CTAs / 32] CTAs whose partial / partial2 was written this step
    uint32_t nspec;
    double4* posd[2];   // extended model: x, y, z (FP64) and radius
    float4* pos[2];
    F8* vw[2];          // [N] velocity and spin of a particle (xyz 0 each): one 32-byte sector, one load
    // rows: K slots per particle
    uint32_t* ids;      // [N][K] neighbour id of each occupied slot (row-major: a thread walks its own row)
    float* il;          // [K][N] 1/L0 per slot, as the reference layout keeps it (read out only)
    float* cO[2];       // [N][K][3] tangential overlap of type-0 slots, by step parity (read cur, write next)
    uint32_t* live;     // [N] occupied slots
    uint32_t* bond;     // [N] slots holding an intact bond
    uint32_t* cmask;    // [N] type-0 slots whose overlap may be non-zero
    // bond records: the bonds of particle i in slot order, ordinal-major [q][i]. A record is 64
    // bytes, (Rij.xyz Oijt.x) (Oijt.yz Mijn.xy) (Mijn.z Mijt.xyz) and what does not change: the
    // FP64 rest length and the two strengths, or 1/L0 in the reference model. It is read and
    // written as two whole 32-byte pieces: records of broken bonds in between cost nothing, and
    // no sector is written in part.
    Rec* rec;           // [QB][N]
    Rec* rec0;          // rec at the start of the current quasi-static increment (FIRE mode)
    uint2* bjk;         // [QB][N] partner id and slot of the record (slot 0xFF: record retired)
    uint32_t* nbq;      // [N] records of the particle
    uint32_t* bmask;    // [N] records holding an intact bond
    // Verlet candidates
    uint32_t* cand;     // [KC][N]
    uint32_t* cand_n;   // [N]
    unsigned long long* member;   // [N]
    float4* pos_ref;    // [N]
    float* cmargin;     // [N] smallest (distance - a_farcut) of the non-member candidates at the build
    uint32_t* cbound;   // [N] ends of the candidates' margin buckets (bytes 0-2, see k_rb_cand)
    uint32_t* cg_key;   // [N]
    uint32_t* cg_count; // [cells+1]
    uint32_t* cg_start; // [cells+1]
    uint32_t* cg_fill;  // [cells+1]
    uint32_t* cg_bsum;
    uint32_t* cg_sorted;   // [N] particle ids in cell order
    uint32_t* cg_slot;     // [N] place of each particle in that order
    float4* cg_pos;        // [N] positions (x, y, z, radius) in that order
    double2* partial;   // [CTAs] load partials (extended model: where the CTA has any, see nz)
    // FIRE relaxation (allocated on first use)
    float4* frc;        // [N] net force after the platen clamp
    float4* mom;        // [N] net moment
    double* fpart;      // [CTAs][FIRE_SUMS] FP64 partial sums (of a CTA's first specimen)
    double* fpart2;     // [CTAs][FIRE_SUMS] the same for a CTA's second specimen (batches)
    double* fgrp;       // [groups][FIRE_SUMS] sums over FIRE_GROUP CTAs of a specimen
    uint32_t* fgrp_n;   // [groups] CTAs of the group that have arrived
    double4* rot;       // [N] accumulated rotation of the increment (sum of w dt)
    double* xax;        // [N] coordinate along the load axis that the last force pass read
    double4* x0;        // [N] positions at the start of the increment
    unsigned long long n_particles;
    uint32_t QB;
    double* curve;      // [cap][3]
    DevScalars* sc;
};

__device__ __forceinline__ f3 f4to3(const float4 v) { return mk3(v.x, v.y, v.z); }
// Position of particle j as float4 (x, y, z, radius) in either model.
__device__ __forceinline__ float4 posf(const Dev& d, const Consts& c, uint32_t buf, uint32_t j) {
    if (c.ext) {
        const double4 p = d.posd[buf][j];
        return make_float4((float)p.x, (float)p.y, (float)p.z, (float)p.w);
    }
    return d.pos[buf][j];
}
// 32-byte loads and stores (one instruction each on sm_100).
__device__ __forceinline__ F8 ldg8(const F8* p) {
    F8 v;
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(v.a.x), "=f"(v.a.y), "=f"(v.a.z), "=f"(v.a.w), "=f"(v.b.x), "=f"(v.b.y), "=f"(v.b.z), "=f"(v.b.w)
        : "l"(p));
    return v;
}
__device__ __forceinline__ void ld8(const void* p, float4& a, float4& b) {
    asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
                 : "l"(p)
                 : "memory");
}
__device__ __forceinline__ void st8(void* p, const float4 a, const float4 b) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(a.x), "f"(a.y), "f"(a.z), "f"(a.w),
                 "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w)
                 : "memory");
}
__device__ __forceinline__ double rec_L0(const float4 k) { return __hiloint2double(__float_as_int(k.y), __float_as_int(k.x)); }
__device__ __forceinline__ float4 rec_const(double L0, const float2 str) {
    return make_float4(__int_as_float(__double2loint(L0)), __int_as_float(__double2hiint(L0)), str.x, str.y);
}
__device__ __forceinline__ void zero_record(const Dev& d, size_t s) {     // the state; the constants stay
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    d.rec[s].s0 = z; d.rec[s].s1 = z; d.rec[s].s2 = z;
}

// ---------------------------------------------------------------------------
// Candidate-list rebuild (runs only when the displacement flag is set)
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool gate_closed(const Dev& d, const Consts& c) {
    // In graph mode the IF node gates the rebuild; on a plain stream the kernels check.
    return !c.use_graph && (d.sc->rebuild == 0 || d.sc->done);
}

__device__ __forceinline__ uint32_t cg_cell_of(const float4 x, const Consts& c) {
    const float fx = floorf((x.x - c.cg_ox) * c.cg_inv_h);
    const float fy = floorf((x.y - c.cg_oy) * c.cg_inv_h);
    const float fz = floorf((x.z - c.cg_oz) * c.cg_inv_h);
    if (!(fx >= 0.f && fy >= 0.f && fz >= 0.f)) return 0xFFFFFFFFu;
    const uint32_t ix = (uint32_t)fx, iy = (uint32_t)fy, iz = (uint32_t)fz;
    if (ix >= c.cg_nx || iy >= c.cg_ny || iz >= c.cg_nz) return 0xFFFFFFFFu;
    return ix + c.cg_nx * (iy + c.cg_ny * iz);
}

__global__ void k_rb_zero(Dev d, Consts c) {
    if (gate_closed(d, c)) return;
    for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q <= c.cg_cells; q += gridDim.x * blockDim.x) {
        d.cg_count[q] = 0;
        d.cg_fill[q] = 0;
    }
}

__global__ void k_rb_bin(Dev d, Consts c) {
    if (gate_closed(d, c)) return;
    const uint32_t cur = (uint32_t)(d.sc->steps & 1);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < c.N; i += gridDim.x * blockDim.x) {
        uint32_t key = cg_cell_of(posf(d, c, cur, i), c);
        if (key == 0xFFFFFFFFu) key = c.cg_cells;          // parked or outside: tail bin, no candidates
        d.cg_key[i] = key;
        atomicAdd(&d.cg_count[key], 1u);
    }
}

__global__ void k_rb_scan_sums(Dev d, Consts c) {
    if (gate_closed(d, c)) return;
    __shared__ uint32_t sh[32];
    const size_t n = (size_t)c.cg_cells + 1, base = (size_t)blockIdx.x * 4096;
    uint32_t s = 0;
    for (int t = threadIdx.x; t < 4096; t += blockDim.x)
        if (base + t < n) s += d.cg_count[base + t];
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        uint32_t v = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : 0;
        for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (threadIdx.x == 0) d.cg_bsum[blockIdx.x] = v;
    }
}

__global__ void k_rb_scan_totals(Dev d, Consts c) {
    if (gate_closed(d, c)) return;
    const uint32_t nb = (c.cg_cells + 1 + 4095) / 4096;
    const uint32_t lane = threadIdx.x;             // one warp
    uint32_t acc = 0;
    for (uint32_t b0 = 0; b0 < nb; b0 += 32) {
        const uint32_t v = b0 + lane < nb ? d.cg_bsum[b0 + lane] : 0;
        uint32_t incl = v;
        for (int o = 1; o < 32; o <<= 1) { const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= (uint32_t)o) incl += y; }
        if (b0 + lane < nb) d.cg_bsum[b0 + lane] = acc + incl - v;
        acc += __shfl_sync(0xffffffffu, incl, 31);
    }
}

__global__ void k_rb_scan_apply(Dev d, Consts c) {
    if (gate_closed(d, c)) return;
    __shared__ uint32_t wsum[32];
    const size_t n = (size_t)c.cg_cells + 1;
    const size_t base = (size_t)blockIdx.x * 4096 + (size_t)threadIdx.x * 4;
    uint32_t v[4], t = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) { v[q] = (base + q < n) ? d.cg_count[base + q] : 0; t += v[q]; }
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
    uint32_t run = d.cg_bsum[blockIdx.x] + wsum[w] + incl - t;
#pragma unroll
    for (int q = 0; q < 4; ++q) { if (base + q < n) d.cg_start[base + q] = run; run += v[q]; }
}

__global__ void k_rb_scatter(Dev d, Consts c) {
    if (gate_closed(d, c)) return;
    const uint32_t cur = (uint32_t)(d.sc->steps & 1);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < c.N; i += gridDim.x * blockDim.x) {
        const uint32_t key = d.cg_key[i];
        const uint32_t s = d.cg_start[key] + atomicAdd(&d.cg_fill[key], 1u);
        d.cg_sorted[s] = i;
        d.cg_slot[i] = s;
        d.cg_pos[s] = posf(d, c, cur, i);
    }
}

// Candidates: every j != i within rc of i (27 cells), in the order of their margin bucket (a
// scan needs no candidate of a bucket whose lower bound the displacements since this build
// cannot have closed, see scan_limit), which of them sit in i's row, and the margin of the
// nearest that does not. Positions are read in cell order (three x-neighbouring cells are one
// run of float4 records, nine runs a particle). A particle first only collects, in shared memory,
// the places of its candidates in that order (what else a candidate needs would be run by the
// whole warp for each of its lanes' hits in turn); the buckets and the row's members, found by
// their places, follow. A build of 4M particles takes 2.2 ms (2.03 of it this kernel), 3.0 with
// an id and a position gathered for every occupant and the list ordered and matched in memory.
#define RF_RB_CTA 128
__global__ void __launch_bounds__(RF_RB_CTA) k_rb_cand(Dev d, Consts c) {
    if (gate_closed(d, c)) return;
    __shared__ uint32_t s_c[64][RF_RB_CTA];
    const uint32_t tid = threadIdx.x, mine = blockIdx.x * RF_RB_CTA + tid;
    if (mine < c.N) {
        const uint32_t i = d.cg_sorted[mine], key = d.cg_key[i];
        const float4 xi = d.cg_pos[mine];
        d.pos_ref[i] = xi;
        auto cut_of = [&](const float4 xj) { return c.lgap_f > 0.f ? fminf(c.acut_f, (xi.w + xj.w) + c.lgap_f) : c.acut_f; };
        uint32_t n = 0;
        if (key < c.cg_cells) {
            const int ix = key % c.cg_nx, iy = (key / c.cg_nx) % c.cg_ny, iz = key / (c.cg_nx * c.cg_ny);
            const uint32_t xa = ix > 0 ? ix - 1 : 0, xb = ix + 1 < (int)c.cg_nx ? ix + 1 : ix;
            for (int z = max(iz - 1, 0); z <= min(iz + 1, (int)c.cg_nz - 1); ++z) {
                for (int y = max(iy - 1, 0); y <= min(iy + 1, (int)c.cg_ny - 1); ++y) {
                    const uint32_t line = c.cg_nx * (y + c.cg_ny * z);
                    const uint32_t e = d.cg_start[line + xb + 1];
#pragma unroll 4
                    for (uint32_t q = d.cg_start[line + xa]; q < e; ++q) {
                        const float4 xj = __ldg(&d.cg_pos[q]);
                        const float ddx = xj.x - xi.x, ddy = xj.y - xi.y, ddz = xj.z - xi.z;
                        const float d2 = ddx * ddx + ddy * ddy + ddz * ddz;
                        // (with one cutoff for all, reach is rc up to rounding: rc2 alone decides)
                        const float reach = c.lgap_f > 0.f ? fminf(c.acut_f, (xi.w + xj.w) + c.lgap_f) + c.skin_f : 3.0e18f;
                        if (!(d2 < c.rc2) || !(d2 < reach * reach) || q == mine) continue;
                        if (n < c.KC) s_c[n++][tid] = q;
                        else raise_status(&d.sc->err, RF_ERR_CAPACITY);
                    }
                }
            }
        }
        unsigned long long k0 = 0ull, k1 = 0ull;           // bits 0 and 1 of the candidates' buckets
#pragma unroll 4
        for (uint32_t q = 0; q < n; ++q) {
            const float4 xj = __ldg(&d.cg_pos[s_c[q][tid]]);
            const float ddx = xj.x - xi.x, ddy = xj.y - xi.y, ddz = xj.z - xi.z;
            const float mg = sqrtf(ddx * ddx + ddy * ddy + ddz * ddz) - cut_of(xj);
            const uint32_t b = mg < RF_CB1 * c.skin_f ? 0u : mg < RF_CB2 * c.skin_f ? 1u : mg < RF_CB3 * c.skin_f ? 2u : 3u;
            k0 |= (unsigned long long)(b & 1u) << q;
            k1 |= (unsigned long long)(b >> 1) << q;
        }
        d.cand_n[i] = n;
        unsigned long long in_row = 0ull;                  // candidates already in the row
        uint32_t live = d.live[i];
        while (live) {
            const uint32_t k = __ffs(live) - 1;
            live &= live - 1;
            const uint32_t sj = d.cg_slot[d.ids[(size_t)i * c.K + k]];
            for (uint32_t q = 0; q < n; ++q)
                if (s_c[q][tid] == sj) { in_row |= 1ull << q; break; }
        }
        const unsigned long long all = n < 64 ? (1ull << n) - 1ull : ~0ull;
        const uint32_t n0 = __popcll(~k1 & ~k0 & all), n1 = n0 + __popcll(~k1 & k0 & all), n2 = n1 + __popcll(k1 & ~k0);
        d.cbound[i] = n0 | (n1 << 8) | (n2 << 16);
        uint32_t next = (n0 << 8) | (n1 << 16) | (n2 << 24);   // next place of each bucket (bytes; at most 64)
        unsigned long long mem = 0ull;
        // margin of the nearest non-member candidate: until the displacements since this
        // build add up to it, no candidate can come within its list cutoff
        float mg = 3.0e38f;
        for (uint32_t q = 0; q < n; ++q) {
            const uint32_t sh = 8u * ((uint32_t)((k0 >> q) & 1ull) + 2u * (uint32_t)((k1 >> q) & 1ull));
            const uint32_t at = (next >> sh) & 0xFFu, s = s_c[q][tid];
            next += 1u << sh;
            d.cand[(size_t)at * c.N + i] = d.cg_sorted[s];
            if ((in_row >> q) & 1ull) { mem |= 1ull << at; continue; }
            const float4 xj = __ldg(&d.cg_pos[s]);
            const float ddx = xj.x - xi.x, ddy = xj.y - xi.y, ddz = xj.z - xi.z;
            mg = fminf(mg, sqrtf(ddx * ddx + ddy * ddy + ddz * ddz) - cut_of(xj));
        }
        d.member[i] = mem;
        d.cmargin[i] = mg;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        atomicAdd(&d.sc->rebuilds, 1ull);
        d.sc->dmax = 0.f;                     // positions == build positions
    }
}

// ---------------------------------------------------------------------------
// The step kernel
// ---------------------------------------------------------------------------
// Retire the bond record of slot k of particle i, if it has one: its state is
// zeroed (DeleteFarLinks zeroes Rij, Oijt, Mijn, Mijt of the slot) and it stops
// belonging to the slot.
__device__ __forceinline__ void retire_record(const Dev& d, const Consts& c, uint32_t i, uint32_t k, uint32_t nbq,
                                              uint32_t& bmask) {
    const uint32_t N = c.N;
    for (uint32_t q = 0; q < nbq; ++q) {
        const size_t s = (size_t)q * N + i;
        if (d.bjk[s].y == k) {
            d.bjk[s].y = 0xFFu;
            zero_record(d, s);
            bmask &= ~(1u << q);
            return;
        }
    }
}

// DeleteFarLinks (md_interaction_list_reconstructbpm.cu:141-186) of one slot.
__device__ __forceinline__ void delete_slot(const Dev& d, const Consts& c, uint32_t i, uint32_t k, uint32_t j,
                                            uint32_t ncand, uint32_t nbq, uint32_t& live, uint32_t& bond, uint32_t& cm,
                                            uint32_t& bmask, unsigned long long& mem) {
    const uint32_t N = c.N;
    const size_t s = (size_t)i * c.K + k;
    d.ids[s] = EMPTY32;                       // its overlap reads as zero once the cmask bit is clear
    d.cmargin[i] = 0.f;                       // the deleted partner may come back: scan until the next build
    retire_record(d, c, i, k, nbq, bmask);
    const uint32_t bit = 1u << k;
    live &= ~bit; bond &= ~bit; cm &= ~bit;
    for (uint32_t q = 0; q < ncand; ++q)
        if (d.cand[(size_t)q * N + i] == j) { mem &= ~(1ull << q); break; }
}

// DeleteFarLinks for every occupied slot of particle i with the current positions.
__device__ __forceinline__ void delete_far(const Dev& d, const Consts& c, const float4* __restrict__ P, uint32_t i,
                                           const f3 xi, uint32_t ncand, uint32_t nbq, uint32_t& live, uint32_t& bond,
                                           uint32_t& cm, uint32_t& bmask, unsigned long long& mem) {
    const uint32_t* row = d.ids + (size_t)i * c.K;
    uint32_t m = live;
    while (m) {
        const uint32_t k = __ffs(m) - 1;
        m &= m - 1;
        const uint32_t j = row[k];
        const float rr = dist2_rn(xi, f4to3(__ldg(&P[j])));
        if (rr > c.aa_farcut || (double)rr < 1e-10) delete_slot(d, c, i, k, j, ncand, nbq, live, bond, cm, bmask, mem);
    }
}

// How many of particle i's candidates (in bucket order) the add pass must test, of n.
// None when the scan cannot find anything: every non-member candidate was at least cmargin
// beyond a_farcut at the last build, and since then this particle moved by |x - x_build| and
// none by more than dmax (the largest displacement of the positions this step reads). 10 % and
// 1e-4 a_farcut of slack cover the float rounding of the margins and displacements. Else those
// of the buckets whose lower bound, by the same test, the displacements can have closed. After
// a deletion (cmargin 0) every candidate is tested. (All loads side by side.)
__device__ __forceinline__ uint32_t scan_limit(const Dev& d, const Consts& c, uint32_t i, float x, float y, float z,
                                               uint32_t n) {
    const float4 pr = d.pos_ref[i];
    const float margin = d.cmargin[i], dmax = d.sc->dmax;
    const uint32_t b = d.cbound[i];
    const float ex = x - pr.x, ey = y - pr.y, ez = z - pr.z;
    const float moved = sqrtf(ex * ex + ey * ey + ez * ez) + dmax;
    if (moved < 0.9f * margin - 1e-4f * c.acut_f) return 0u;
    if (!(margin > 0.f)) return n;
    const float reach = moved + 1e-4f * c.acut_f;
    if (reach < 0.9f * RF_CB1 * c.skin_f) return b & 0xFFu;
    if (reach < 0.9f * RF_CB2 * c.skin_f) return (b >> 8) & 0xFFu;
    if (reach < 0.9f * RF_CB3 * c.skin_f) return (b >> 16) & 0xFFu;
    return n;
}

// The delete pass of the last step, applied before the state is read out: the step
// kernel defers each step's DeleteFarLinks to the start of the next step (same
// positions), so a snapshot taken between steps applies it first. Idempotent.
__global__ void k_delete_pending(Dev d, Consts c) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = i < c.N;
    const float4* P = d.pos[d.sc->steps & 1ull];
    f3 xi = mk3(0.f, 0.f, 0.f);
    uint32_t live = 0, bond = 0, cm = 0, ncand = 0, nbq = 0, bmask = 0;
    unsigned long long mem = 0ull;
    if (valid) {
        xi = f4to3(P[i]);
        live = d.live[i]; bond = d.bond[i]; cm = d.cmask[i]; mem = d.member[i]; ncand = d.cand_n[i];
        nbq = d.nbq[i]; bmask = d.bmask[i];
    }
    const uint32_t live0 = live;
    delete_far(d, c, P, i, xi, ncand, nbq, live, bond, cm, bmask, mem);
    if (valid && live != live0) {
        d.live[i] = live; d.bond[i] = bond; d.cmask[i] = cm; d.member[i] = mem; d.bmask[i] = bmask;
    }
}

// ===========================================================================
// Extended model step: FP64 positions (x, y, z, radius), per-particle mass and
// inertia from the radius, bond records with an FP64 rest length and their own
// strengths, contacts with equivalent radius and mass; list maintenance compares FP64
// squared distances. (The reference model's k_step follows below with the same structure.)
// ===========================================================================
// Read-only load of a particle's 32-byte position and radius.
__device__ __forceinline__ double4 ldg_d4(const double4* p) {
    double4 v;
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ double3 dsub(const double4 a, const double4 b) {
    return make_double3(a.x - b.x, a.y - b.y, a.z - b.z);
}
__device__ __forceinline__ double dlen2(const double3 r) { return r.x * r.x + r.y * r.y + r.z * r.z; }

// Squared list cutoffs of a pair of the extended model (radii ri, rj): the add test and
// the delete test. With a list gap g the pair's cutoff is min(a_farcut, ri + rj + g).
__device__ __forceinline__ double cut2_add(const Consts& c, double ri, double rj) {
    if (c.lgap_d > 0.0) {
        const double q = fmin(c.a_farcut_d, (ri + rj) + c.lgap_d);
        return q * q;
    }
    return c.aacut_d;
}
__device__ __forceinline__ double cut2_del(const Consts& c, double ri, double rj) {
    if (c.lgap_d > 0.0) {
        const double q = fmin(c.a_farcut_d, (ri + rj) + c.lgap_d);
        return q * q;
    }
    return c.aa_farcut_d;
}

// The reference removes a listed pair beyond a_farcut = 2.9 p_r, 1.45 times the contact
// distance 2 p_r of its mono-sized particles, intact bonds included
// (md_interaction_list_reconstructbpm.cu:141-186). With a list gap, or radii that span a
// range, a pair cutoff can lie within a bond's failure stretch (a bond of two r_max
// particles sits just inside a_farcut = 2.02 r_max), so list maintenance would remove
// intact bonds that their strengths still hold. In the extended model an intact bond is
// therefore removed by distance only beyond the same relative margin of its own rest
// length, |r| > 1.45 L0; the reference-constants mode keeps the reference's rule.
#define RF_BOND_KEEP_RATIO 1.45
__device__ __forceinline__ double bond_cut2_del(const Consts& c, double ri, double rj, double L0) {
    if (c.ref_mode) return cut2_del(c, ri, rj);
    const double q = RF_BOND_KEEP_RATIO * L0;
    return q * q;
}
// Rest length of the intact bond in slot k of particle i (its record's).
__device__ __forceinline__ double slot_rest_length(const Dev& d, const Consts& c, uint32_t i, uint32_t k, uint32_t nbq) {
    for (uint32_t q = 0; q < nbq; ++q) {
        const size_t s = (size_t)q * c.N + i;
        if (d.bjk[s].y == k) return rec_L0(d.rec[s].k);
    }
    return 0.0;
}

__device__ __forceinline__ void delete_far_ext(const Dev& d, const Consts& c, const double4* __restrict__ P,
                                               uint32_t i, const double4 xi, uint32_t ncand, uint32_t nbq,
                                               uint32_t& live, uint32_t& bond, uint32_t& cm, uint32_t& bmask,
                                               unsigned long long& mem) {
    const uint32_t* row = d.ids + (size_t)i * c.K;
    uint32_t m = live;
    while (m) {
        const uint32_t k = __ffs(m) - 1;
        m &= m - 1;
        const uint32_t j = row[k];
        const double4 xj = ldg_d4(&P[j]);
        const double rr = dlen2(dsub(xj, xi));
        const double cut = ((bond >> k) & 1u) ? bond_cut2_del(c, xi.w, xj.w, slot_rest_length(d, c, i, k, nbq))
                                              : cut2_del(c, xi.w, xj.w);
        if (rr > cut || rr < 1e-10)
            delete_slot(d, c, i, k, j, ncand, nbq, live, bond, cm, bmask, mem);
    }
}

__global__ void k_delete_pending_ext(Dev d, Consts c) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.N) return;
    const double4* P = d.posd[d.sc->steps & 1ull];
    uint32_t live = d.live[i], bond = d.bond[i], cm = d.cmask[i], ncand = d.cand_n[i], nbq = d.nbq[i],
             bmask = d.bmask[i];
    unsigned long long mem = d.member[i];
    const uint32_t live0 = live;
    delete_far_ext(d, c, P, i, P[i], ncand, nbq, live, bond, cm, bmask, mem);
    if (live != live0) {
        d.live[i] = live; d.bond[i] = bond; d.cmask[i] = cm; d.member[i] = mem; d.bmask[i] = bmask;
    }
}

// Platen contact and clamp with FP64 positions (d_UniaxialCompression3_simple /
// d_braziltest_simple2 with the coordinates kept in double). The platens act on the
// particle surfaces: the coordinate tested and clamped along the load axis is the
// centre plus (radius - p_r) towards the top platen and minus it towards the bottom
// one, so a polydisperse specimen meets a flat platen with every particle that
// touches it; for radius p_r this is the reference's centre rule.
// hold: inside a quasi-static increment's FIRE iterations a particle held by a platen
// does not slide along it either (removes the specimen's rigid tilting and sliding).
__device__ __forceinline__ void uniaxial_particle_ext(double& Rx, double& Ry, double& Rz, float& Vx, float& Vy,
                                                      float& Vz, float& Fx, float& Fy, float& Fz, const rf_float3 c,
                                                      float RR, double Zt, double Zb, double Ztr, double Zbr, float vt,
                                                      double Zcut, double off, double& sfb, double& sft, bool hold) {
    const float rx = (float)(Rx - c.x), ry = (float)(Ry - c.y);
    const double rz = Rz;
    if (rx * rx + ry * ry < RR && rz < Zcut) {
        if (rz + off - Ztr > -1e-9) {
            if (Fz > 0) sft += (double)Fz;
            if (rz + off - Zt > -1e-9) {
                Rz = Zt - off; Vz = vt; Fz = 0.f;
                if (hold) { Fx = 0.f; Fy = 0.f; Vx = 0.f; Vy = 0.f; }
            }
        }
        if (rz - off - Zbr < 1e-9) {
            if (Fz < 0) sfb += (double)Fz;
            if (rz - off - Zb < 1e-9) {
                Rz = Zb + off; Vz = 0.f; Fz = 0.f;
                if (hold) { Fx = 0.f; Fy = 0.f; Vx = 0.f; Vy = 0.f; }
            }
        }
    }
}
__device__ __forceinline__ void brazil_particle_ext(double& Rx, double& Ry, double& Rz, float& Vx, float& Vy,
                                                    float& Vz, float& Fx, float& Fy, float& Fz, const rf_float3 c,
                                                    float RR, double Yt, double Yb, double Ytr, double Ybr, float vt,
                                                    double Zcut, double off, double& sfb, double& sft, bool hold) {
    const float rx = (float)(Rx - c.x), rz = (float)(Rz - c.z);
    const double ry = Ry;
    if (rx * rx + rz * rz < RR && (double)rz < Zcut) {
        if (ry + off - Ytr > -1e-9) {
            const float fy = Fy;
            if (fy > 0) {
                sft += (double)fy;
                float iv = Vx * Vx + Vz * Vz;
                if ((double)iv > 1e-9) {
                    iv = __frsqrt_rn(iv);
                    Fx -= 0.45f * fy * Vx * iv;
                    Fz -= 0.45f * fy * Vz * iv;
                }
            }
            if (ry + off - Yt > -1e-9) {
                Ry = Yt - off; Vy = vt; Fy = 0.f;
                if (hold) { Fx = 0.f; Fz = 0.f; Vx = 0.f; Vz = 0.f; }
            }
        }
        if (ry - off - Ybr < 1e-9) {
            const float fy = Fy;
            if (fy < 0) {
                sfb += (double)fy;
                float iv = Vx * Vx + Vz * Vz;
                if ((double)iv > 1e-9) {
                    iv = __frsqrt_rn(iv);
                    Fx += 0.45f * fy * Vx * iv;
                    Fz += 0.45f * fy * Vz * iv;
                }
            }
            if (ry - off - Yb < 1e-9) {
                Ry = Yb + off; Vy = 0.f; Fy = 0.f;
                if (hold) { Fx = 0.f; Fz = 0.f; Vx = 0.f; Vz = 0.f; }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// End of a step or force pass. A CTA of the extended kernels holds 4 * PW particles (PW per
// warp). Its warps leave their sums in shared memory and return; the one that arrives last
// combines them, and the last CTA of a specimen finishes that specimen, so a batch's
// specimens are finished side by side and nobody waits at a barrier.
// ---------------------------------------------------------------------------
// CTAs of a specimen's particles [p0, p1) in CTAs of `n` particles. A CTA touches at most
// two specimens (each has at least 128 particles): it counts as the second one's too.
__device__ __forceinline__ uint32_t spec_first_cta(const SpecGeom& G, uint32_t n) { return G.p0 / n; }
__device__ __forceinline__ uint32_t spec_last_cta(const SpecGeom& G, uint32_t n) { return (G.p1 - 1u) / n; }

// Arrival of one CTA's last warp at specimen s; true (on every lane) for the last CTA.
__device__ __forceinline__ bool arrive_last(uint32_t* counter, uint32_t expected) {
    uint32_t t = 0;
    if ((threadIdx.x & 31) == 0) t = atomicAdd(counter, 1u);
    t = __shfl_sync(0xffffffffu, t, 0);
    if (t != expected - 1u) return false;
    __threadfence();
    return true;
}

// Platen sums of a specimen: only the CTAs at the platens have any, so a CTA whose sums are
// zero writes nothing, one that has some sets its bit (nz: the CTA's first specimen, nz2: its
// second), and the specimen's last CTA reads the bits and the partials behind them, a lane a
// bit (the platens' CTAs are neighbours in the numbering: whole words of bits), adds them in
// a fixed order and clears the bits again.
__device__ __forceinline__ void spec_platen_sums(const Dev& d, const SpecGeom& G, uint32_t n, double& pb, double& pt) {
    const uint32_t FULL = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t b0 = spec_first_cta(G, n), b1 = spec_last_cta(G, n), w0 = b0 >> 5, w1 = b1 >> 5;
    const bool shared0 = b0 * n < G.p0;              // the first CTA's first specimen is the one before
    pb = 0.0; pt = 0.0;
    if (w1 - w0 < 8u) {
        // a small specimen: bits and partials are asked for together, and a partial counts if its
        // bit is set (the bits first, then the partials behind them, were two latencies of the
        // chain that ends every step)
        uint32_t m[8];
        double2 v[8];
#pragma unroll
        for (uint32_t u = 0; u < 8; ++u) {
            m[u] = 0u;
            v[u] = make_double2(0.0, 0.0);
            if (w0 + u > w1) continue;
            m[u] = __ldcg(&d.nz[w0 + u]);
            const uint32_t b = (w0 + u) * 32u + lane;
            if (b >= b0 && b <= b1) v[u] = __ldcg(&d.partial[b]);
        }
#pragma unroll
        for (uint32_t u = 0; u < 8; ++u) {
            const uint32_t w = w0 + u;
            if (w == w0) m[u] &= (0xffffffffu << (b0 & 31u)) & (shared0 ? ~(1u << (b0 & 31u)) : 0xffffffffu);
            if (w == w1) m[u] &= 0xffffffffu >> (31u - (b1 & 31u));
            if (m[u] && lane == 0) atomicAnd(&d.nz[w], ~m[u]);
            if ((m[u] >> lane) & 1u) { pb += v[u].x; pt += v[u].y; }
        }
    } else
    for (uint32_t wb = w0; wb <= w1; wb += 256u) {
        uint32_t m[8];
#pragma unroll
        for (uint32_t u = 0; u < 8; ++u) {
            const uint32_t w = wb + u * 32u + lane;
            m[u] = w <= w1 ? __ldcg(&d.nz[w]) : 0u;
            if (w == w0) m[u] &= (0xffffffffu << (b0 & 31u)) & (shared0 ? ~(1u << (b0 & 31u)) : 0xffffffffu);
            if (w == w1) m[u] &= 0xffffffffu >> (31u - (b1 & 31u));
        }
#pragma unroll
        for (uint32_t u = 0; u < 8; ++u) {
            if (m[u]) atomicAnd(&d.nz[wb + u * 32u + lane], ~m[u]);
            uint32_t has = __ballot_sync(FULL, m[u] != 0u);
            while (has) {                            // four words' partials in flight
                double2 v[4];
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    v[t] = make_double2(0.0, 0.0);
                    if (has) {
                        const uint32_t l = (uint32_t)__ffs(has) - 1u, bits = __shfl_sync(FULL, m[u], l);
                        has &= has - 1u;
                        if ((bits >> lane) & 1u) v[t] = __ldcg(&d.partial[(wb + u * 32u + l) * 32u + lane]);
                    }
                }
#pragma unroll
                for (int t = 0; t < 4; ++t) { pb += v[t].x; pt += v[t].y; }
            }
        }
    }
    if (shared0 && lane == 0) {
        const uint32_t bit = 1u << (b0 & 31u);
        if (__ldcg(&d.nz2[w0]) & bit) {
            atomicAnd(&d.nz2[w0], ~bit);
            const double2 v = __ldcg(&d.partial2[b0]);
            pb += v.x; pt += v.y;
        }
    }
    for (int o = 16; o; o >>= 1) {
        pb += __shfl_xor_sync(FULL, pb, o);
        pt += __shfl_xor_sync(FULL, pt, o);
    }
}

// What a specimen's scalar step reads, taken while its platen sums are on the way.
struct SpecIn {
    double VLoad, Top, FractureStress, MinStress, ZeroStress, MaxStrain, Size0, size_d, size_z, center_d, sz0, keep_frac;
    float Area;
    int32_t Loading, Fracture;
    unsigned long long steps, curve_n;
};
template <int KIND>
__device__ __forceinline__ SpecIn spec_read(const DevScalars* S) {
    constexpr int ax = (KIND == RF_TEST_BRAZIL) ? 1 : 2;
    SpecIn q;
    q.VLoad = S->VLoad; q.Top = S->Top; q.FractureStress = S->FractureStress;
    q.MinStress = S->MinStress; q.ZeroStress = S->ZeroStress; q.MaxStrain = S->MaxStrain; q.Size0 = S->Size0;
    q.size_d = S->size_d[ax]; q.size_z = S->size_d[2]; q.center_d = S->center_d[ax]; q.sz0 = S->sz0; q.keep_frac = S->keep_frac;
    q.Area = S->_1d_Area; q.Loading = S->Loading; q.Fracture = S->Fracture;
    q.steps = S->steps; q.curve_n = S->curve_n;
    return q;
}

// A specimen's scalar step (one thread): SumForcesULoading (md_results.cu:34-74), the
// fracture test and CompressB/U (md_data_types.h:223-293) from its platen sums; true while
// the specimen runs on. (Every field is read before the first is written: a load behind a store
// that may be to the same place waits for it, one memory latency after another.)
template <int KIND>
__device__ __forceinline__ bool spec_scalars(const Dev& d, const Consts& c, DevScalars* S, uint32_t s, const SpecIn& in,
                                             double sfb_all, double sft_all) {
    constexpr int ax = (KIND == RF_TEST_BRAZIL) ? 1 : 2;
    const double a1 = (double)in.Area;
    const double strain = (in.size_z - in.sz0) / in.sz0;
    const double stress = 0.5 * (fabs(sfb_all) + fabs(sft_all)) * a1;
    const bool loading = in.Loading || stress > in.MinStress;
    const bool peak = in.FractureStress < stress;
    const double fstress = peak ? stress : in.FractureStress;
    const bool fracture = in.Fracture || (loading && stress < in.ZeroStress) ||
                          (loading && stress < in.keep_frac * fstress);
    const double V = (stress < 1e-9) ? 10.0 * in.VLoad : in.VLoad;
    const double size = in.size_d + V * c.dt_d, top = in.Top + V * c.dt_d, center = in.center_d + V * c.dt_d;
    const float half = (float)(0.5 * size);
    const double total = (size - in.Size0) / in.Size0;
    const bool running = (total < in.MaxStrain) && !fracture;
    if (in.curve_n < c.curve_cap) {
        double* rec = d.curve + 3 * ((size_t)s * c.curve_cap + in.curve_n);
        rec[0] = strain;
        rec[1] = sfb_all * a1;
        rec[2] = sft_all * a1;
    }
    S->curve_n = in.curve_n + 1;
    S->Stress = stress;
    if (loading && !in.Loading) S->Loading = 1;
    if (peak) {
        S->FractureStress = stress;
        S->FractureStrain = (in.sz0 - in.size_z) / in.sz0;
    }
    if (fracture && !in.Fracture) S->Fracture = 1;
    S->V = V;
    S->size_d[ax] = size;
    S->Top = top;
    S->TopR = top - 2.0 * c.p_r_d;
    S->size[ax] = (float)size;
    S->sized2[ax] = half;
    S->center_d[ax] = center;
    S->center[ax] = (float)center;
    S->Hd2 = half;
    S->Strain = total;
    S->steps = in.steps + 1;                          // the specimen's own step count
    S->done = running ? 0u : 1u;
    return running;
}

// Shared memory of the end of a step: the warps' sums and their arrivals.
struct FinishSmem {
    double b[2][4], t[2][4];
    uint32_t nb[4], mv[4], e2[4];
    uint32_t arrived;
};

template <int KIND, int PW>
__device__ __forceinline__ void step_finish_ext(const Dev& d, const Consts& c, double sfb, double sft, float e2max,
                                                uint32_t nbroken, uint32_t moved, uint32_t sA, bool second,
                                                FinishSmem& sh) {
    DevScalars* sc = d.sc;
    constexpr uint32_t CTA = 4u * PW;
    const uint32_t FULL = 0xffffffffu;
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const bool has = sfb != 0.0 || sft != 0.0;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        double b = (second == (q == 1)) ? sfb : 0.0, t = (second == (q == 1)) ? sft : 0.0;
        if (__any_sync(FULL, has && second == (q == 1)))
            for (int o = 16; o; o >>= 1) {
                b += __shfl_xor_sync(FULL, b, o);
                t += __shfl_xor_sync(FULL, t, o);
            }
        if (l == 0) { sh.b[q][w] = b; sh.t[q][w] = t; }
    }
    const uint32_t wn = __reduce_add_sync(FULL, nbroken), wm = __reduce_or_sync(FULL, moved);
    const uint32_t we = __reduce_max_sync(FULL, __float_as_uint(e2max));
    const bool two = __any_sync(FULL, second);
    uint32_t t = 0;
    if (l == 0) {
        sh.nb[w] = wn; sh.mv[w] = wm | (two ? 0x100u : 0u); sh.e2[w] = we;
        __threadfence_block();
        t = atomicAdd(&sh.arrived, 1u);
    }
    if (__shfl_sync(FULL, t, 0) != 3u) return;
    // the CTA's last warp
    __threadfence_block();
    const uint32_t mv = sh.mv[0] | sh.mv[1] | sh.mv[2] | sh.mv[3];
    if (l == 0) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const double b = (sh.b[q][0] + sh.b[q][1]) + (sh.b[q][2] + sh.b[q][3]);
            const double tt = (sh.t[q][0] + sh.t[q][1]) + (sh.t[q][2] + sh.t[q][3]);
            if (b != 0.0 || tt != 0.0) {
                (q ? d.partial2 : d.partial)[blockIdx.x] = make_double2(b, tt);
                atomicOr(&(q ? d.nz2 : d.nz)[blockIdx.x >> 5], 1u << (blockIdx.x & 31u));
            }
        }
        const uint32_t nb = sh.nb[0] + sh.nb[1] + sh.nb[2] + sh.nb[3];
        if (nb) atomicAdd(&sc->broken, (unsigned long long)nb);
        if (mv & 0xFFu) atomicOr(&sc->moved, 1u);
        const uint32_t e2 = max(max(sh.e2[0], sh.e2[1]), max(sh.e2[2], sh.e2[3]));
        if (e2) atomicMax(&sc->d2max_next, e2);
        __threadfence();
    }
    __syncwarp();
    const uint32_t sN = sA + (((mv & 0x100u) && sA + 1u < d.nspec) ? 1u : 0u);
    for (uint32_t s = sA; s <= sN; ++s) {
        DevScalars* S = d.spec + s;
        const SpecGeom& G = d.geom[s];
        if (!arrive_last(&S->block_counter, spec_last_cta(G, CTA) - spec_first_cta(G, CTA) + 1u)) continue;
        // (final once the last CTA has arrived; read here, beside the platen sums)
        uint32_t d2max = 0, moved_any = 0;
        if (l == 0) { d2max = __ldcg(&sc->d2max_next); moved_any = __ldcg(&sc->moved); }
        bool running = false;
        const uint32_t done = S->done;
        const SpecIn in = spec_read<KIND>(S);
        if (!done) {
            double pb, pt;
            spec_platen_sums(d, G, CTA, pb, pt);
            if (l == 0) running = spec_scalars<KIND>(d, c, S, s, in, pb, pt);
        }
        if (l == 0) S->block_counter = 0;
        if (d.nspec > 1) {
            __threadfence();
            if (!arrive_last(&sc->spec_counter, d.nspec)) continue;
            running = false;
            for (uint32_t q = l; q < d.nspec; q += 32) running = running || !__ldcg(&d.spec[q].done);
            running = __any_sync(FULL, running);
            if (l == 0) { d2max = __ldcg(&sc->d2max_next); moved_any = __ldcg(&sc->moved); }
        }
        if (l == 0) {
            const unsigned long long steps = sc->steps + (d.nspec > 1 ? 1u : 0u);    // (with one specimen sc == spec)
            if (d.nspec > 1) { sc->steps = steps; sc->spec_counter = 0; }
            sc->dmax = sqrtf(__uint_as_float(d2max));
            sc->d2max_next = 0;
            sc->done = running ? 0u : 1u;
            sc->moved = 0;
            sc->rebuild = moved_any;
            if (c.use_graph) {
                cudaGraphSetConditional(c.h_rebuild, moved_any ? 1u : 0u);
                cudaGraphSetConditional(c.h_loop, (running && steps < sc->target) ? 1u : 0u);
            }
        }
    }
}

#define FIRE_SUMS 9     // F.v + M.w, |F|^2, |v|^2, |M|^2, |w|^2, sum |f_n|, pair count, platen sums (2)
#define FIRE_GROUP 128  // CTAs whose partials the last of them adds up before the specimen's last CTA does

struct FireSmem {
    double a[2][4][FIRE_SUMS];
    uint32_t mv[4];
    uint32_t arrived;
};

template <int PW>
__device__ __forceinline__ void fire_force_finish(const Dev& d, const Consts& c, double (&acc)[FIRE_SUMS], uint32_t sA,
                                                  bool second, FireSmem& sh);

// A bond record in a FIRE pass: its state at the increment's start (in rij, oijt, mijn, mijt)
// carried to the current configuration by the pair's motion since then.
__device__ __forceinline__ bool fire_bond(const Dev& d, const BondExt& b, uint32_t i, uint32_t j, const f3 r, const double3 rd,
                                          const double rr, f3& rij, f3& oijt, f3& mijn, f3& mijt, f3& fr, f3& mr,
                                          float& fnr, float& ktr, float& krr) {
    const double4 xi0 = ldg_d4(&d.x0[i]), ri0 = ldg_d4(&d.rot[i]);
    const double4 xj0 = ldg_d4(&d.x0[j]), rj0 = ldg_d4(&d.rot[j]);
    const double hx = 0.5 * (ri0.x + rj0.x), hy = 0.5 * (ri0.y + rj0.y), hz = 0.5 * (ri0.z + rj0.z);
    const f3 du = mk3((float)(rd.x - (xj0.x - xi0.x) - (hy * rd.z - hz * rd.y)),
                      (float)(rd.y - (xj0.y - xi0.y) - (hz * rd.x - hx * rd.z)),
                      (float)(rd.z - (xj0.z - xi0.z) - (hx * rd.y - hy * rd.x)));
    return bond_slot_ext_total(b, r, rr, du, mk3((float)ri0.x, (float)ri0.y, (float)ri0.z),
                               mk3((float)rj0.x, (float)rj0.y, (float)rj0.z), rij, oijt, mijn, mijt, rij, oijt, mijn, mijt,
                               fr, mr, fnr, ktr, krr);
}

// MODE 0: explicit step (Verlet increments, platen moving at V). MODE 1: force evaluation
// of one FIRE iteration: the same forces with the FIRE time step, platens at rest; net
// force and moment are stored for k_fire_update and FP64 sums of the FIRE power, the
// squared norms and the mean normal pair force are reduced for the FIRE decision.
// MINB: resident 128-thread CTAs per SM the kernel is compiled for (the register cap);
// rf_engine_autotune picks among the compiled variants by timing them.
// PW: particles of a warp (particles_per_warp). 32 where they fill the GPU, fewer where not:
// the lanes beyond the particles take part in the record and contact rounds and share the
// particles' slot and candidate scans, so the chain of a warp (its rounds and scans, one
// memory latency after another) is shorter, over more warps.
template <int KIND, int MODE, int MINB = RF_STEP_MIN_BLOCKS, int PW = 32>
__global__ void __launch_bounds__(128, MINB) k_step_ext(Dev d, Consts c) {
    constexpr int SUB = 32 / PW;                   // lanes a particle has in the scans
    DevScalars* sc = d.sc;
    // (the loop state, the particles' record masks and the CTA's specimen are asked for side by side)
    const uint32_t ip = (blockIdx.x * 4u + (threadIdx.x >> 5)) * PW + (threadIdx.x & 31u) % PW;
    const bool first = SUB == 1 || (threadIdx.x & 31u) < (uint32_t)PW;
    const uint32_t stopped = MODE == 0 ? sc->done : sc->fstop;
    const unsigned long long steps = sc->steps, target = sc->target;
    uint32_t bmask = ip < c.N && first ? d.bmask[ip] : 0u;
    uint32_t sA = 0u;
    if (d.blk_spec) sA = (uint32_t)d.blk_spec[(blockIdx.x * 4u * PW) >> 7];
    if (MODE == 1 && c.fire_skip && sc->rebuild) return;
    if (c.use_graph && blockIdx.x == 0 && threadIdx.x == 0) cudaGraphSetConditional(c.h_loop, 0u);
    if (stopped || (MODE == 0 && steps >= target)) return;
    union Finish { FinishSmem step; FireSmem fire; };
    __shared__ Finish s_fin;
    if (threadIdx.x == 0) { if (MODE == 0) s_fin.step.arrived = 0u; else s_fin.fire.arrived = 0u; }
    __syncthreads();
    const uint32_t cur = (uint32_t)(steps & 1ull), nxt = cur ^ 1u;
    const double4* __restrict__ P = d.posd[cur];
    const F8* __restrict__ VW = d.vw[cur];
    const uint32_t N = c.N;
    const uint32_t lane = threadIdx.x & 31u, wp = threadIdx.x >> 5;
    const uint32_t pl = lane % PW, sub = lane / PW;            // particle of the warp, share of its scans
    const uint32_t wbase = (blockIdx.x * 4u + wp) * PW;
    const uint32_t i = wbase + pl;
    const bool mine = i < N && (SUB == 1 || sub == 0);         // the lane keeps the particle's state
    // specimen of this particle: the CTA's first one, or the next
    // (a batch; one specimen runs until the loop stops)
    uint32_t sI = 0u, ended = 0u;
    if (d.blk_spec) {
        if (blockIdx.x * 4u * PW >= d.geom[sA].p1) ++sA;
        const uint32_t p1 = d.geom[sA].p1;
        ended = MODE == 0 ? d.spec[sA].done : d.spec[sA].fstop;
        sI = sA;
        if (i < N && i >= p1) {
            sI = sA + 1u;
            ended = MODE == 0 ? d.spec[sI].done : d.spec[sI].fstop;
        }
    }
    const SpecGeom& G = d.geom[sI];
    const DevScalars* S = d.spec + sI;
    // a finished specimen of a batch is frozen: its state is carried to the next buffer
    // (explicit steps: it reached its stop rule; FIRE: its relaxation of this increment stopped)
    const bool frozen = i < N && ended != 0u;
    const bool active = i < N && !frozen;                      // (on every lane of the particle)
    const bool valid = mine && !frozen;
    const uint32_t FULL = 0xffffffffu;
    if (frozen && mine) {
        d.posd[nxt][i] = P[i];
        d.vw[nxt][i] = VW[i];
        const float* oi = d.cO[cur] + (size_t)i * c.K * 3;
        float* oo = d.cO[nxt] + (size_t)i * c.K * 3;
        uint32_t m = d.cmask[i];
        while (m) {
            const uint32_t k = __ffs(m) - 1;
            m &= m - 1;
            oo[3 * k] = oi[3 * k]; oo[3 * k + 1] = oi[3 * k + 1]; oo[3 * k + 2] = oi[3 * k + 2];
        }
    }
    ExtParams ep = c.ep;
    if (MODE == 1) {
        // FIRE minimises the conservative part of the model: its own velocity mixing
        // and restarts replace the viscous contact damping, and the constant-torque
        // rolling resistance (a set-valued term at rest) is left out.
        ep.dt = (float)S->fdt;
        ep.p_A = 0.f;
        ep.mur = 0.f;
    }
    float fnabs = 0.f, kt = 0.f, kr = 0.f;
    uint32_t npair = 0;
    if (!valid) bmask = 0u;
    bool dirty = false;          // live, bond, bmask or member changed
    // bond slots whose pair overlaps: their contact (in parallel with the bond) was taken
    // in the bond pass, with its tangential overlap kept in the slot's contact state
    uint32_t pc = 0;
    uint32_t nbroken = 0;
    f3 fsb = mk3(0.f, 0.f, 0.f), msb = fsb;        // the particle's bond sums
    uint32_t cm_end = 0, bond_end = 0, del = 0;    // slots whose contact state ends, whose bond broke; deleted records
    // One record's result is 7 words (FIRE: 10), one contact's 12 (15); CH records are evaluated
    // before the particles add them.
    constexpr int CH = PW == 32 ? 128 : 64;
    constexpr int NR = MODE == 1 ? 10 : 7, NC = MODE == 1 ? 15 : 12;
    constexpr int BUF = NR * CH > NC * 32 ? NR * CH : NC * 32;
    __shared__ float s_buf[4][BUF];
    {
        // Bond records, spread over the warp. The warp's active records are listed
        // ordinal-major (every particle's first record, then every second one, ...; lane
        // order within an ordinal), so consecutive lanes read consecutive entries of the
        // [QB][N] record arrays, and in each round every lane takes one record whatever the
        // particles' bond counts. The lane that takes a record forms its force, moment
        // and outcome from zero and leaves them in shared memory; after every CH records each
        // particle adds its own in record order, in registers (added round by round into sums
        // kept in shared memory, that took a third of a round's time). A pair that overlaps is
        // only marked in its round; the marked ones of a chunk are then taken side by side
        // (contacts within the rounds were run for a few lanes at a time). FIRE mode reads the
        // records' increment-start state and the motion since then.
        __shared__ uint32_t s_q0[4][32], s_qb[4][32];  // per ordinal: first list entry, lanes holding one
        extern __shared__ __align__(16) unsigned char rf_step_smem[];
        const uint32_t lt = (1u << lane) - 1u;
        uint16_t* lst = reinterpret_cast<uint16_t*>(rf_step_smem) + (size_t)wp * (uint32_t)PW * d.QB;
        const uint32_t qend = 32u - __clz(__reduce_or_sync(FULL, bmask));
        uint32_t T = 0;
        for (uint32_t q = 0; q < qend; ++q) {
            const bool has = (bmask >> q) & 1u;
            const uint32_t bal = __ballot_sync(FULL, has);
            if (has) lst[T + __popc(bal & lt)] = (uint16_t)(lane | (q << 5));
            if (lane == q) { s_q0[wp][q] = T; s_qb[wp][q] = bal; }
            T += __popc(bal);
        }
        uint32_t rem = bmask;                          // this particle's records not yet added
        __syncwarp();
        const Rec* src = MODE == 1 ? d.rec0 : d.rec;
        float* res = s_buf[wp];
        __shared__ uint8_t s_par[4][CH];               // records of the chunk whose pair overlaps
        for (uint32_t base = 0; base < T; base += CH) {
            uint32_t npar = 0;
            for (uint32_t x0 = 0; x0 < CH && base + x0 < T; x0 += 32u) {
                const uint32_t x = x0 + lane, p = base + x;
                bool par = false;
                if (p < T) {
                    const uint32_t e = lst[p];
                    const uint32_t ol = e & 31u, q = e >> 5, io = wbase + ol;
                    const size_t s = (size_t)q * N + io;
                    // every load of the record is issued before the partner's gathers
                    const uint2 jk = d.bjk[s];
                    float4 s0, s1, s2, kc;
                    ld8(&src[s].s0, s0, s1);
                    ld8(&src[s].s2, s2, kc);
                    const uint32_t j = jk.x;
                    const double4 xo = ldg_d4(&P[io]);
                    const double4 xj = ldg_d4(&P[j]);
                    const F8 vwj = ldg8(&VW[j]);
                    const double L0 = rec_L0(kc);
                    const double3 rd = dsub(xj, xo);
                    const double rr = dlen2(rd);
                    uint32_t fl = jk.y << 8;
                    f3 fr = mk3(0.f, 0.f, 0.f), mr = fr;
                    float fnr = 0.f, ktr = 0.f, krr = 0.f;
                    if (rr > bond_cut2_del(c, xo.w, xj.w, L0) || rr < 1e-10) {
                        fl |= RF_REC_DELETE;
                    } else {
                        const float ro = (float)xo.w, rj = (float)xj.w;
                        // parallel contact (extended model, explicit steps): an overlapping bonded pair
                        // also carries the Hertz-Mindlin contact, and a broken bond's slot keeps that
                        // contact's state. Its overlap counts from min(r_i + r_j, L0), so a bond formed
                        // between overlapping particles is force-free at its rest length. FIRE
                        // relaxation leaves it out: its state would depend on the path.
                        const double sr = fmin(xo.w + xj.w, L0);
                        par = MODE == 0 && !c.ref_mode && rr < sr * sr;
                        BondExt b;
                        b.kn = c.kn; b.ks = c.ks; b.br = c.br_lambda * fminf(ro, rj);
                        b.sc = kc.z; b.tc = kc.w; b.L0 = L0;
                        if (MODE == 0 && c.ref_mode) {
                            const float il = (float)(1.0 / L0);
                            b.kn = c.refE * il; b.ks = c.refG * il; b.br = c.ref_br;
                        }
                        const f3 r = mk3((float)rd.x, (float)rd.y, (float)rd.z);
                        f3 rij = mk3(s0.x, s0.y, s0.z), oijt = mk3(s0.w, s1.x, s1.y);
                        f3 mijn = mk3(s1.z, s1.w, s2.x), mijt = mk3(s2.y, s2.z, s2.w);
                        bool broke;
                        if (MODE == 1) {
                            broke = fire_bond(d, b, io, j, r, rd, rr, rij, oijt, mijn, mijt, fr, mr, fnr, ktr, krr);
                        } else {
                            const F8 vwo = ldg8(&VW[io]);
                            broke = bond_slot_ext(ep, b, r, rr, f4to3(vwo.a), f4to3(vwj.a), f4to3(vwo.b), f4to3(vwj.b), rij, oijt, mijn, mijt, fr, mr, fnr, ktr, krr, c.ref_mode != 0);
                        }
                        // (a FIRE pass reads the increment's start state, so the state it leads to is
                        // only written when the bond breaks; the relaxed one by k_fire_bond_state)
                        if (MODE == 0 || broke) {
                            st8(&d.rec[s].s0, make_float4(rij.x, rij.y, rij.z, oijt.x), make_float4(oijt.y, oijt.z, mijn.x, mijn.y));
                            st8(&d.rec[s].s2, make_float4(mijn.z, mijt.x, mijt.y, mijt.z), kc);
                        }
                        if (broke) fl |= RF_REC_BROKE;
                    }
                    res[x] = fr.x; res[CH + x] = fr.y; res[2 * CH + x] = fr.z;
                    res[3 * CH + x] = mr.x; res[4 * CH + x] = mr.y; res[5 * CH + x] = mr.z;
                    res[6 * CH + x] = __uint_as_float(fl);
                    if (MODE == 1) { res[7 * CH + x] = fnr; res[8 * CH + x] = ktr; res[9 * CH + x] = krr; }
                }
                if (MODE == 0) {
                    const uint32_t bal = __ballot_sync(FULL, par);
                    if (par) s_par[wp][npar + __popc(bal & lt)] = (uint8_t)x;
                    npar += __popc(bal);
                }
            }
            __syncwarp();
            if (MODE == 0) {
                for (uint32_t t0 = 0; t0 < npar; t0 += 32u) {
                    if (t0 + lane < npar) {
                        const uint32_t x = s_par[wp][t0 + lane], e = lst[base + x], io = wbase + (e & 31u);
                        const size_t s = (size_t)(e >> 5) * N + io;
                        const uint2 jk = d.bjk[s];
                        const uint32_t j = jk.x, k = jk.y;
                        const double L0 = rec_L0(d.rec[s].k);
                        const double4 xo = ldg_d4(&P[io]), xj = ldg_d4(&P[j]);
                        const size_t so = ((size_t)io * c.K + k) * 3;
                        const float* oi = d.cO[cur] + so;
                        // (a record's slot is in contact at the step's start until this record is added)
                        f3 o = ((d.cmask[io] >> k) & 1u) ? mk3(oi[0], oi[1], oi[2]) : mk3(0.f, 0.f, 0.f);
                        const F8 vwo = ldg8(&VW[io]), vwj = ldg8(&VW[j]);
                        const f3 wo = f4to3(vwo.b);
                        const double3 rd = dsub(xj, xo);
                        const float ro = (float)xo.w, rj = (float)xj.w;
                        const ContactTerms ct = contact_terms_ext(
                            ep, mk3((float)rd.x, (float)rd.y, (float)rd.z), dlen2(rd), fmin(xo.w + xj.w, L0), ro, rj,
                            c.cmass * ro * ro * ro, c.cmass * rj * rj * rj, f4to3(vwo.a), f4to3(vwj.a), wo,
                            f4to3(vwj.b), o);
                        float* oo = d.cO[nxt] + so;
                        oo[0] = o.x; oo[1] = o.y; oo[2] = o.z;
                        f3 fr = mk3(res[x], res[CH + x], res[2 * CH + x]);
                        f3 mr = mk3(res[3 * CH + x], res[4 * CH + x], res[5 * CH + x]);
                        float u0 = 0.f, u1 = 0.f, u2 = 0.f;    // (FIRE's sums: no contact in parallel there)
                        add_contact(ct, ro, wo, fr, mr, u0, u1, u2);
                        res[x] = fr.x; res[CH + x] = fr.y; res[2 * CH + x] = fr.z;
                        res[3 * CH + x] = mr.x; res[4 * CH + x] = mr.y; res[5 * CH + x] = mr.z;
                        res[6 * CH + x] = __uint_as_float(__float_as_uint(res[6 * CH + x]) | RF_REC_PARALLEL |
                                                          (ct.clear ? RF_REC_CLEAR : 0u));
                    }
                }
                __syncwarp();
            }
            // this particle's records of the chunk, in record order
            while (rem) {
                const uint32_t q = __ffs(rem) - 1u;
                const uint32_t x = s_q0[wp][q] + __popc(s_qb[wp][q] & lt) - base;
                if (x >= (uint32_t)CH) break;
                rem &= rem - 1u;
                const uint32_t fl = __float_as_uint(res[6 * CH + x]);
                const uint32_t bit = 1u << ((fl >> 8) & 31u);
                if (fl & RF_REC_DELETE) { del |= 1u << q; continue; }
                fsb.x += res[x]; fsb.y += res[CH + x]; fsb.z += res[2 * CH + x];
                msb.x += res[3 * CH + x]; msb.y += res[4 * CH + x]; msb.z += res[5 * CH + x];
                if (fl & RF_REC_CLEAR) msb = mk3(0.f, 0.f, 0.f);   // the contact's zero-spin rule clears the moment sum
                if (MODE == 1) {
                    fnabs += res[7 * CH + x]; kt += res[8 * CH + x]; kr += res[9 * CH + x];
                    ++npair;
                }
                if (fl & RF_REC_BROKE) { bmask &= ~(1u << q); bond_end |= bit; ++nbroken; }
                if (fl & RF_REC_PARALLEL) pc |= bit;
                else cm_end |= bit;                    // not in contact: the parallel contact's state ends
            }
            __syncwarp();
        }
    }
    uint32_t live = 0, bond = 0, cm = 0, nbq = 0, ncand = 0;
    unsigned long long mem = 0ull;
    if (valid) {
        live = d.live[i]; bond = d.bond[i]; cm = d.cmask[i];
        mem = d.member[i]; ncand = d.cand_n[i];
        nbq = d.nbq[i];
    }
    const uint32_t cm0 = cm;
    bond &= ~bond_end;
    cm &= ~cm_end;
    dirty = (bond_end | del) != 0u;
    while (del) {
        const uint32_t q = __ffs(del) - 1u;
        del &= del - 1u;
        const size_t s = (size_t)q * N + i;
        delete_slot(d, c, i, d.bjk[s].y, d.bjk[s].x, ncand, nbq, live, bond, cm, bmask, mem);
    }

    // the particle's own position (the bond pass read it through the cache; its velocity
    // and spin are read where they are used)
    double4 xi = make_double4(0, 0, 0, 1);
    if (active) xi = P[i];
    const float ri = (float)xi.w;
    const uint32_t* row = d.ids + (size_t)i * c.K;

    // ---- open slots: the previous step's DeleteFarLinks on them, and which of them overlap
    uint32_t ct = 0;                             // slots in contact
    {
        uint32_t m = live & ~bond & ~pc, far = 0;
        if (SUB > 1) {                           // every SUB-th open slot of the particle
            uint32_t all = __shfl_sync(FULL, m, pl), q = 0;
            m = 0;
            while (all) {
                if ((q++ % SUB) == sub) m |= all & (0u - all);
                all &= all - 1u;
            }
        }
        while (m) {                              // two slots' ids, then their positions, in flight
            uint32_t bit[2], j[2];
            double4 xj[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) { bit[u] = m & (0u - m); m &= m - 1u; }
#pragma unroll
            for (int u = 0; u < 2; ++u) j[u] = bit[u] ? row[__ffs(bit[u]) - 1] : i;
#pragma unroll
            for (int u = 0; u < 2; ++u) xj[u] = ldg_d4(&P[j[u]]);
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const double rr = dlen2(dsub(xj[u], xi));
                const double sr = xi.w + xj[u].w;
                if (rr > cut2_del(c, xi.w, xj[u].w) || rr < 1e-10) far |= bit[u];
                else if (rr < sr * sr) ct |= bit[u];
            }
        }
#pragma unroll
        for (int o = PW; o < 32; o <<= 1) {
            far |= __shfl_xor_sync(FULL, far, o);
            ct |= __shfl_xor_sync(FULL, ct, o);
        }
        if (SUB > 1 && sub) { far = 0; ct = 0; }
        while (far) {
            const uint32_t k = __ffs(far) - 1;
            far &= far - 1;
            delete_slot(d, c, i, k, row[k], ncand, nbq, live, bond, cm, bmask, mem);
            dirty = true;
        }
    }

    // ---- new neighbours, in the reference's insertion order
    {
        const f3 xif = mk3((float)xi.x, (float)xi.y, (float)xi.z);
        uint32_t qlim = valid ? scan_limit(d, c, i, xif.x, xif.y, xif.z, ncand) : 0u;
        unsigned long long tried = mem;
        if (SUB > 1) {                           // the particle's lanes share the candidates
            qlim = __shfl_sync(FULL, qlim, pl);
            tried = __shfl_sync(FULL, tried, pl);
        }
        bool scan = qlim != 0u;
        bool have_cells = false;
        Octant oc;
        while (SUB > 1 ? __any_sync(FULL, scan) : (int)scan) {
            unsigned long long best = ~0ull;
            uint32_t best_q = 0;
            // the candidates to test: most are in the row already (or were tried)
            unsigned long long m = scan ? ~tried & (~0ull >> (64u - qlim)) : 0ull;
            if (SUB > 1) {                       // every SUB-th of them
                unsigned long long all = m;
                m = 0ull;
                for (uint32_t r = 0; all; ++r) {
                    if (r % SUB == sub) m |= all & (0ull - all);
                    all &= all - 1ull;
                }
            }
            while (m) {                          // two in flight
                uint32_t j[2], q[2];
                double4 xj[2];
#pragma unroll
                for (uint32_t u = 0; u < 2; ++u) {
                    q[u] = (uint32_t)__ffsll((long long)m) - 1u;     // (none left: i itself)
                    j[u] = m ? __ldg(&d.cand[(size_t)q[u] * N + i]) : i;
                    m &= m - 1ull;
                }
#pragma unroll
                for (uint32_t u = 0; u < 2; ++u) xj[u] = ldg_d4(&P[j[u]]);
#pragma unroll
                for (uint32_t u = 0; u < 2; ++u) {
                    const double rr = dlen2(dsub(xj[u], xi));
                    if (j[u] == i || !(rr < cut2_add(c, xi.w, xj[u].w) && rr > 1e-10)) continue;
                    if (!have_cells) { oc = octant_of(xif, c.g); have_cells = true; }
                    const int rank = octant_rank(oc, ref_cell(mk3((float)xj[u].x, (float)xj[u].y, (float)xj[u].z), c.g));
                    if (rank < 0) continue;
                    const unsigned long long key = ((unsigned long long)rank << 32) | j[u];
                    if (key < best) { best = key; best_q = q[u]; }
                }
            }
#pragma unroll
            for (int o = PW; o < 32; o <<= 1) {
                const unsigned long long b = __shfl_xor_sync(FULL, best, o);
                const uint32_t bq = __shfl_xor_sync(FULL, best_q, o);
                if (b < best) { best = b; best_q = bq; }
            }
            if (best == ~0ull) { scan = false; continue; }
            tried |= 1ull << best_q;
            if (SUB > 1 && sub) continue;
            const uint32_t free = ~live & (c.K >= 32 ? 0xffffffffu : ((1u << c.K) - 1u));
            if (!free) { raise_status(&sc->err, RF_ERR_ROW_OVERFLOW); continue; }
            uint32_t k;
            if (i == G.p0 && (free & 1u) && (free & ~1u)) k = __ffs(free & ~1u) - 1;   // kdxfree==0 quirk
            else k = __ffs(free) - 1;
            const uint32_t j = (uint32_t)(best & 0xffffffffull);
            d.ids[(size_t)i * c.K + k] = j;
            live |= 1u << k;
            mem |= 1ull << best_q;
            dirty = true;
            const double4 xj = ldg_d4(&P[j]);
            const double sr = xi.w + xj.w;
            if (dlen2(dsub(xj, xi)) < sr * sr) ct |= 1u << k;      // a new link already in contact
        }
    }

    // ---- contacts (_21's pairs), gathered over the warp like the bond records: few particles
    // have one, so a lane takes one contact of the warp's list and the particle adds its
    // contacts' terms in slot order
    f3 fsc = mk3(0.f, 0.f, 0.f), msc = fsc;
    float fnc = 0.f, ktc = 0.f, krc = 0.f;       // contact force magnitudes and stiffness
    {
        __shared__ uint16_t s_ent[4][32];
        float* res = s_buf[wp];
        const uint32_t n = __popc(ct);
        uint32_t rk = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, rk, o);
            if (lane >= (uint32_t)o) rk += y;
        }
        const uint32_t total = __shfl_sync(FULL, rk, 31);
        rk -= n;
        uint32_t rem = ct;
        for (uint32_t base = 0; base < total; base += 32u) {
            {
                uint32_t r2 = rem, x = rk;
                while (r2 && x < base + 32u) {
                    const uint32_t k = __ffs(r2) - 1u;
                    r2 &= r2 - 1u;
                    // cm: step-start contacts minus slots deleted this step (a refilled slot starts at zero)
                    s_ent[wp][x - base] = (uint16_t)(pl | (k << 5) | (((cm >> k) & 1u) << 10));
                    ++x;
                }
            }
            __syncwarp();
            const uint32_t e = base + lane < total ? s_ent[wp][lane] : 0u;
            // (FIRE: the time step of the contact's specimen, not of the lane's: a warp may hold particles of two)
            ExtParams cp = ep;
            if (MODE == 1) cp.dt = __shfl_sync(FULL, ep.dt, e & 31u);
            if (base + lane < total) {
                const uint32_t io = wbase + (e & 31u), k = (e >> 5) & 31u;
                const size_t so = (size_t)io * c.K + k;
                const uint32_t j = d.ids[so];
                const double4 xo = ldg_d4(&P[io]), xj = ldg_d4(&P[j]);
                const float* oi = d.cO[cur] + 3 * so;
                f3 o = (e & 1024u) ? mk3(oi[0], oi[1], oi[2]) : mk3(0.f, 0.f, 0.f);
                const double3 rd = dsub(xj, xo);
                const float ro = (float)xo.w, rj = (float)xj.w;
                const F8 vwo = ldg8(&VW[io]), vwj = ldg8(&VW[j]);
                const ContactTerms t =
                    contact_terms_ext(cp, mk3((float)rd.x, (float)rd.y, (float)rd.z), dlen2(rd), xo.w + xj.w, ro, rj,
                                      c.cmass * ro * ro * ro, c.cmass * rj * rj * rj, f4to3(vwo.a), f4to3(vwj.a),
                                      f4to3(vwo.b), f4to3(vwj.b), o);
                float* oo = d.cO[nxt] + 3 * so;
                oo[0] = o.x; oo[1] = o.y; oo[2] = o.z;
                res[lane] = t.n.x; res[1 * 32 + lane] = t.n.y; res[2 * 32 + lane] = t.n.z;
                res[3 * 32 + lane] = t.fnd;
                res[4 * 32 + lane] = t.ft.x; res[5 * 32 + lane] = t.ft.y; res[6 * 32 + lane] = t.ft.z;
                res[7 * 32 + lane] = t.cr.x; res[8 * 32 + lane] = t.cr.y; res[9 * 32 + lane] = t.cr.z;
                res[10 * 32 + lane] = t.roll;
                res[11 * 32 + lane] = t.clear ? 1.f : 0.f;
                if (MODE == 1) { res[12 * 32 + lane] = t.fn; res[13 * 32 + lane] = t.k1; res[14 * 32 + lane] = t.kt; }
            }
            __syncwarp();
            if (rem && rk < base + 32u) {
                const f3 wi = f4to3(ldg8(&VW[i]).b);
                while (rem && rk < base + 32u) {
                    const uint32_t x = rk - base;
                    rem &= rem - 1u;
                    ++rk;
                    ContactTerms t;
                    t.n = mk3(res[x], res[1 * 32 + x], res[2 * 32 + x]);
                    t.fnd = res[3 * 32 + x];
                    t.ft = mk3(res[4 * 32 + x], res[5 * 32 + x], res[6 * 32 + x]);
                    t.cr = mk3(res[7 * 32 + x], res[8 * 32 + x], res[9 * 32 + x]);
                    t.roll = res[10 * 32 + x];
                    t.clear = res[11 * 32 + x] != 0.f;
                    t.rolling = ep.mur != 0.f;
                    t.fn = MODE == 1 ? res[12 * 32 + x] : 0.f;
                    t.k1 = MODE == 1 ? res[13 * 32 + x] : 0.f;
                    t.kt = MODE == 1 ? res[14 * 32 + x] : 0.f;
                    add_contact(t, ri, wi, fsc, msc, fnc, ktc, krc);
                }
            }
            __syncwarp();
        }
        npair += n;
    }
    cm = ct | pc;
    fnabs = fnc + fnabs;
    kt = ktc + kt;
    kr = krc + kr;

    float e2max = 0.f;
    double sfb = 0.0, sft = 0.0;
    uint32_t moved = 0;
    double acc[FIRE_SUMS];
#pragma unroll
    for (int q = 0; q < FIRE_SUMS; ++q) acc[q] = 0.0;
    if (valid) {
        const F8 vwi = ldg8(&VW[i]);
        float4 pr = make_float4(0.f, 0.f, 0.f, 0.f);
        if (MODE == 0) pr = d.pos_ref[i];
        const f3 vi = f4to3(vwi.a), wi = f4to3(vwi.b);
        const float mi = c.cmass * ri * ri * ri;
        if (dirty) { d.live[i] = live; d.bond[i] = bond; d.member[i] = mem; d.bmask[i] = bmask; }
        if (cm != cm0) d.cmask[i] = cm;
        // platens of this particle's specimen (with the reference constants their
        // coordinates are rounded to float, as the reference's drivers pass them)
        const double Top = c.ref_mode ? (double)(float)S->Top : S->Top;
        const double Bottom = c.ref_mode ? (double)(float)S->Bottom : S->Bottom;
        const double TopR = c.ref_mode ? (double)(float)S->TopR : S->TopR;
        const double BottomR = c.ref_mode ? (double)(float)S->BottomR : S->BottomR;
        const float vt = MODE == 0 ? (float)S->V : 0.f, RR = S->RR;
        rf_float3 cc;
        cc.x = S->center[0]; cc.y = S->center[1]; cc.z = S->center[2];
        float Fx = 0.0f + fsb.x, Fy = 0.0f + fsb.y, Fz = 0.0f + fsb.z;
        Fx += fsc.x; Fy += fsc.y; Fz += fsc.z;
        float Mx = 0.0f + msb.x, My = 0.0f + msb.y, Mz = 0.0f + msb.z;
        Mx += msc.x; My += msc.y; Mz += msc.z;
        double Rx = xi.x, Ry = xi.y, Rz = xi.z;
        float Vx = vi.x, Vy = vi.y, Vz = vi.z;
        if (KIND == RF_TEST_BRAZIL)
            brazil_particle_ext(Rx, Ry, Rz, Vx, Vy, Vz, Fx, Fy, Fz, cc, RR, Top, Bottom, TopR, BottomR, vt,
                                (double)G.zcut, xi.w - c.p_r_d, sfb, sft, MODE == 1);
        else
            uniaxial_particle_ext(Rx, Ry, Rz, Vx, Vy, Vz, Fx, Fy, Fz, cc, RR, Top, Bottom, TopR, BottomR, vt,
                                  (double)G.zcut, xi.w - c.p_r_d, sfb, sft, MODE == 1);
        if (MODE == 1) {
            // FIRE: keep the clamped state for the update kernel (and the coordinate the platens
            // may have clamped, for k_fire_bond_state); reduce the FIRE sums
            d.xax[i] = KIND == RF_TEST_BRAZIL ? xi.y : xi.z;
            d.posd[nxt][i] = make_double4(Rx, Ry, Rz, xi.w);
            st8(&d.vw[nxt][i], make_float4(Vx, Vy, Vz, 0.f), make_float4(wi.x, wi.y, wi.z, 0.f));
            d.frc[i] = make_float4(Fx, Fy, Fz, kt);
            d.mom[i] = make_float4(Mx, My, Mz, kr);
            acc[0] = (double)Fx * Vx + (double)Fy * Vy + (double)Fz * Vz + (double)Mx * wi.x + (double)My * wi.y +
                     (double)Mz * wi.z;
            acc[1] = (double)Fx * Fx + (double)Fy * Fy + (double)Fz * Fz;
            acc[2] = (double)Vx * Vx + (double)Vy * Vy + (double)Vz * Vz;
            acc[3] = (double)Mx * Mx + (double)My * My + (double)Mz * Mz;
            acc[4] = (double)wi.x * wi.x + (double)wi.y * wi.y + (double)wi.z * wi.z;
            acc[5] = (double)fnabs;
            acc[6] = (double)npair;
            acc[7] = sfb;
            acc[8] = sft;
        }
        if (MODE == 0) {
        const float dtm = ep.dt / mi, dtI = ep.dt / (0.4f * mi * ri * ri);
        Vx += Fx * dtm; Vy += Fy * dtm; Vz += Fz * dtm;
        Rx += (double)(Vx * ep.dt); Ry += (double)(Vy * ep.dt); Rz += (double)(Vz * ep.dt);
        const float Wx = wi.x + Mx * dtI, Wy = wi.y + My * dtI, Wz = wi.z + Mz * dtI;
        const double dx = Rx - G.box_c.x, dy = Ry - G.box_c.y, dz = Rz - G.box_c.z;
        if ((dx - G.box_h.x > 0) || (dx + G.box_h.x < 0) || (dy - G.box_h.y > 0) || (dy + G.box_h.y < 0) ||
            (dz - G.box_h.z > 0) || (dz + G.box_h.z < 0)) {
            Rx = G.hp.x; Ry = G.hp.y; Rz = G.hp.z;
            Vx = 0.f; Vy = 0.f; Vz = 0.f;
        }
        d.posd[nxt][i] = make_double4(Rx, Ry, Rz, xi.w);
        st8(&d.vw[nxt][i], make_float4(Vx, Vy, Vz, 0.f), make_float4(Wx, Wy, Wz, 0.f));
        const float ex = (float)Rx - pr.x, ey = (float)Ry - pr.y, ez = (float)Rz - pr.z;
        const float e2 = ex * ex + ey * ey + ez * ez;
        moved = (e2 > c.disp2) ? 1u : 0u;
        // lists may have missed a neighbour (a particle moved to the hidden point has none)
        const bool hidden = Rx == (double)G.hp.x && Ry == (double)G.hp.y && Rz == (double)G.hp.z;
        if (e2 > c.hard2 && !hidden) raise_status(&d.sc->err, RF_ERR_CAPACITY);
        if (!hidden) e2max = e2;
        }
    }
    if (MODE == 0) {
        step_finish_ext<KIND, PW>(d, c, sfb, sft, e2max, nbroken, moved, sA, sI != sA, s_fin.step);
    } else {
        const uint32_t nb = __reduce_add_sync(FULL, nbroken);
        if (lane == 0 && nb) atomicAdd(&sc->broken, (unsigned long long)nb);
        fire_force_finish<PW>(d, c, acc, sA, sI != sA, s_fin.fire);
    }
}

// The reference model's step. Same structure as the extended model's k_step_ext above (bond
// records and contacts spread over the warp, PW particles a warp); a record's and a contact's
// terms are kept apart and added by the particle's lane one by one, as the reference's slot
// loops add them.
template <int KIND, int PW>
__global__ void __launch_bounds__(128, RF_STEP_MIN_BLOCKS) k_step(Dev d, Consts c) {
    constexpr int SUB = 32 / PW;                   // lanes a particle has in the scans
    DevScalars* sc = d.sc;
    // Loop safety: clear the WHILE condition first. Only the last block's finalize,
    // which runs after every block has passed this point and advances the step
    // counter towards the target, sets it again, so the device loop always ends.
    // (the loop state and the particles' are asked for side by side, see k_step_ext)
    const uint32_t ip = (blockIdx.x * 4u + (threadIdx.x >> 5)) * PW + (threadIdx.x & 31u) % PW;
    const bool first = SUB == 1 || (threadIdx.x & 31u) < (uint32_t)PW;
    const uint32_t stopped = sc->done;
    const unsigned long long steps = sc->steps, target = sc->target;
    uint32_t live = 0, bond = 0, cm = 0, nbq = 0, bmask = 0, ncand = 0;
    unsigned long long mem = 0ull;
    if (ip < c.N && first) {
        live = d.live[ip]; bond = d.bond[ip]; cm = d.cmask[ip];
        mem = d.member[ip]; ncand = d.cand_n[ip];
        nbq = d.nbq[ip]; bmask = d.bmask[ip];
    }
    if (c.use_graph && blockIdx.x == 0 && threadIdx.x == 0) cudaGraphSetConditional(c.h_loop, 0u);
    if (stopped || steps >= target) return;
    __shared__ FinishSmem s_fin;
    if (threadIdx.x == 0) s_fin.arrived = 0u;
    __syncthreads();
    const uint32_t cur = (uint32_t)(steps & 1ull), nxt = cur ^ 1u;
    const float4* __restrict__ P = d.pos[cur];
    const F8* __restrict__ VW = d.vw[cur];
    const uint32_t N = c.N;
    const uint32_t lane = threadIdx.x & 31u, wp = threadIdx.x >> 5;
    const uint32_t pl = lane % PW, sub = lane / PW;            // particle of the warp, share of its scans
    const uint32_t wbase = (blockIdx.x * 4u + wp) * PW;
    const uint32_t i = wbase + pl;
    const bool active = i < N;                                 // (on every lane of the particle)
    const bool valid = active && (SUB == 1 || sub == 0);       // the lane keeps the particle's state
    const uint32_t FULL = 0xffffffffu;
    const uint32_t lt = (1u << lane) - 1u;

    const uint32_t cm0 = cm;
    bool dirty = false;
    uint32_t nbroken = 0;

    // ---- bonds: d_CalculateForcesDEM_22 (md_calculateforcesdem3.cu:424-483) over the bond
    // records, with the DeleteFarLinks test of each bond slot on the same gathered position
    // (md_interaction_list_reconstructbpm.cu:141-186)
    constexpr int NB = 16, NC = 13;               // words of a record's and of a contact's result
    __shared__ float s_res[4][NB][32];
    f3 fsb = mk3(0.f, 0.f, 0.f), msb = fsb;
    {
        __shared__ uint32_t s_q0[4][32], s_qb[4][32];
        extern __shared__ __align__(16) unsigned char rf_step_smem[];
        uint16_t* lst = reinterpret_cast<uint16_t*>(rf_step_smem) + (size_t)wp * (uint32_t)PW * d.QB;
        const uint32_t qend = 32u - __clz(__reduce_or_sync(FULL, bmask));
        uint32_t T = 0;
        for (uint32_t q = 0; q < qend; ++q) {
            const bool has = (bmask >> q) & 1u;
            const uint32_t bal = __ballot_sync(FULL, has);
            if (has) lst[T + __popc(bal & lt)] = (uint16_t)(lane | (q << 5));
            if (lane == q) { s_q0[wp][q] = T; s_qb[wp][q] = bal; }
            T += __popc(bal);
        }
        uint32_t rem = bmask;                          // this particle's records not yet added
        __syncwarp();
        for (uint32_t base = 0; base < T; base += 32u) {
            if (base + lane < T) {
                const uint32_t e = lst[base + lane];
                const uint32_t q = e >> 5, io = wbase + (e & 31u);
                const size_t s = (size_t)q * N + io;
                const uint2 jk = d.bjk[s];
                float4 s0, s1, s2, kc;
                ld8(&d.rec[s].s0, s0, s1);
                ld8(&d.rec[s].s2, s2, kc);
                const uint32_t j = jk.x;
                const float il = kc.x;
                uint32_t fl = jk.y << 8;
                const f3 xo = f4to3(__ldg(&P[io])), xj = f4to3(__ldg(&P[j]));
                const F8 vwo = ldg8(&VW[io]), vwj = ldg8(&VW[j]);
                const f3 vo = f4to3(vwo.a), wo = f4to3(vwo.b), vj = f4to3(vwj.a), wj = f4to3(vwj.b);
                const float rr = dist2_rn(xo, xj);
                if (rr > c.aa_farcut || below_1em10(rr)) {
                    fl |= RF_REC_DELETE;
                    s_res[wp][0][lane] = __uint_as_float(j);
                } else {
                    const f3 r = mk3(xj.x - xo.x, xj.y - xo.y, xj.z - xo.z);
                    f3 rij = mk3(s0.x, s0.y, s0.z), oijt = mk3(s0.w, s1.x, s1.y);
                    f3 mijn = mk3(s1.z, s1.w, s2.x), mijt = mk3(s2.y, s2.z, s2.w);
                    KeepTerms t;
                    if (bond_slot(c.bp, r, vo, vj, wo, wj, il, rij, oijt, mijn, mijt, t)) fl |= RF_REC_BROKE;
                    st8(&d.rec[s].s0, make_float4(rij.x, rij.y, rij.z, oijt.x), make_float4(oijt.y, oijt.z, mijn.x, mijn.y));
                    st8(&d.rec[s].s2, make_float4(mijn.z, mijt.x, mijt.y, mijt.z), kc);
#pragma unroll
                    for (int a = 0; a < 2; ++a) {
                        s_res[wp][3 * a][lane] = t.ft[a].x; s_res[wp][3 * a + 1][lane] = t.ft[a].y;
                        s_res[wp][3 * a + 2][lane] = t.ft[a].z;
                    }
#pragma unroll
                    for (int a = 0; a < 3; ++a) {
                        s_res[wp][6 + 3 * a][lane] = t.mt[a].x; s_res[wp][7 + 3 * a][lane] = t.mt[a].y;
                        s_res[wp][8 + 3 * a][lane] = t.mt[a].z;
                    }
                }
                s_res[wp][15][lane] = __uint_as_float(fl);
            }
            __syncwarp();
            while (rem) {                              // this particle's records of the round, in record order
                const uint32_t q = __ffs(rem) - 1u;
                const uint32_t x = s_q0[wp][q] + __popc(s_qb[wp][q] & lt) - base;
                if (x >= 32u) break;
                rem &= rem - 1u;
                const uint32_t fl = __float_as_uint(s_res[wp][15][x]), k = fl >> 8;
                if (fl & RF_REC_DELETE) {
                    delete_slot(d, c, i, k, __float_as_uint(s_res[wp][0][x]), ncand, nbq, live, bond, cm, bmask, mem);
                    dirty = true;
                    continue;
                }
#pragma unroll
                for (int a = 0; a < 2; ++a) {
                    fsb.x += s_res[wp][3 * a][x]; fsb.y += s_res[wp][3 * a + 1][x]; fsb.z += s_res[wp][3 * a + 2][x];
                }
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    msb.x += s_res[wp][6 + 3 * a][x]; msb.y += s_res[wp][7 + 3 * a][x]; msb.z += s_res[wp][8 + 3 * a][x];
                }
                if (fl & RF_REC_BROKE) { bmask &= ~(1u << q); bond &= ~(1u << k); ++nbroken; dirty = true; }
            }
            __syncwarp();
        }
    }

    // ---- open slots (bonds broken above included): the rest of the previous step's
    // DeleteFarLinks, and which of them overlap
    f3 xi = mk3(0.f, 0.f, 0.f);
    if (active) xi = f4to3(__ldg(&P[i]));
    const uint32_t* row = d.ids + (size_t)i * c.K;
    const float twoR = 2.0f * c.cp.rP;
    uint32_t ct = 0;                             // slots in contact
    {
        uint32_t m = live & ~bond, far = 0;
        if (SUB > 1) {                           // every SUB-th open slot of the particle
            uint32_t all = __shfl_sync(FULL, m, pl), q = 0;
            m = 0;
            while (all) {
                if ((q++ % SUB) == sub) m |= all & (0u - all);
                all &= all - 1u;
            }
        }
        while (m) {                              // four slots' ids, then their positions, in flight
            uint32_t bit[4], j[4];
            float4 xj[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) { bit[u] = m & (0u - m); m &= m - 1u; }
#pragma unroll
            for (int u = 0; u < 4; ++u) j[u] = bit[u] ? row[__ffs(bit[u]) - 1] : i;
#pragma unroll
            for (int u = 0; u < 4; ++u) xj[u] = __ldg(&P[j[u]]);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const float rr = dist2_rn(xi, f4to3(xj[u]));
                if (rr > c.aa_farcut || below_1em10(rr)) far |= bit[u];
                else if (norm3(xj[u].x - xi.x, xj[u].y - xi.y, xj[u].z - xi.z) < twoR) ct |= bit[u];
            }
        }
#pragma unroll
        for (int o = PW; o < 32; o <<= 1) {
            far |= __shfl_xor_sync(FULL, far, o);
            ct |= __shfl_xor_sync(FULL, ct, o);
        }
        if (SUB > 1 && sub) { far = 0; ct = 0; }
        while (far) {
            const uint32_t k = __ffs(far) - 1;
            far &= far - 1;
            delete_slot(d, c, i, k, row[k], ncand, nbq, live, bond, cm, bmask, mem);
            dirty = true;
        }
    }

    // ---- add: InteractionListReConstructBPM (md_interaction_list_reconstructbpm.cu:13-46,80-139)
    // (skipped when no candidate can have come within a_farcut since the build: the scan
    // would add nothing)
    {
        uint32_t qlim = valid ? scan_limit(d, c, i, xi.x, xi.y, xi.z, ncand) : 0u;
        unsigned long long tried = mem;
        if (SUB > 1) {                           // the particle's lanes share the candidates
            qlim = __shfl_sync(FULL, qlim, pl);
            tried = __shfl_sync(FULL, tried, pl);
        }
        bool scan = qlim != 0u;
        bool have_cells = false;
        Octant oc;
        while (SUB > 1 ? __any_sync(FULL, scan) : (int)scan) {
            unsigned long long best = ~0ull;
            uint32_t best_q = 0;
            // the candidates to test: most are in the row already (or were tried)
            unsigned long long m = scan ? ~tried & (~0ull >> (64u - qlim)) : 0ull;
            if (SUB > 1) {                       // every SUB-th of them
                unsigned long long all = m;
                m = 0ull;
                for (uint32_t r = 0; all; ++r) {
                    if (r % SUB == sub) m |= all & (0ull - all);
                    all &= all - 1ull;
                }
            }
            while (m) {                          // four in flight
                uint32_t j[4], q[4];
                float4 xj[4];
#pragma unroll
                for (uint32_t u = 0; u < 4; ++u) {
                    q[u] = (uint32_t)__ffsll((long long)m) - 1u;     // (none left: i itself)
                    j[u] = m ? __ldg(&d.cand[(size_t)q[u] * N + i]) : i;
                    m &= m - 1ull;
                }
#pragma unroll
                for (uint32_t u = 0; u < 4; ++u) xj[u] = __ldg(&P[j[u]]);
#pragma unroll
                for (uint32_t u = 0; u < 4; ++u) {
                    const float rr = dist2_rn(xi, f4to3(xj[u]));
                    if (j[u] == i || !(rr < c.aacut && above_1em10(rr))) continue;
                    if (!have_cells) { oc = octant_of(xi, c.g); have_cells = true; }
                    const int rank = octant_rank(oc, ref_cell(f4to3(xj[u]), c.g));
                    if (rank < 0) continue;
                    const unsigned long long key = ((unsigned long long)rank << 32) | j[u];
                    if (key < best) { best = key; best_q = q[u]; }
                }
            }
#pragma unroll
            for (int o = PW; o < 32; o <<= 1) {
                const unsigned long long b = __shfl_xor_sync(FULL, best, o);
                const uint32_t bq = __shfl_xor_sync(FULL, best_q, o);
                if (b < best) { best = b; best_q = bq; }
            }
            if (best == ~0ull) { scan = false; continue; }
            tried |= 1ull << best_q;
            if (SUB > 1 && sub) continue;
            const uint32_t free = ~live & (c.K >= 32 ? 0xffffffffu : ((1u << c.K) - 1u));
            if (!free) { raise_status(&sc->err, RF_ERR_ROW_OVERFLOW); continue; }
            uint32_t k;
            if (i == 0 && (free & 1u) && (free & ~1u)) k = __ffs(free & ~1u) - 1;   // kdxfree==0 quirk
            else k = __ffs(free) - 1;
            const uint32_t j = (uint32_t)(best & 0xffffffffull);
            d.ids[(size_t)i * c.K + k] = j;
            live |= 1u << k;
            mem |= 1ull << best_q;
            dirty = true;
            const f3 xj = f4to3(__ldg(&P[j]));
            if (norm3(xj.x - xi.x, xj.y - xi.y, xj.z - xi.z) < twoR) ct |= 1u << k;    // already in contact
        }
    }

    // ---- contacts: d_CalculateForcesDEM_21 (md_calculateforcesdem3.cu:338-422) over the
    // warp's overlapping type-0 slots, each particle's in slot order. Overlaps are read from
    // this step's buffer and written to the next one.
    f3 fsc = mk3(0.f, 0.f, 0.f), msc = fsc;
    {
        __shared__ uint16_t s_ent[4][32];
        uint32_t rk = __popc(ct);
        const uint32_t n = rk;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, rk, o);
            if (lane >= (uint32_t)o) rk += y;
        }
        const uint32_t total = __shfl_sync(FULL, rk, 31);
        rk -= n;
        uint32_t rem = ct;
        for (uint32_t base = 0; base < total; base += 32u) {
            {
                uint32_t r2 = rem, x = rk;
                while (r2 && x < base + 32u) {
                    const uint32_t k = __ffs(r2) - 1u;
                    r2 &= r2 - 1u;
                    s_ent[wp][x - base] = (uint16_t)(pl | (k << 5) | (((cm >> k) & 1u) << 10));
                    ++x;
                }
            }
            __syncwarp();
            if (base + lane < total) {
                const uint32_t e = s_ent[wp][lane], io = wbase + (e & 31u), k = (e >> 5) & 31u;
                const size_t so = (size_t)io * c.K + k;
                const uint32_t j = d.ids[so];
                const f3 xo = f4to3(__ldg(&P[io])), xj = f4to3(__ldg(&P[j]));
                const float* oi = d.cO[cur] + 3 * so;
                f3 o = (e & 1024u) ? mk3(oi[0], oi[1], oi[2]) : mk3(0.f, 0.f, 0.f);
                const f3 r = mk3(xj.x - xo.x, xj.y - xo.y, xj.z - xo.z);
                KeepTerms t;
                const F8 vwo = ldg8(&VW[io]), vwj = ldg8(&VW[j]);
                contact_pair(c.cp, r, norm3(r.x, r.y, r.z), f4to3(vwo.a), f4to3(vwj.a), f4to3(vwo.b), f4to3(vwj.b), o, t);
                float* oo = d.cO[nxt] + 3 * so;
                oo[0] = o.x; oo[1] = o.y; oo[2] = o.z;
                if (t.clear) t.mt[1] = mk3(0.f, 0.f, 0.f);
#pragma unroll
                for (int a = 0; a < 2; ++a) {
                    s_res[wp][3 * a][lane] = t.ft[a].x; s_res[wp][3 * a + 1][lane] = t.ft[a].y;
                    s_res[wp][3 * a + 2][lane] = t.ft[a].z;
                    s_res[wp][6 + 3 * a][lane] = t.mt[a].x; s_res[wp][7 + 3 * a][lane] = t.mt[a].y;
                    s_res[wp][8 + 3 * a][lane] = t.mt[a].z;
                }
                s_res[wp][NC - 1][lane] = t.clear ? 1.f : 0.f;
            }
            __syncwarp();
            while (rem && rk < base + 32u) {
                const uint32_t x = rk - base;
                rem &= rem - 1u;
                ++rk;
#pragma unroll
                for (int a = 0; a < 2; ++a) {
                    fsc.x += s_res[wp][3 * a][x]; fsc.y += s_res[wp][3 * a + 1][x]; fsc.z += s_res[wp][3 * a + 2][x];
                }
                if (s_res[wp][NC - 1][x] != 0.f) { msc = mk3(0.f, 0.f, 0.f); continue; }   // zero spin: sum cleared
#pragma unroll
                for (int a = 0; a < 2; ++a) {
                    msc.x += s_res[wp][6 + 3 * a][x]; msc.y += s_res[wp][7 + 3 * a][x]; msc.z += s_res[wp][8 + 3 * a][x];
                }
            }
            __syncwarp();
        }
    }
    cm = ct;

    float e2max = 0.f;
    double sfb = 0.0, sft = 0.0;
    uint32_t moved = 0;
    if (valid) {
        if (dirty) { d.live[i] = live; d.bond[i] = bond; d.member[i] = mem; d.bmask[i] = bmask; }
        if (cm != cm0) d.cmask[i] = cm;
        // platen arguments of this step, as the driver passes them (double -> float)
        const float Top = (float)sc->Top, Bottom = (float)sc->Bottom, TopR = (float)sc->TopR,
                    BottomR = (float)sc->BottomR, vt = (float)sc->V, RR = sc->RR;
        rf_float3 cc;
        cc.x = sc->center[0]; cc.y = sc->center[1]; cc.z = sc->center[2];
        const F8 vwi = ldg8(&VW[i]);
        const f3 vi = f4to3(vwi.a), wi = f4to3(vwi.b);
        // F = 0 after the memset, then += _22 sums, then += _21 sums
        float Fx = 0.0f + fsb.x, Fy = 0.0f + fsb.y, Fz = 0.0f + fsb.z;
        Fx += fsc.x; Fy += fsc.y; Fz += fsc.z;
        float Mx = 0.0f + msb.x, My = 0.0f + msb.y, Mz = 0.0f + msb.z;
        Mx += msc.x; My += msc.y; Mz += msc.z;
        float Rx = xi.x, Ry = xi.y, Rz = xi.z, Vx = vi.x, Vy = vi.y, Vz = vi.z;
        if (KIND == RF_TEST_BRAZIL)
            brazil_particle(Rx, Ry, Rz, Vx, Vy, Vz, Fx, Fy, Fz, cc, RR, Top, Bottom, TopR, BottomR, vt, c.zcut, sfb, sft);
        else
            uniaxial_particle(Rx, Ry, Rz, Vz, Fz, cc, RR, Top, Bottom, TopR, BottomR, vt, c.zcut, sfb, sft);
        // d_CalculateIncrementsDEM (md_calculateincrementsdem.cu:19-49)
        Vx += __fmul_rn(Fx, c.dtm); Vy += __fmul_rn(Fy, c.dtm); Vz += __fmul_rn(Fz, c.dtm);
        Rx += __fmul_rn(Vx, c.dt); Ry += __fmul_rn(Vy, c.dt); Rz += __fmul_rn(Vz, c.dt);
        float Wx = wi.x + __fmul_rn(Mx, c.dtI), Wy = wi.y + __fmul_rn(My, c.dtI), Wz = wi.z + __fmul_rn(Mz, c.dtI);
        // d_ParallelepipedCutRestriction (md_parallelepipedrestriction.cu:73-159)
        if (outside_box(Rx, Ry, Rz, c.box_c, c.box_h)) {
            Rx = c.hp.x; Ry = c.hp.y; Rz = c.hp.z;
            Vx = 0.f; Vy = 0.f; Vz = 0.f;
        }
        d.pos[nxt][i] = make_float4(Rx, Ry, Rz, 0.f);
        st8(&d.vw[nxt][i], make_float4(Vx, Vy, Vz, 0.f), make_float4(Wx, Wy, Wz, 0.f));
        const float4 pr = d.pos_ref[i];
        const float ex = Rx - pr.x, ey = Ry - pr.y, ez = Rz - pr.z;
        const float e2 = ex * ex + ey * ey + ez * ez;
        moved = (e2 > c.disp2) ? 1u : 0u;
        // lists may have missed a neighbour (a particle moved to the hidden point has none)
        const bool hidden = Rx == c.hp.x && Ry == c.hp.y && Rz == c.hp.z;
        if (e2 > c.hard2 && !hidden) raise_status(&d.sc->err, RF_ERR_CAPACITY);
        if (!hidden) e2max = e2;
    }
    step_finish_ext<KIND, PW>(d, c, sfb, sft, e2max, nbroken, moved, 0u, false, s_fin);
}

// The FIRE decision of one specimen from its sums tot (FP64; n its particle count), by
// the last CTA's thread 0 (Bitzek et al. 2006):
//   residual = sqrt(sum |F_i|^2 / n) / (mean normal pair force); converged when <= tol;
//   P = F.v + M.w > 0: mixing v <- (1-a) v + a (|v|/|F|) F (same for w with M), and after
//   n_delay such steps dt <- min(dt f_inc, dt_max), a <- a f_alpha;
//   P <= 0: dt <- max(dt f_dec, dt_min), a <- a0, v = w = 0.
// (The quotients and roots are formed side by side and every field is read before the first
// is written, as in spec_scalars.)
__device__ __forceinline__ void fire_decide(DevScalars* S, const Consts& c, const double* tot, uint32_t n) {
    const double P = tot[0], FF = tot[1], VV = tot[2], MM = tot[3], WW = tot[4], FN = tot[5], NP = tot[6];
    const double ftol = S->ftol, a = S->falpha, fdt = S->fdt, finc = S->finc, fdtmax = S->fdtmax, fshrink = S->fshrink,
                 fdec = S->fdec, fdtmin = S->fdtmin, falpha0 = S->falpha0;
    const unsigned long long iter = S->fiter + 1, max_iter = S->fmax_iter, total = S->fiter_total, npos = S->fnpos;
    const uint32_t ndelay = S->fndelay, warm = S->fwarm;
    const double a1 = (double)S->_1d_Area;
    const double mean = NP > 0.0 ? FN / NP : 0.0;
    const double rms = sqrt(FF / (double)n);
    const double vf = sqrt(VV / FF), wm = sqrt(WW / MM);
    const double residual = mean > 0.0 ? rms / mean : (FF > 0.0 ? 1e300 : 0.0);
    S->fmean = mean;
    S->fresidual = residual;
    S->fpower = P;
    // platen stress of this configuration (SumForcesULoading's formula)
    S->Stress = 0.5 * (fabs(tot[7]) + fabs(tot[8])) * a1;
    S->fiter = iter;
    S->fiter_total = total + 1;
    if (residual <= ftol) { S->fconverged = 1; S->fstop = 1; return; }
    if (iter >= max_iter) { S->fstop = 1; return; }
    if (warm) {
        // first pass of an increment: the velocities only carried the start motion into
        // the state; the dynamics starts from rest
        S->fwarm = 0;
        S->fuphill = 1;
        S->fnpos = 0;
        S->fcv = 0.0; S->fcf = 0.0; S->fcm = 0.0;
    } else if (P > 0.0) {
        S->fcv = 1.0 - a;
        S->fcf = FF > 0.0 ? a * vf : 0.0;
        S->fcm = MM > 0.0 ? a * wm : 0.0;
        S->fuphill = 0;
        S->fnpos = npos + 1;
        if (npos + 1 > ndelay) {
            S->fdt = fmin(fdt * finc, fdtmax);
            S->falpha = a * fshrink;
        }
    } else {
        S->fnpos = 0;
        S->fdt = fmax(fdt * fdec, fdtmin);
        S->falpha = falpha0;
        S->fuphill = 1;
        S->fcv = 0.0; S->fcf = 0.0; S->fcm = 0.0;
    }
}

// The FIRE sums of a force pass: warps to CTA as in step_finish_ext, then in a fixed order the
// last CTA of every FIRE_GROUP of a specimen's CTAs adds that group's partials and the
// specimen's last CTA the groups' (a lane's share, then the warp tree), and makes the
// specimen's FIRE decision. (One CTA adding all partials of a 1M-particle specimen was a
// tail of 61 dependent rounds of loads.)
template <int PW>
__device__ __forceinline__ void fire_force_finish(const Dev& d, const Consts& c, double (&acc)[FIRE_SUMS], uint32_t sA,
                                                  bool second, FireSmem& sh) {
    DevScalars* sc = d.sc;
    constexpr uint32_t CTA = 4u * PW;
    const uint32_t FULL = 0xffffffffu;
    const uint32_t w = threadIdx.x >> 5, l = threadIdx.x & 31u;
    const bool two = __any_sync(FULL, second);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        if (q == 1 && !two) break;                            // (uniform; read only if a warp has two)
#pragma unroll
        for (int k = 0; k < FIRE_SUMS; ++k) {
            double v = (second == (q == 1)) ? acc[k] : 0.0;
            for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
            if (l == 0) sh.a[q][w][k] = v;
        }
    }
    uint32_t t = 0;
    if (l == 0) {
        if (!two)
            for (int k = 0; k < FIRE_SUMS; ++k) sh.a[1][w][k] = 0.0;
        sh.mv[w] = two ? 1u : 0u;
        __threadfence_block();
        t = atomicAdd(&sh.arrived, 1u);
    }
    if (__shfl_sync(FULL, t, 0) != 3u) return;
    __threadfence_block();
    const bool any2 = (sh.mv[0] | sh.mv[1] | sh.mv[2] | sh.mv[3]) != 0u;
    if (l < FIRE_SUMS) {
        d.fpart[(size_t)blockIdx.x * FIRE_SUMS + l] = (sh.a[0][0][l] + sh.a[0][1][l]) + (sh.a[0][2][l] + sh.a[0][3][l]);
        if (any2)
            d.fpart2[(size_t)blockIdx.x * FIRE_SUMS + l] =
                (sh.a[1][0][l] + sh.a[1][1][l]) + (sh.a[1][2][l] + sh.a[1][3][l]);
        __threadfence();
    }
    __syncwarp();
    const uint32_t sN = sA + ((any2 && sA + 1u < d.nspec) ? 1u : 0u);
    for (uint32_t s = sA; s <= sN; ++s) {
        DevScalars* S = d.spec + s;
        const SpecGeom& G = d.geom[s];
        const uint32_t b0 = spec_first_cta(G, CTA), b1 = spec_last_cta(G, CTA);
        // the specimen's groups follow one another in the group arrays; consecutive specimens'
        // never meet (the +1 a specimen makes up for the rounding of b0 / FIRE_GROUP)
        const uint32_t g = (blockIdx.x - b0) / FIRE_GROUP, glast = (b1 - b0) / FIRE_GROUP;
        const size_t gbase = (size_t)s + b0 / FIRE_GROUP;
        const uint32_t first = b0 + g * FIRE_GROUP, count = min((uint32_t)FIRE_GROUP, b1 + 1u - first);
        if (!arrive_last(&d.fgrp_n[gbase + g], count)) continue;
        double v[FIRE_SUMS];
#pragma unroll
        for (int k = 0; k < FIRE_SUMS; ++k) v[k] = 0.0;
#pragma unroll
        for (uint32_t u = 0; u < FIRE_GROUP; u += 32u) {
            const uint32_t b = first + u + l;
            if (u + l >= count) continue;
            const double* src = (b * CTA >= G.p0 ? d.fpart : d.fpart2) + (size_t)b * FIRE_SUMS;
#pragma unroll
            for (int k = 0; k < FIRE_SUMS; ++k) v[k] += __ldcg(&src[k]);
        }
#pragma unroll
        for (int k = 0; k < FIRE_SUMS; ++k)
            for (int o = 16; o; o >>= 1) v[k] += __shfl_xor_sync(FULL, v[k], o);
        if (l == 0) d.fgrp_n[gbase + g] = 0u;
        if (glast) {                                 // (the sums of a single group are the specimen's)
            if (l == 0) {
#pragma unroll
                for (int k = 0; k < FIRE_SUMS; ++k) d.fgrp[(gbase + g) * FIRE_SUMS + k] = v[k];
                __threadfence();
            }
            __syncwarp();
            if (!arrive_last(&S->fcounter, glast + 1u)) continue;
#pragma unroll
            for (int k = 0; k < FIRE_SUMS; ++k) v[k] = 0.0;
            for (uint32_t q = l; q <= glast; q += 32u)
#pragma unroll
                for (int k = 0; k < FIRE_SUMS; ++k) v[k] += __ldcg(&d.fgrp[(gbase + q) * FIRE_SUMS + k]);
#pragma unroll
            for (int k = 0; k < FIRE_SUMS; ++k)
                for (int o = 16; o; o >>= 1) v[k] += __shfl_xor_sync(FULL, v[k], o);
        }
        if (l == 0 && !S->fstop) fire_decide(S, c, v, G.p1 - G.p0);
        bool running = false;
        if (l == 0) { S->fcounter = 0u; __threadfence(); }
        if (d.nspec > 1) {
            if (!arrive_last(&sc->spec_counter, d.nspec)) continue;
            for (uint32_t q = l; q < d.nspec; q += 32u) running = running || !__ldcg(&d.spec[q].fstop);
            running = __any_sync(FULL, running);
        }
        if (l == 0) {
            sc->spec_counter = 0u;
            sc->steps += 1;                     // buffer parity: the update works on what this pass wrote
            if (d.nspec > 1) sc->fstop = running ? 0u : 1u;      // (with one specimen sc == spec)
        }
    }
}

// State of the intact bond records at the end of an increment: each from its state at the
// increment's start, at the positions and rotations the specimen's last force pass read (the
// positions that pass wrote, less the platens' clamp). Once an increment instead of in every
// pass: 64 bytes a record written were a quarter of a pass's traffic.
template <int KIND>
__global__ void __launch_bounds__(128) k_fire_bond_state(Dev d, Consts c) {
    const uint32_t cur = (uint32_t)(d.sc->steps & 1ull);
    const double4* __restrict__ P = d.posd[cur];
    const uint32_t i = blockIdx.x * 128u + threadIdx.x;
    if (i >= c.N) return;
    auto read_at = [&](uint32_t q) {
        double4 x = ldg_d4(&P[q]);
        (KIND == RF_TEST_BRAZIL ? x.y : x.z) = d.xax[q];
        return x;
    };
    const double4 xi = read_at(i);
    uint32_t m = d.bmask[i];
    while (m) {
        const uint32_t q = __ffs(m) - 1u;
        m &= m - 1u;
        const size_t s = (size_t)q * c.N + i;
        const uint32_t j = d.bjk[s].x;
        float4 s0, s1, s2, kc;
        ld8(&d.rec0[s].s0, s0, s1);
        ld8(&d.rec0[s].s2, s2, kc);
        const double4 xj = read_at(j);
        const double3 rd = dsub(xj, xi);
        const double rr = dlen2(rd);
        BondExt b;
        b.kn = c.kn; b.ks = c.ks; b.br = c.br_lambda * fminf((float)xi.w, (float)xj.w);
        b.sc = kc.z; b.tc = kc.w; b.L0 = rec_L0(kc);
        f3 rij = mk3(s0.x, s0.y, s0.z), oijt = mk3(s0.w, s1.x, s1.y);
        f3 mijn = mk3(s1.z, s1.w, s2.x), mijt = mk3(s2.y, s2.z, s2.w), fr = mk3(0.f, 0.f, 0.f), mr = fr;
        float u0 = 0.f, u1 = 0.f, u2 = 0.f;
        fire_bond(d, b, i, j, mk3((float)rd.x, (float)rd.y, (float)rd.z), rd, rr, rij, oijt, mijn, mijt, fr, mr, u0, u1, u2);
        st8(&d.rec[s].s0, make_float4(rij.x, rij.y, rij.z, oijt.x), make_float4(oijt.y, oijt.z, mijn.x, mijn.y));
        st8(&d.rec[s].s2, make_float4(mijn.z, mijt.x, mijt.y, mijt.z), kc);
    }
}

// FIRE update of one iteration, in place on the buffers the force pass wrote:
// mixing (or, on uphill power, stop), then semi-implicit Euler in FP64
// positions; the rotation of the increment is accumulated for the warm-start data.
// (What does not depend on the loop state is loaded beside it.)
__global__ void __launch_bounds__(128) k_fire_update(Dev d, Consts c) {
    DevScalars* sc = d.sc;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = i < c.N;
    const uint32_t stop = sc->fstop, rebuild = sc->rebuild;
    const uint32_t cur = (uint32_t)(sc->steps & 1ull);
    float4 F = make_float4(0.f, 0.f, 0.f, 0.f), M = F, pr = F;
    double4 r = make_double4(0.0, 0.0, 0.0, 0.0);
    if (in) { F = d.frc[i]; M = d.mom[i]; pr = d.pos_ref[i]; r = d.rot[i]; }
    // the particle's specimen (a batch's specimens relax on their own FIRE scalars; one
    // whose relaxation stopped stays where it is)
    const DevScalars* S = d.spec;
    if (d.blk_spec) {
        const uint32_t sA = (uint32_t)d.blk_spec[blockIdx.x];
        S += (in && i >= d.geom[sA].p1) ? sA + 1u : sA;
    }
    const uint32_t ended = S->fstop, uphill = S->fuphill;
    const float dt = (float)S->fdt, cv = (float)S->fcv, cf = (float)S->fcf, cm = (float)S->fcm;
    if (c.fire_skip && rebuild) return;
    uint32_t moved = 0;
    float e2max = 0.f;
    if (!stop && in && !ended) {
        double4 x = d.posd[cur][i];
        float4 v = d.vw[cur][i].a, w = d.vw[cur][i].b;
        const double dtd = (double)dt;
        if (uphill) {
            // stop (no half step back: the bond and contact state integrates v dt, so every
            // position change must be a v dt of the force pass that follows)
            v = make_float4(0.f, 0.f, 0.f, 0.f);
            w = v;
        } else {
            v.x = cv * v.x + cf * F.x; v.y = cv * v.y + cf * F.y; v.z = cv * v.z + cf * F.z;
            w.x = cv * w.x + cm * M.x; w.y = cv * w.y + cm * M.y; w.z = cv * w.z + cm * M.z;
        }
        // stiffness-scaled (Jacobi) masses: every particle's own frequency is 1, so the
        // FIRE step is dimensionless and stiffness contrasts do not slow the relaxation
        const float dtm = dt / fmaxf(F.w, 1e-30f), dtI = dt / fmaxf(M.w, 1e-30f);
        v.x += F.x * dtm; v.y += F.y * dtm; v.z += F.z * dtm;
        w.x += M.x * dtI; w.y += M.y * dtI; w.z += M.z * dtI;
        x.x += (double)v.x * dtd; x.y += (double)v.y * dtd; x.z += (double)v.z * dtd;
        r.x += (double)w.x * dtd; r.y += (double)w.y * dtd; r.z += (double)w.z * dtd;
        d.rot[i] = r;
        d.posd[cur][i] = x;
        st8(&d.vw[cur][i], v, w);
        const float ex = (float)x.x - pr.x, ey = (float)x.y - pr.y, ez = (float)x.z - pr.z;
        const float e2 = ex * ex + ey * ey + ez * ez;
        moved = (e2 > c.disp2) ? 1u : 0u;
        if (e2 > c.hard2) raise_status(&d.sc->err, RF_ERR_CAPACITY);   // lists may have missed a neighbour
        e2max = e2;
    }
    __shared__ uint32_t s_m[4], s_e[4];
    const uint32_t wm = __reduce_or_sync(0xffffffffu, moved), we = __reduce_max_sync(0xffffffffu, __float_as_uint(e2max));
    if ((threadIdx.x & 31) == 0) { s_m[threadIdx.x >> 5] = wm; s_e[threadIdx.x >> 5] = we; }
    __syncthreads();
    if (threadIdx.x != 0) return;
    const uint32_t e2 = max(max(s_e[0], s_e[1]), max(s_e[2], s_e[3]));
    if (s_m[0] | s_m[1] | s_m[2] | s_m[3]) atomicOr(&sc->moved, 1u);
    if (e2) atomicMax(&sc->d2max_next, e2);
    __threadfence();
    if (atomicAdd(&sc->block_counter, 1u) != gridDim.x - 1) return;
    __threadfence();
    const uint32_t mv = __ldcg(&sc->moved), d2max = __ldcg(&sc->d2max_next);
    sc->block_counter = 0;
    // largest displacement since the last candidate build of the positions the next force
    // pass reads (this update wrote them): the force pass's add-pass scan skip uses it
    sc->dmax = sqrtf(__uint_as_float(d2max));
    sc->d2max_next = 0;
    sc->moved = 0;
    sc->rebuild = mv;
    if (c.use_graph) {
        cudaGraphSetConditional(c.h_rebuild, (mv && !stop) ? 1u : 0u);
        cudaGraphSetConditional(c.h_loop, stop ? 0u : 1u);
    }
}

// Start of a quasi-static load increment: advance the loading platen by the increment
// (CompressU / CompressB with V dt replaced by -delta), reset the FIRE state, start
// from rest, remember the start positions, and apply a warm start if given:
// warm[i*6 + 0..2] is added to the position, warm[i*6 + 3..5] / dt0 becomes the
// initial angular velocity (so the first iteration's bond and contact state advance
// by that rotation).
template <int KIND>
__global__ void k_qs_begin_scalars(Dev d, Consts c, double sinc) {
    const int ax = (KIND == RF_TEST_BRAZIL) ? 1 : 2;
    for (uint32_t sp = threadIdx.x; sp < d.nspec; sp += blockDim.x) {
        DevScalars* S = d.spec + sp;
        const double delta = sinc * S->Size0;      // the specimen's platen advance
        S->V = 0.0;
        S->size_d[ax] -= delta;
        S->Top -= delta;
        S->TopR = S->Top - 2.0 * c.p_r_d;
        S->size[ax] = (float)S->size_d[ax];
        S->sized2[ax] = (float)(0.5 * S->size_d[ax]);
        S->center_d[ax] -= delta;
        S->center[ax] = (float)S->center_d[ax];
        S->Hd2 = S->sized2[ax];
        S->Strain = (S->size_d[ax] - S->Size0) / S->Size0;
        S->fdt = S->fdt0;
        S->falpha = S->falpha0;
        S->fnpos = 0; S->fiter = 0; S->fuphill = 0; S->fconverged = 0; S->fstop = 0;
        S->fcv = 1.0; S->fcf = 0.0; S->fcm = 0.0;
        S->fwarm = 1;
        S->done = 0;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        DevScalars* sc = d.sc;     // (with one specimen sc == spec)
        sc->fstop = 0;
        sc->fcounter = 0;
        sc->done = 0;
        sc->dmax = 3.0e38f;        // the increment moves particles (platen, warm start): the first pass scans
        sc->d2max_next = 0;
        sc->rebuild = 1;          // positions jumped (platen clamp, warm start): rebuild the candidates
    }
}
template <int KIND>
__global__ void k_qs_begin(Dev d, Consts c, const float* __restrict__ warm, int ldw, int scaled, double sinc) {
    const DevScalars* sc = d.sc;
    const uint32_t cur = (uint32_t)(sc->steps & 1ull);
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;      // one particle per thread, 128-thread CTAs
    if (i >= c.N) return;
    const uint32_t sA = d.blk_spec ? (uint32_t)d.blk_spec[blockIdx.x] : 0u;
    const uint32_t sI = i >= d.geom[sA].p1 ? sA + 1u : sA;
    const DevScalars* S = d.spec + sI;
    const double zcut = (double)d.geom[sI].zcut;
    const float idt0 = (float)(1.0 / S->fdt0);
    const double D = sinc * S->Size0;                          // the specimen's platen advance
    const double Top = S->Top, Bottom = S->Bottom, TopR = S->TopR, BottomR = S->BottomR;
    const float RR = S->RR;
    rf_float3 cc;
    cc.x = S->center[0]; cc.y = S->center[1]; cc.z = S->center[2];
    {
        double4 x = d.posd[cur][i];
        d.x0[i] = x;
        float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
        float v0 = 0.f, v1 = 0.f, v2 = 0.f;
        double4 rot = make_double4(0.0, 0.0, 0.0, 0.0);
        if (warm) {
            // predicted displacement and rotation; as velocities over dt0 they make the first
            // force pass advance the bond and contact state by exactly that motion (the
            // first update then starts from rest)
            const float* q = warm + (size_t)i * ldw;
            float u[6];
            for (int a = 0; a < 6; ++a) u[a] = q[a];
            if (scaled) {                   // MLP units: displacement / D, rotation * r / D
                const float sd = (float)D, sr = (float)(D / x.w);
                u[0] *= sd; u[1] *= sd; u[2] *= sd; u[3] *= sr; u[4] *= sr; u[5] *= sr;
            }
            // a particle the platens held at the end of the last increment stays on its
            // platen (the top one has moved by D): the prediction's error along the load
            // axis must not lift it off
            const double off = x.w - c.p_r_d;
            const double a0 = KIND == RF_TEST_BRAZIL ? x.y : x.z;
            const float q0 = (float)(x.x - cc.x), q1 = KIND == RF_TEST_BRAZIL ? (float)(x.z - cc.z) : (float)(x.y - cc.y);
            const bool zone = q0 * q0 + q1 * q1 < RR && (KIND == RF_TEST_BRAZIL ? (double)(float)(x.z - cc.z) : a0) <
                                                          zcut;
            const bool at_top = zone && a0 + off - (Top + D) > -1e-9;
            const bool at_bottom = zone && a0 - off - Bottom < 1e-9;
            x.x += (double)u[0]; x.y += (double)u[1]; x.z += (double)u[2];
            v0 = u[0] * idt0; v1 = u[1] * idt0; v2 = u[2] * idt0;
            w = make_float4(u[3] * idt0, u[4] * idt0, u[5] * idt0, 0.f);
            rot = make_double4(u[3], u[4], u[5], 0.0);
            double& ax = KIND == RF_TEST_BRAZIL ? x.y : x.z;
            if (at_top) ax = Top - off;
            else if (at_bottom) ax = Bottom + off;
        }
        // the platen pushes the particles it passed: clamp them now, so the first force
        // pass (and its convergence test) sees the loaded configuration
        float f0 = 0.f, f1 = 0.f, f2 = 0.f;
        double sb = 0.0, st = 0.0;
        if (KIND == RF_TEST_BRAZIL)
            brazil_particle_ext(x.x, x.y, x.z, v0, v1, v2, f0, f1, f2, cc, RR, Top, Bottom, TopR, BottomR, 0.f,
                                zcut, x.w - c.p_r_d, sb, st, false);
        else
            uniaxial_particle_ext(x.x, x.y, x.z, v0, v1, v2, f0, f1, f2, cc, RR, Top, Bottom, TopR, BottomR, 0.f,
                                  zcut, x.w - c.p_r_d, sb, st, false);
        d.posd[cur][i] = x;
        st8(&d.vw[cur][i], make_float4(v0, v1, v2, 0.f), w);
        d.rot[i] = rot;
    }
}

// The specimen of particle i in a kernel of 128-thread CTAs, one particle per thread.
__device__ __forceinline__ const DevScalars* spec_of(const Dev& d, uint32_t i) {
    const uint32_t sA = d.blk_spec ? (uint32_t)d.blk_spec[blockIdx.x] : 0u;
    return d.spec + (i >= d.geom[sA].p1 ? sA + 1u : sA);
}

// Warm-start features of each particle from the last increment's motion (layout in the
// header); sinc = strain_inc, D = sinc * the specimen's initial size (its platen advance).
template <int KIND>
__global__ void k_warm_features(Dev d, Consts c, double sinc, __nv_bfloat16* __restrict__ feat) {
    const uint32_t cur = (uint32_t)(d.sc->steps & 1ull);
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.N) return;
    const DevScalars* sc = spec_of(d, i);
    const double D = sinc * sc->Size0;
    const int ax = (KIND == RF_TEST_BRAZIL) ? 1 : 2;
    const double iD = 1.0 / D;
    const double4 x = d.posd[cur][i], x0 = d.x0[i], r = d.rot[i];
    float f[64];
#pragma unroll
    for (int q = 0; q < 64; ++q) f[q] = 0.f;
    const double dxi = x.x - x0.x, dyi = x.y - x0.y, dzi = x.z - x0.z;
    f[0] = (float)(dxi * iD); f[1] = (float)(dyi * iD); f[2] = (float)(dzi * iD);
    f[3] = (float)(r.x * x.w * iD); f[4] = (float)(r.y * x.w * iD); f[5] = (float)(r.z * x.w * iD);
    const double p[3] = {x.x - sc->center_d[0], x.y - sc->center_d[1], x.z - sc->center_d[2]};
    f[6] = (float)(p[ax] / (0.5 * sc->size_d[ax]));
    const double o0 = p[ax == 2 ? 0 : 0], o1 = p[ax == 2 ? 1 : 2];
    f[7] = (float)(sqrt(o0 * o0 + o1 * o1) / (0.5 * sc->size_d[0]));
    const uint32_t bm = d.bmask[i], nq = d.nbq[i];
    int nb = 0;
    for (uint32_t q = 0; q < nq && nb < 12; ++q) {
        if (!((bm >> q) & 1u)) continue;
        const size_t s = (size_t)q * c.N + i;
        const uint32_t j = d.bjk[s].x;
        const double4 xj = d.posd[cur][j], xj0 = d.x0[j];
        const double ex = (xj.x - xj0.x) - dxi, ey = (xj.y - xj0.y) - dyi, ez = (xj.z - xj0.z) - dzi;
        const double rx = xj.x - x.x, ry = xj.y - x.y, rz = xj.z - x.z;
        const double L0 = rec_L0(d.rec[s].k);
        float* g = f + 8 + 4 * nb;
        g[0] = (float)(ex * iD); g[1] = (float)(ey * iD); g[2] = (float)(ez * iD);
        g[3] = (float)((sqrt(rx * rx + ry * ry + rz * rz) - L0) / (L0 * sinc));
        ++nb;
    }
    f[56] = (float)nb * (1.0f / 12.0f);
    const double xa = ax == 1 ? x.y : x.z, off = x.w - c.p_r_d;
    f[57] = (xa + off - sc->Top > -1e-9 || xa - off - sc->Bottom < 1e-9) ? 1.f : 0.f;
    f[58] = 1.f;
    uint4* out = reinterpret_cast<uint4*>(feat + (size_t)i * 64);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        __nv_bfloat162 h0 = __floats2bfloat162_rn(f[8 * q + 0], f[8 * q + 1]);
        __nv_bfloat162 h1 = __floats2bfloat162_rn(f[8 * q + 2], f[8 * q + 3]);
        __nv_bfloat162 h2 = __floats2bfloat162_rn(f[8 * q + 4], f[8 * q + 5]);
        __nv_bfloat162 h3 = __floats2bfloat162_rn(f[8 * q + 6], f[8 * q + 7]);
        uint4 u;
        u.x = *reinterpret_cast<uint32_t*>(&h0); u.y = *reinterpret_cast<uint32_t*>(&h1);
        u.z = *reinterpret_cast<uint32_t*>(&h2); u.w = *reinterpret_cast<uint32_t*>(&h3);
        out[q] = u;
    }
}

// Targets of the last increment: displacement / D and rotation * r / D.
__global__ void k_warm_targets(Dev d, Consts c, double sinc, float* __restrict__ t) {
    const uint32_t cur = (uint32_t)(d.sc->steps & 1ull);
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.N) return;
    const double D = sinc * spec_of(d, i)->Size0;
    const double iD = 1.0 / D;
    const double4 x = d.posd[cur][i], x0 = d.x0[i], r = d.rot[i];
    float* o = t + (size_t)i * 6;
    o[0] = (float)((x.x - x0.x) * iD); o[1] = (float)((x.y - x0.y) * iD); o[2] = (float)((x.z - x0.z) * iD);
    o[3] = (float)(r.x * x.w * iD); o[4] = (float)(r.y * x.w * iD); o[5] = (float)(r.z * x.w * iD);
}

// Start positions of the first increment: x0 = x, no rotation.
__global__ void k_fire_buffers_init(Dev d, Consts c) {
    const uint32_t cur = (uint32_t)(d.sc->steps & 1ull);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < c.N; i += gridDim.x * blockDim.x) {
        d.x0[i] = d.posd[cur][i];
        d.rot[i] = make_double4(0.0, 0.0, 0.0, 0.0);
    }
}

// Sets the FIRE loop's graph conditions at the start of a launch.
__global__ void k_fire_prologue(Dev d, Consts c) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        DevScalars* sc = d.sc;
        const bool go = !sc->fstop;
        cudaGraphSetConditional(c.h_rebuild, (go && sc->rebuild) ? 1u : 0u);
        cudaGraphSetConditional(c.h_loop, go ? 1u : 0u);
    }
}

// Sets both graph conditions at the start of a launch.
__global__ void k_prologue(Dev d, Consts c) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        DevScalars* sc = d.sc;
        const bool go = !sc->done && sc->steps < sc->target;
        if (c.use_graph) {
            cudaGraphSetConditional(c.h_rebuild, (go && sc->rebuild) ? 1u : 0u);
            cudaGraphSetConditional(c.h_loop, go ? 1u : 0u);
        }
    }
}

// On a plain stream: stop once the target step count is reached.
__global__ void k_stream_gate(Dev d) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        DevScalars* sc = d.sc;
        if (sc->steps >= sc->target) sc->done = sc->done | 2u;
    }
}
__global__ void k_stream_ungate(Dev d) {
    if (threadIdx.x == 0 && blockIdx.x == 0) d.sc->done &= 1u;
}

// ---------------------------------------------------------------------------
// Layout conversion (reference layout <-> engine layout)
// ---------------------------------------------------------------------------
// (stride: float4 records a particle, 2 for the velocities and spins)
__global__ void k_planar_to_f4(const float* __restrict__ R, uint32_t N, float4* __restrict__ out, uint32_t stride) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x)
        out[(size_t)i * stride] = make_float4(R[i], R[i + N], R[i + 2 * (size_t)N], 0.f);
}
__global__ void k_f4_to_planar(const float4* __restrict__ in, uint32_t N, float* __restrict__ R, uint32_t stride) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
        const float4 v = in[(size_t)i * stride];
        R[i] = v.x; R[i + N] = v.y; R[i + 2 * (size_t)N] = v.z;
    }
}

// Bond records a reference-layout row needs: its intact bonds, and broken bonds that
// still carry a bond direction (Rij is kept until the slot is deleted).
__device__ __forceinline__ bool needs_record(uint8_t type, const rf_float3 r) {
    return type == 1 || r.x != 0.f || r.y != 0.f || r.z != 0.f;
}

__global__ void k_count_records(const uint_fast32_t* __restrict__ IL, const uint8_t* __restrict__ type,
                                const rf_float3* __restrict__ Rij, uint32_t N, uint32_t K, uint32_t* maxq) {
    const uint_fast32_t E = empty_id<uint_fast32_t>();
    uint32_t m = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
        uint32_t n = 0;
        for (uint32_t k = 0; k < K; ++k) {
            const size_t r = (size_t)i * K + k;
            if (IL[r] != E && IL[r] < N && needs_record(type[r], Rij[r])) ++n;
        }
        m = max(m, n);
    }
    atomicMax(maxq, m);
}

// Reference-layout rows (uint_fast32_t ids, AoS float3 state) -> engine rows and records.
__global__ void k_rows_import(const uint_fast32_t* __restrict__ IL, const uint8_t* __restrict__ type,
                              const float* __restrict__ iL, const rf_float3* __restrict__ Rij,
                              const rf_float3* __restrict__ Oijt, const rf_float3* __restrict__ Mijn,
                              const rf_float3* __restrict__ Mijt, Dev d, Consts c) {
    const uint_fast32_t E = empty_id<uint_fast32_t>();
    const uint32_t cur = (uint32_t)(d.sc->steps & 1ull);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < c.N; i += gridDim.x * blockDim.x) {
        uint32_t live = 0, bond = 0, cm = 0, nq = 0, bmask = 0;
        for (uint32_t k = 0; k < c.K; ++k) {
            const size_t r = (size_t)i * c.K + k, s = (size_t)k * c.N + i;
            const uint_fast32_t j = IL[r];
            const bool ok = (j != E && j < c.N);
            d.ids[r] = ok ? (uint32_t)j : EMPTY32;
            d.il[s] = iL[r];
            const bool t1 = ok && type[r] == 1;
            float* co = d.cO[cur] + 3 * r;
            co[0] = t1 ? 0.f : Oijt[r].x; co[1] = t1 ? 0.f : Oijt[r].y; co[2] = t1 ? 0.f : Oijt[r].z;
            if (!ok) continue;
            live |= 1u << k;
            if (t1) bond |= 1u << k;
            else if (Oijt[r].x != 0.f || Oijt[r].y != 0.f || Oijt[r].z != 0.f) cm |= 1u << k;
            if (needs_record(type[r], Rij[r]) && nq < d.QB) {
                const size_t b = (size_t)nq * c.N + i;
                d.bjk[b] = make_uint2((uint32_t)j, k);
                const float ox = t1 ? Oijt[r].x : 0.f, oy = t1 ? Oijt[r].y : 0.f, oz = t1 ? Oijt[r].z : 0.f;
                st8(&d.rec[b].s0, make_float4(Rij[r].x, Rij[r].y, Rij[r].z, ox), make_float4(oy, oz, Mijn[r].x, Mijn[r].y));
                st8(&d.rec[b].s2, make_float4(Mijn[r].z, Mijt[r].x, Mijt[r].y, Mijt[r].z),
                    make_float4(iL[r], 0.f, 0.f, 0.f));
                if (t1) bmask |= 1u << nq;
                ++nq;
            }
        }
        for (uint32_t q = nq; q < d.QB; ++q) {          // unused records: retired, zero
            const size_t b = (size_t)q * c.N + i;
            d.bjk[b] = make_uint2(0u, 0xFFu);
            d.rec[b].k = make_float4(0.f, 0.f, 0.f, 0.f);
            zero_record(d, b);
        }
        d.live[i] = live; d.bond[i] = bond; d.cmask[i] = cm; d.nbq[i] = nq; d.bmask[i] = bmask;
    }
}

__global__ void k_rows_export(uint_fast32_t* __restrict__ IL, uint8_t* __restrict__ type, float* __restrict__ iL,
                              rf_float3* __restrict__ Rij, rf_float3* __restrict__ Oijt, rf_float3* __restrict__ Mijn,
                              rf_float3* __restrict__ Mijt, Dev d, Consts c) {
    const uint_fast32_t E = empty_id<uint_fast32_t>();
    const uint32_t cur = (uint32_t)(d.sc->steps & 1ull);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < c.N; i += gridDim.x * blockDim.x) {
        const uint32_t live = d.live[i], bond = d.bond[i], nq = d.nbq[i];
        for (uint32_t k = 0; k < c.K; ++k) {
            const size_t r = (size_t)i * c.K + k, s = (size_t)k * c.N + i;
            IL[r] = ((live >> k) & 1u) ? (uint_fast32_t)d.ids[r] : E;
            type[r] = (uint8_t)((bond >> k) & 1u);
            iL[r] = d.il[s];
            Rij[r].x = 0.f; Rij[r].y = 0.f; Rij[r].z = 0.f;
            Mijn[r] = Rij[r]; Mijt[r] = Rij[r];
            const bool has = ((d.cmask[i] >> k) & 1u) != 0;
            const float* co = d.cO[cur] + 3 * r;
            Oijt[r].x = has ? co[0] : 0.f; Oijt[r].y = has ? co[1] : 0.f; Oijt[r].z = has ? co[2] : 0.f;
        }
        for (uint32_t q = 0; q < nq; ++q) {
            const size_t b = (size_t)q * c.N + i;
            const uint32_t k = d.bjk[b].y;
            if (k == 0xFFu) continue;
            const size_t r = (size_t)i * c.K + k;
            const float4 s0 = d.rec[b].s0, s1 = d.rec[b].s1, s2 = d.rec[b].s2;
            Rij[r].x = s0.x; Rij[r].y = s0.y; Rij[r].z = s0.z;
            Mijn[r].x = s1.z; Mijn[r].y = s1.w; Mijn[r].z = s2.x;
            Mijt[r].x = s2.y; Mijt[r].y = s2.z; Mijt[r].z = s2.w;
            if ((bond >> k) & 1u) { Oijt[r].x = s0.w; Oijt[r].y = s1.x; Oijt[r].z = s1.y; }
        }
    }
}

// Bond construction of the extended model: slot (i, k) -> j becomes a bond when the
// gap |r_ij| - r_i - r_j is below gap_frac * min(r_i, r_j) (distances in double). The
// rest length is |r_ij| in double; tensile and shear strengths are Weibull draws
// scale * (-ln U)^(1/m) keyed on the unordered pair, so both directed slots of a pair
// share them. The slot state starts at zero, as d_ConstructBoundInteractions leaves it.
__device__ __forceinline__ uint64_t mix64(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
__device__ __forceinline__ double pair_uniform(uint64_t seed, uint32_t a, uint32_t b, uint32_t stream) {
    const uint64_t lo = a < b ? a : b, hi = a < b ? b : a;
    const uint64_t h = mix64(mix64(seed ^ (0x51ED270B27F3A4C1ull * (stream + 1))) + (hi << 32 | lo));
    return ((double)(h >> 11) + 0.5) * (1.0 / 9007199254740992.0);       // in (0, 1)
}
// Bond rule and strength distribution of one specimen of a batch.
struct BondSpec {
    double gap_frac, wm, sig, tau;
    uint64_t seed;
    uint32_t p0, p1;            // its particles
    int ref_mode;               // reference constants: bonds below the centre distance bd, strengths sig, tau
    double bd;
};
// Initial rows of an engine, in the reference's construction order (md_interaction_list_
// construct.cu:13-98: the 8 octant cells in visiting order, their occupants in cell order, slots
// filled in order), by eight lanes a particle as md_InteractionListConstruct builds them, but
// straight into the engine's rows. gap < 0: pairs with float |r|^2 < aacut (the reference's
// test); else the extended model's pair test |r| < min(a_farcut, r_i + r_j + gap) on the FP64
// positions. Nothing of a row exists in the reference layout in between: seven FP32 triples a
// slot, their zeroing and about 60 allocations were most of a creation. Creation, an affine
// strain, 100 steps and the read-back of 200k particles: 43 -> 15 ms (with the faster steps).
__global__ void __launch_bounds__(128) k_rows_list(const float* __restrict__ R, Dev d, Consts c,
                                                   const uint_fast32_t* __restrict__ CIs,
                                                   const uint_fast32_t* __restrict__ pnC, double a_farcut, double gap,
                                                   uint32_t* err) {
    const size_t N = c.N;
    const int sub = threadIdx.x & 7;
    const size_t i = (size_t)blockIdx.x * 16 + (threadIdx.x >> 3);
    const bool valid = i < N;
    f3 xi = mk3(0.f, 0.f, 0.f);
    double4 xd = make_double4(0, 0, 0, 0);
    uint64_t s = 0, cnt = 0;
    if (valid) {
        xi = mk3(R[i], R[i + N], R[i + 2 * N]);
        if (gap >= 0.0) xd = d.posd[0][i];
        const int64_t cell = octant_cell(octant_of(xi, c.g), sub);
        if (cell < 0 || (uint64_t)cell >= c.g.CN) raise_status(err, RF_ERR_CELL_RANGE);
        else { s = (uint64_t)pnC[cell]; cnt = (uint64_t)pnC[cell + c.g.CN]; }
        if (s > N) s = N;
        if (cnt > N - s) cnt = N - s;
    }
    auto hit = [&](uint64_t m, uint32_t& j) {
        const uint_fast32_t id = CIs[s + m + N];
        if (id >= N || id == i) return false;
        j = (uint32_t)id;
        if (gap >= 0.0) {
            const double4 xj = ldg_d4(&d.posd[0][j]);
            const double q = fmin(a_farcut, (xd.w + xj.w) + gap);
            return dlen2(dsub(xj, xd)) < q * q;
        }
        return dist2_rn(xi, mk3(R[j], R[j + N], R[j + 2 * N])) < c.aacut;
    };
    uint32_t n = 0, j = 0;
    for (uint64_t m = 0; m < cnt; ++m) n += hit(m, j) ? 1u : 0u;
    uint32_t at = n;
    for (int o = 1; o < 8; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, at, o, 8);
        if (sub >= o) at += y;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, at, 7, 8);
    at -= n;
    if (!valid) return;
    uint32_t* row = d.ids + i * c.K;
    if (n && at + n > c.K) raise_status(err, RF_ERR_ROW_OVERFLOW);
    for (uint64_t m = 0; n && m < cnt; ++m)
        if (hit(m, j)) {
            if (at < c.K) row[at] = j;
            ++at; --n;
        }
    const uint32_t held = min(total, c.K);       // (the row is cut at K: the mask has no slot beyond it)
    for (uint32_t k = held + sub; k < c.K; k += 8) row[k] = EMPTY32;
    if (sub == 0) d.live[i] = held >= 32u ? 0xffffffffu : (1u << held) - 1u;
}

// Bonds of the rows, a warp a particle and a lane a slot. Reference model: pairs below the
// squared length aa_create, 1/L0 = rsqrt(|r|^2) (md_boundinteractions_construct.cu). Extended
// model: gap below gap_frac * min(r_i, r_j) (or, in the reference-constants mode, centre
// distance below b_d), with the FP64 rest length and the pair's strengths. aa_far > 0: then
// DeleteFarLinks on the float positions, as the drivers run it before their first step.
// PASS 0 finds the rows' bonds and the most of any row (the record planes to allocate); PASS 1
// writes the records, the per-slot 1/L0 and the particles' masks.
template <int PASS>
__global__ void __launch_bounds__(128) k_rows_bonds(const float* __restrict__ R, Dev d, Consts c, float aa_create, float aa_far,
                                                    const BondSpec* __restrict__ bs, uint32_t nspec, uint32_t* maxq) {
    __shared__ float s_il[32][33];
    const uint32_t FULL = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31u, wp = threadIdx.x >> 5;
    const size_t N = c.N, i0 = (size_t)blockIdx.x * 32;
    uint32_t most = 0;
    for (uint32_t u = wp; u < 32u; u += 4u) {
        const size_t i = i0 + u;
        float il = 0.f;
        if (i < N) {
            const f3 xi = mk3(R[i], R[i + N], R[i + 2 * N]);
            uint32_t live = d.live[i];
            const bool occ = lane < c.K && ((live >> lane) & 1u);
            const uint32_t j = occ ? d.ids[i * c.K + lane] : 0u;
            bool bond = false, far = false;
            double L = 1.0;
            float2 str = make_float2(0.f, 0.f);
            if (occ) {
                const f3 xj = mk3(R[j], R[j + N], R[j + 2 * N]);
                if (c.ext) {
                    uint32_t sp = 0;
                    while (sp + 1 < nspec && i >= bs[sp].p1) ++sp;
                    const BondSpec& B = bs[sp];
                    const double4 a = ldg_d4(&d.posd[0][i]), b = ldg_d4(&d.posd[0][j]);
                    const double dx = b.x - a.x, dy = b.y - a.y, dz = b.z - a.z;
                    const double len = sqrt(dx * dx + dy * dy + dz * dz);
                    // md_boundinteractions_construct.cu:62 on the FP64 distance in the reference-constants mode
                    bond = (B.ref_mode ? len < B.bd : len - a.w - b.w < B.gap_frac * fmin(a.w, b.w)) && len > 0;
                    if (bond) {
                        il = (float)(1.0 / len);
                        L = len;
                        if (PASS == 1) {
                            if (B.ref_mode) {
                                str = make_float2((float)B.sig, (float)B.tau);
                            } else {
                                // strengths keyed on specimen-local ids
                                const double inv_m = 1.0 / B.wm;
                                const uint32_t li = (uint32_t)i - B.p0, lj = j - B.p0;
                                const double us = pair_uniform(B.seed, li, lj, 0), ut = pair_uniform(B.seed, li, lj, 1);
                                str = make_float2((float)(B.sig * pow(-log(us), inv_m)), (float)(B.tau * pow(-log(ut), inv_m)));
                            }
                        }
                    }
                } else {
                    const float rm2 = rm2_bond(xj.x - xi.x, xj.y - xi.y, xj.z - xi.z);
                    bond = rm2 < aa_create && (double)rm2 > 1e-18;
                    if (bond) il = __frsqrt_rn(rm2);
                }
                if (aa_far > 0.f) {
                    const float rr = dist2_rn(xi, xj);
                    far = rr > aa_far || below_1em10(rr);
                }
            }
            const uint32_t bm = __ballot_sync(FULL, bond && !far), fm = __ballot_sync(FULL, far);
            const uint32_t nq = __popc(bm);
            most = max(most, nq);
            if (PASS == 1) {
                if (far) d.ids[i * c.K + lane] = EMPTY32;
                if ((bm >> lane) & 1u) {
                    const size_t b = (size_t)__popc(bm & ((1u << lane) - 1u)) * N + i;
                    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
                    d.bjk[b] = make_uint2(j, lane);
                    st8(&d.rec[b].s0, z, z);
                    st8(&d.rec[b].s2, z, c.ext ? rec_const(L, str) : make_float4(il, 0.f, 0.f, 0.f));
                }
                for (uint32_t q = nq + lane; q < d.QB; q += 32u) {         // unused records: retired, zero
                    const size_t b = (size_t)q * N + i;
                    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
                    d.bjk[b] = make_uint2(0u, 0xFFu);
                    st8(&d.rec[b].s0, z, z);
                    st8(&d.rec[b].s2, z, c.ext ? rec_const(1.0, make_float2(0.f, 0.f)) : z);
                }
                if (lane == 0) {
                    live &= ~fm;
                    d.live[i] = live; d.bond[i] = bm; d.cmask[i] = 0u; d.nbq[i] = nq;
                    d.bmask[i] = nq >= 32u ? 0xffffffffu : (1u << nq) - 1u;
                }
            }
        }
        if (PASS == 1) s_il[u][lane] = il;
    }
    if (PASS == 0) {
        if (lane == 0 && most > *(volatile uint32_t*)maxq) atomicMax(maxq, most);
        return;
    }
    __syncthreads();
    for (uint32_t k = wp; k < c.K; k += 4u)
        if (i0 + lane < N) d.il[(size_t)k * N + i0 + lane] = s_il[lane][k];
}
__global__ void k_posd_from_planar(const double* __restrict__ R, const double* __restrict__ rad, uint32_t N,
                                   double4* __restrict__ out, float* __restrict__ Rf) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
        const double x = R[i], y = R[i + N], z = R[i + 2 * (size_t)N];
        out[i] = make_double4(x, y, z, rad[i]);
        if (Rf) { Rf[i] = (float)x; Rf[i + N] = (float)y; Rf[i + 2 * (size_t)N] = (float)z; }
    }
}
__global__ void k_posd_to_planar(const double4* __restrict__ in, uint32_t N, double* __restrict__ R) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
        const double4 v = in[i];
        R[i] = v.x; R[i + N] = v.y; R[i + 2 * (size_t)N] = v.z;
    }
}
__global__ void k_posd_to_planar_f(const double4* __restrict__ in, uint32_t N, float* __restrict__ R) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
        const double4 v = in[i];
        R[i] = (float)v.x; R[i + N] = (float)v.y; R[i + 2 * (size_t)N] = (float)v.z;
    }
}

__global__ void k_counters(Dev d, Consts c, unsigned long long* out) {
    uint32_t nb = 0, nc = 0, nl = 0;              // (a warp's share: below 2^32)
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < c.N; i += gridDim.x * blockDim.x) {
        nl += __popc(d.live[i]); nb += __popc(d.bond[i]); nc += __popc(d.cmask[i]);
    }
    nb = __reduce_add_sync(0xffffffffu, nb); nc = __reduce_add_sync(0xffffffffu, nc); nl = __reduce_add_sync(0xffffffffu, nl);
    if ((threadIdx.x & 31) == 0) {
        if (nb) atomicAdd(&out[0], (unsigned long long)nb);
        if (nc) atomicAdd(&out[1], (unsigned long long)nc);
        if (nl) atomicAdd(&out[2], (unsigned long long)nl);
    }
}

__global__ void k_set_target(DevScalars* sc, unsigned long long n) { sc->target = sc->steps + n; }
__global__ void k_force_rebuild(DevScalars* sc) { sc->rebuild = 1u; }

// Homogeneous strain of the specimen about the platen box's centre: every position (and
// the load axis's platens with them) scaled by 1 + eps per axis; the platen zone's radius
// grows with the larger lateral strain. Rest lengths, slot state and velocities stay, so
// the bonds and contacts carry the strain from the next step on.
__global__ void k_affine_positions(Dev d, Consts c, double ex, double ey, double ez) {
    const uint32_t cur = (uint32_t)(d.sc->steps & 1ull);
    const double cx = d.sc->center_d[0], cy = d.sc->center_d[1], cz = d.sc->center_d[2];
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < c.N; i += gridDim.x * blockDim.x) {
        if (c.ext) {
            double4 x = d.posd[cur][i];
            x.x = cx + (1.0 + ex) * (x.x - cx); x.y = cy + (1.0 + ey) * (x.y - cy); x.z = cz + (1.0 + ez) * (x.z - cz);
            d.posd[cur][i] = x;
        } else {
            float4 x = d.pos[cur][i];
            x.x = (float)(cx + (1.0 + ex) * ((double)x.x - cx));
            x.y = (float)(cy + (1.0 + ey) * ((double)x.y - cy));
            x.z = (float)(cz + (1.0 + ez) * ((double)x.z - cz));
            d.pos[cur][i] = x;
        }
    }
}
template <int KIND>
__global__ void k_affine_scalars(Dev d, Consts c, double ex, double ey, double ez) {
    DevScalars* sc = d.sc;
    if (blockIdx.x || threadIdx.x) return;
    const int ax = (KIND == RF_TEST_BRAZIL) ? 1 : 2;
    const double e = ax == 1 ? ey : ez, el = ax == 1 ? fmax(ex, ez) : fmax(ex, ey);
    const double ca = sc->center_d[ax];
    const double dtr = sc->TopR - sc->Top, dbr = sc->BottomR - sc->Bottom;
    sc->Top = ca + (1.0 + e) * (sc->Top - ca);
    sc->Bottom = ca + (1.0 + e) * (sc->Bottom - ca);
    sc->TopR = sc->Top + dtr;
    sc->BottomR = sc->Bottom + dbr;
    sc->size_d[ax] *= 1.0 + e;
    sc->size[ax] = (float)sc->size_d[ax];
    sc->sized2[ax] = (float)(0.5 * sc->size_d[ax]);
    sc->Hd2 = sc->sized2[ax];
    sc->Strain = (sc->size_d[ax] - sc->Size0) / sc->Size0;
    sc->RR = (float)((double)sc->RR * (1.0 + el) * (1.0 + el));
    sc->dmax = 3.0e38f;          // positions jumped: the next add pass scans
    sc->d2max_next = 0;
    sc->rebuild = 1;             // and the candidate lists are rebuilt first
}
__global__ void k_planar_to_cur(const float* __restrict__ R, Dev d) {
    const uint32_t N = (uint32_t)(d.n_particles);
    if (d.posd[0]) {                      // extended model: keep the radius
        double4* out = d.posd[d.sc->steps & 1ull];
        for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x)
            out[i] = make_double4(R[i], R[i + N], R[i + 2 * (size_t)N], out[i].w);
    } else {
        float4* out = d.pos[d.sc->steps & 1ull];
        for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x)
            out[i] = make_float4(R[i], R[i + N], R[i + 2 * (size_t)N], 0.f);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) d.sc->rebuild = 1u;
}
__global__ void k_cur_to_planar(Dev d, float* __restrict__ R) {
    const uint32_t N = (uint32_t)(d.n_particles);
    if (d.posd[0]) {
        const double4* in = d.posd[d.sc->steps & 1ull];
        for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
            const double4 v = in[i];
            R[i] = (float)v.x; R[i + N] = (float)v.y; R[i + 2 * (size_t)N] = (float)v.z;
        }
        return;
    }
    const float4* in = d.pos[d.sc->steps & 1ull];
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
        const float4 v = in[i];
        R[i] = v.x; R[i + N] = v.y; R[i + 2 * (size_t)N] = v.z;
    }
}

}  // namespace rf

using namespace rf;

struct rf_engine {
    rf_task task;
    Dev d;
    Consts c;
    int device;
    cudaStream_t stream;
    cudaGraph_t graph;
    cudaGraphExec_t exec;
    uint32_t nblocks;                      // 128-particle blocks of the per-particle kernels
    int pw = 32;                           // particles a warp of the step kernel takes
    uint32_t ncta;                         // CTAs of the step kernel (4 warps each)
    uint32_t cg_nb;
    bool graph_ok;
    std::vector<void*> allocs;
    std::vector<size_t> alloc_bytes;
    int step_minb = RF_STEP_MIN_BLOCKS;    // register-cap variant of the extended step (autotuned)
    unsigned long long* counters_dev;
    float* staging;
    uint64_t bonds_initial;
    uint32_t* maxq_dev;
    // batch of specimens
    std::vector<rf_task> spec_tasks;   // per specimen, shifted, with the batch's cell grid
    std::vector<uint32_t> spec_p0, spec_n;
    std::vector<double> spec_xoff;
    // FIRE relaxation graph (built on the first load increment)
    Consts cf;
    cudaGraph_t fgraph;
    cudaGraphExec_t fexec;
    bool fire_ready;
};

namespace {

// A set of device arrays in one allocation, each on a 256-byte boundary: an allocation and its
// free cost about 0.1 ms each, and an engine has some sixty arrays.
struct Arrays {
    std::vector<std::pair<void**, size_t>> list;
    size_t bytes = 0;
    template <class T> void add(T** p, size_t n) {
        list.push_back({(void**)p, bytes});
        bytes += ((n ? n : 1) * sizeof(T) + 255) / 256 * 256;
    }
    cudaError_t alloc(void** base) const {
        *base = nullptr;
        const cudaError_t ce = cudaMalloc(base, bytes);
        if (!ce) for (auto& a : list) *a.first = (char*)*base + a.second;
        return ce;
    }
};
// ... owned by an engine
rf_status dalloc(rf_engine* e, const Arrays& a) {
    void* q = nullptr;
    RF_CUDA(a.alloc(&q));
    e->allocs.push_back(q);
    e->alloc_bytes.push_back(a.bytes);
    return RF_OK;
}

// Rows in the reference layout, for a read-out or an import (released with the object).
struct RowBuffers {
    uint_fast32_t* IL = nullptr;
    uint8_t* type = nullptr;
    float* iL = nullptr;
    rf_float3* S = nullptr;                  // Rij, Oijt, Mijn, Mijt, NK each
    void* base = nullptr;
    cudaError_t alloc(size_t NK) {
        Arrays A;
        A.add(&IL, NK); A.add(&type, NK); A.add(&iL, NK); A.add(&S, 4 * NK);
        return A.alloc(&base);
    }
    ~RowBuffers() { cudaFree(base); }
};

#define TRY(x) do { rf_status s__ = (x); if (s__ != RF_OK) return s__; } while (0)

// Explicit extended-model step kernels: compiled for 5, 6 and 8 CTAs per SM at 32 particles a
// warp (96, 80 and 64 registers), for 6 alone with fewer (80 registers, 164 to 172 bytes of
// spill stores), where minb has no effect.
template <int KIND>
void* ext_step_kind(int pw, int minb) {
    switch (pw) {
        case 4: return (void*)k_step_ext<KIND, 0, RF_STEP_MIN_BLOCKS, 4>;
        case 8: return (void*)k_step_ext<KIND, 0, RF_STEP_MIN_BLOCKS, 8>;
        case 16: return (void*)k_step_ext<KIND, 0, RF_STEP_MIN_BLOCKS, 16>;
    }
    return minb == 8 ? (void*)k_step_ext<KIND, 0, 8> : minb == 5 ? (void*)k_step_ext<KIND, 0, 5> : (void*)k_step_ext<KIND, 0, 6>;
}
void* ext_step_variant(const rf_engine* e, int minb) {
    return e->task.kind == RF_TEST_BRAZIL ? ext_step_kind<RF_TEST_BRAZIL>(e->pw, minb) : ext_step_kind<RF_TEST_UNIAXIAL>(e->pw, minb);
}
template <int KIND>
void* fire_force_kind(int pw) {
    switch (pw) {
        case 4: return (void*)k_step_ext<KIND, 1, RF_STEP_MIN_BLOCKS, 4>;
        case 8: return (void*)k_step_ext<KIND, 1, RF_STEP_MIN_BLOCKS, 8>;
        case 16: return (void*)k_step_ext<KIND, 1, RF_STEP_MIN_BLOCKS, 16>;
    }
    return (void*)k_step_ext<KIND, 1>;
}
void* fire_force_kernel(const rf_engine* e) {
    return e->task.kind == RF_TEST_BRAZIL ? fire_force_kind<RF_TEST_BRAZIL>(e->pw) : fire_force_kind<RF_TEST_UNIAXIAL>(e->pw);
}

// Particles a warp of the step kernels takes. While all CTAs of a step are resident at once
// the chain of a warp (its rounds and scans, one memory latency after another) is what a
// step waits for, and a warp of fewer particles has a shorter one; beyond that the step is a
// matter of throughput. 8 or 16 as long as their CTAs are resident together, 4 while they are
// at most three an SM. Measured, us per step at 4 / 8 / 16 / 32 particles a warp, extended
// model: 900 particles 19 / 21 / 24 / 31, 8k 22 / 23 / 27 / 35, 14k 26 / 25 / 29 / 36, 26k 40 / 30 / 32 /
// 40, 40k 55 / 44 / 35 / 42, 55k 70 / 48 / 38 / 44, 70k 87 / 63 / 57 / 48; reference model: 570
// particles 16 / 18 / 21 / 23, 4.6k 17 / 18 / 22 / 27, 17k 28 / 22 / 24 / 28, 36k 41 / 35 / 28 / 32.
int particles_per_warp(uint32_t N, int sms) {
    const uint64_t resident = (uint64_t)sms * RF_STEP_MIN_BLOCKS * 4u;      // warps
    return N <= 4u * (uint64_t)sms * 3u * 4u ? 4 : N <= 8u * resident ? 8 : N <= 16u * resident ? 16 : 32;
}

// dynamic shared memory of a step launch: the per-warp record list (pw particles x QB
// records, 2 bytes each, 4 warps)
unsigned step_smem(const rf_engine* e) { return 4u * (unsigned)e->pw * e->d.QB * 2u; }

template <int KIND>
void* ref_step_kind(int pw) {
    return pw == 4 ? (void*)k_step<KIND, 4> : pw == 8 ? (void*)k_step<KIND, 8> : pw == 16 ? (void*)k_step<KIND, 16> : (void*)k_step<KIND, 32>;
}
void* step_kernel(const rf_engine* e) {
    if (e->c.ext) return ext_step_variant(e, e->step_minb);
    return e->task.kind == RF_TEST_BRAZIL ? ref_step_kind<RF_TEST_BRAZIL>(e->pw) : ref_step_kind<RF_TEST_UNIAXIAL>(e->pw);
}

rf_status build_graph(rf_engine* e) {
    cudaGraph_t g;
    RF_CUDA(cudaGraphCreate(&g, 0));
    e->graph = g;
    // The loop body is RF_GRAPH_UNROLL steps, each preceded by IF(rebuild) {rebuild
    // kernels} or, for specimens below RF_REBUILD_EACH_STEP_N particles, only the first:
    // there a conditional node costs as much as a few percent of a step, and the rebuild
    // condition is evaluated once per RF_GRAPH_UNROLL steps. The rebuild trigger is set at
    // 0.3 of the skin so that the particles' motion until the next evaluation stays within
    // the 0.5 skin the candidate lists are complete for; a step that finds a particle beyond
    // 0.5 skin reports RF_ERR_CAPACITY. Evaluating before every step lets particles move 0.2
    // skin per step (fragments of a damaged large specimen), against 0.2 skin per
    // RF_GRAPH_UNROLL steps otherwise. Each IF node has its own conditional handle (a handle
    // drives one conditional node); a step node's parameters carry the handle of the IF
    // node after it (the last step's: the body's first IF, evaluated on the next iteration),
    // the prologue's the first. The WHILE condition is evaluated once per body. A step
    // whose step count has reached the target returns at once, so the target is kept exactly.
    const int every = e->c.N >= RF_REBUILD_EACH_STEP_N ? 1 : RF_GRAPH_UNROLL;
    const int nif = RF_GRAPH_UNROLL / every;
    cudaGraphConditionalHandle hif[RF_GRAPH_UNROLL];
    RF_CUDA(cudaGraphConditionalHandleCreate(&e->c.h_loop, g, 0, 0));
    for (int q = 0; q < nif; ++q) RF_CUDA(cudaGraphConditionalHandleCreate(&hif[q], g, 0, 0));
    e->c.h_rebuild = hif[0];
    e->c.use_graph = 1;
    Dev d = e->d;
    Consts c = e->c;
    void* args[] = {&d, &c};
    auto kparams = [&](void* fn, unsigned grid, unsigned block, void** a) {
        cudaKernelNodeParams kp = {};
        kp.func = fn; kp.gridDim = dim3(grid); kp.blockDim = dim3(block);
        kp.sharedMemBytes = 0; kp.kernelParams = a; kp.extra = nullptr;
        return kp;
    };
    // prologue -> WHILE
    cudaGraphNode_t pro;
    cudaKernelNodeParams kp = kparams((void*)k_prologue, 1, 32, args);
    RF_CUDA(cudaGraphAddKernelNode(&pro, g, nullptr, 0, &kp));
    cudaGraphNodeParams wp = {};
    wp.type = cudaGraphNodeTypeConditional;
    wp.conditional.handle = e->c.h_loop;
    wp.conditional.type = cudaGraphCondTypeWhile;
    wp.conditional.size = 1;
    cudaGraphNode_t wnode;
    RF_CUDA(cudaGraphAddNode(&wnode, g, &pro, 1, &wp));
    cudaGraph_t body = wp.conditional.phGraph_out[0];
    const unsigned gN = (e->c.N + 255) / 256;
    const unsigned gC = (e->c.cg_cells + 1 + 255) / 256;
    struct { void* fn; unsigned grid, block; } seq[] = {
        {(void*)k_rb_zero, gC, 256},      {(void*)k_rb_bin, gN, 256},
        {(void*)k_rb_scan_sums, e->cg_nb, 1024}, {(void*)k_rb_scan_totals, 1, 32},
        {(void*)k_rb_scan_apply, e->cg_nb, 1024}, {(void*)k_rb_scatter, gN, 256},
        {(void*)k_rb_cand, (e->c.N + RF_RB_CTA - 1) / RF_RB_CTA, RF_RB_CTA},
    };
    void* fn = step_kernel(e);
    // per step node: Consts with the handle of the IF node that follows it (node parameters
    // are copied when the node is added, so one slot per step suffices until then)
    Consts cs[RF_GRAPH_UNROLL];
    void* sargs[RF_GRAPH_UNROLL][2];
    cudaGraphNode_t last = nullptr;
    for (int u = 0; u < RF_GRAPH_UNROLL; ++u) {
        if (u % every == 0) {
            cudaGraphNodeParams ip = {};
            ip.type = cudaGraphNodeTypeConditional;
            ip.conditional.handle = hif[u / every];
            ip.conditional.type = cudaGraphCondTypeIf;
            ip.conditional.size = 1;
            cudaGraphNode_t inode;
            RF_CUDA(cudaGraphAddNode(&inode, body, last ? &last : nullptr, last ? 1 : 0, &ip));
            cudaGraph_t rb = ip.conditional.phGraph_out[0];
            cudaGraphNode_t prev = nullptr;
            for (auto& q : seq) {
                cudaGraphNode_t n;
                kp = kparams(q.fn, q.grid, q.block, args);
                RF_CUDA(cudaGraphAddKernelNode(&n, rb, prev ? &prev : nullptr, prev ? 1 : 0, &kp));
                prev = n;
            }
            last = inode;
        }
        cs[u] = c;
        cs[u].h_rebuild = hif[((u + 1) / every) % nif];
        sargs[u][0] = &d;
        sargs[u][1] = &cs[u];
        cudaGraphNode_t step;
        kp = kparams(fn, e->ncta, 128, sargs[u]);
        kp.sharedMemBytes = step_smem(e);
        RF_CUDA(cudaGraphAddKernelNode(&step, body, &last, 1, &kp));
        last = step;
    }
    RF_CUDA(cudaGraphInstantiate(&e->exec, g, 0));
    return RF_OK;
}

// FIRE loop graph: prologue -> WHILE(not stopped) { IF(moved) {candidate rebuild}; RF_GRAPH_UNROLL
// times forces, update }. A conditional node costs several microseconds, so the body holds more
// than one iteration; once an update finds that the candidates have to be rebuilt, the rest of the
// body leaves at once (fire_skip), and the rebuild precedes the next force pass as if every
// iteration had its IF. Six specimens of 3000 particles: 34.8 -> 28.8 us an iteration. An increment
// that stops inside a body still launches its other iterations, which leave at once: with 20k
// particles one iteration takes 297 us (237 with an IF each), 16 take as long as before, and
// from there on the longer body gains.
rf_status build_fire_graph(rf_engine* e) {
    cudaGraph_t g;
    RF_CUDA(cudaGraphCreate(&g, 0));
    e->fgraph = g;
    Consts& c = e->cf;
    RF_CUDA(cudaGraphConditionalHandleCreate(&c.h_loop, g, 0, 0));
    RF_CUDA(cudaGraphConditionalHandleCreate(&c.h_rebuild, g, 0, 0));
    c.use_graph = 1;
    Dev d = e->d;
    Consts cc = c;
    void* args[] = {&d, &cc};
    auto kparams = [&](void* fn, unsigned grid, unsigned block) {
        cudaKernelNodeParams kp = {};
        kp.func = fn; kp.gridDim = dim3(grid); kp.blockDim = dim3(block);
        kp.sharedMemBytes = 0; kp.kernelParams = args; kp.extra = nullptr;
        return kp;
    };
    cudaGraphNode_t pro;
    cudaKernelNodeParams kp = kparams((void*)k_fire_prologue, 1, 32);
    RF_CUDA(cudaGraphAddKernelNode(&pro, g, nullptr, 0, &kp));
    cudaGraphNodeParams wp = {};
    wp.type = cudaGraphNodeTypeConditional;
    wp.conditional.handle = c.h_loop;
    wp.conditional.type = cudaGraphCondTypeWhile;
    wp.conditional.size = 1;
    cudaGraphNode_t wnode;
    RF_CUDA(cudaGraphAddNode(&wnode, g, &pro, 1, &wp));
    cudaGraph_t body = wp.conditional.phGraph_out[0];
    cudaGraphNodeParams ip = {};
    ip.type = cudaGraphNodeTypeConditional;
    ip.conditional.handle = c.h_rebuild;
    ip.conditional.type = cudaGraphCondTypeIf;
    ip.conditional.size = 1;
    cudaGraphNode_t inode;
    RF_CUDA(cudaGraphAddNode(&inode, body, nullptr, 0, &ip));
    cudaGraph_t rb = ip.conditional.phGraph_out[0];
    const unsigned gN = (c.N + 255) / 256;
    const unsigned gC = (c.cg_cells + 1 + 255) / 256;
    struct { void* fn; unsigned grid, block; } seq[] = {
        {(void*)k_rb_zero, gC, 256},      {(void*)k_rb_bin, gN, 256},
        {(void*)k_rb_scan_sums, e->cg_nb, 1024}, {(void*)k_rb_scan_totals, 1, 32},
        {(void*)k_rb_scan_apply, e->cg_nb, 1024}, {(void*)k_rb_scatter, gN, 256},
        {(void*)k_rb_cand, (c.N + RF_RB_CTA - 1) / RF_RB_CTA, RF_RB_CTA},
    };
    cudaGraphNode_t prev = nullptr;
    for (auto& q : seq) {
        cudaGraphNode_t n;
        kp = kparams(q.fn, q.grid, q.block);
        RF_CUDA(cudaGraphAddKernelNode(&n, rb, prev ? &prev : nullptr, prev ? 1 : 0, &kp));
        prev = n;
    }
    cudaGraphNode_t last = inode, node;
    for (int u = 0; u < RF_GRAPH_UNROLL; ++u) {
        cc.fire_skip = u > 0;                        // (node parameters are copied when the node is added)
        kp = kparams(fire_force_kernel(e), e->ncta, 128);
        kp.sharedMemBytes = step_smem(e);
        RF_CUDA(cudaGraphAddKernelNode(&node, body, &last, 1, &kp));
        last = node;
        kp = kparams((void*)k_fire_update, e->nblocks, 128);
        RF_CUDA(cudaGraphAddKernelNode(&node, body, &last, 1, &kp));
        last = node;
    }
    RF_CUDA(cudaGraphInstantiate(&e->fexec, g, 0));
    return RF_OK;
}

// The FIRE loop on a plain stream (no conditional graph nodes): chunks of iterations,
// each kernel returning early once the device has stopped the loop.
rf_status launch_stream_fire(rf_engine* e, uint64_t max_iter) {
    Dev d = e->d;
    Consts c = e->cf;
    c.use_graph = 0;
    const unsigned gN = (c.N + 255) / 256, gC = (c.cg_cells + 1 + 255) / 256;
    cudaStream_t s = e->stream;
    void* ff = fire_force_kernel(e);
    void* args[] = {&d, &c};
    for (uint64_t q = 0; q < max_iter + 1;) {
        for (int u = 0; u < 32; ++u, ++q) {
            k_rb_zero<<<gC, 256, 0, s>>>(d, c);
            k_rb_bin<<<gN, 256, 0, s>>>(d, c);
            k_rb_scan_sums<<<e->cg_nb, 1024, 0, s>>>(d, c);
            k_rb_scan_totals<<<1, 32, 0, s>>>(d, c);
            k_rb_scan_apply<<<e->cg_nb, 1024, 0, s>>>(d, c);
            k_rb_scatter<<<gN, 256, 0, s>>>(d, c);
            k_rb_cand<<<(c.N + RF_RB_CTA - 1) / RF_RB_CTA, RF_RB_CTA, 0, s>>>(d, c);
            RF_CUDA(cudaLaunchKernel(ff, dim3(e->ncta), dim3(128), args, step_smem(e), s));
            k_fire_update<<<e->nblocks, 128, 0, s>>>(d, c);
        }
        RF_CHECK_LAUNCH("engine stream FIRE");
        uint32_t stop = 0;
        RF_CUDA(cudaMemcpyAsync(&stop, &e->d.sc->fstop, sizeof(stop), cudaMemcpyDeviceToHost, s));
        RF_CUDA(cudaStreamSynchronize(s));
        if (stop) break;
    }
    return RF_OK;
}

rf_status launch_stream_steps(rf_engine* e, uint64_t nsteps) {
    Dev d = e->d;
    Consts c = e->c;
    c.use_graph = 0;
    const unsigned gN = (c.N + 255) / 256, gC = (c.cg_cells + 1 + 255) / 256;
    cudaStream_t s = e->stream;
    for (uint64_t q = 0; q < nsteps; ++q) {
        k_stream_gate<<<1, 32, 0, s>>>(d);
        k_rb_zero<<<gC, 256, 0, s>>>(d, c);
        k_rb_bin<<<gN, 256, 0, s>>>(d, c);
        k_rb_scan_sums<<<e->cg_nb, 1024, 0, s>>>(d, c);
        k_rb_scan_totals<<<1, 32, 0, s>>>(d, c);
        k_rb_scan_apply<<<e->cg_nb, 1024, 0, s>>>(d, c);
        k_rb_scatter<<<gN, 256, 0, s>>>(d, c);
        k_rb_cand<<<(c.N + RF_RB_CTA - 1) / RF_RB_CTA, RF_RB_CTA, 0, s>>>(d, c);
        void* sargs[] = {&d, &c};
        if (cudaLaunchKernel(step_kernel(e), dim3(e->ncta), dim3(128), sargs, step_smem(e), s) != cudaSuccess) break;
        k_stream_ungate<<<1, 32, 0, s>>>(d);
    }
    RF_CHECK_LAUNCH("engine stream steps");
    return RF_OK;
}

}  // namespace

// Host-side helpers from the md_* layer.
extern "C" size_t md_CellDistributionScratchBytes(uint_fast32_t N, uint_fast32_t CN);

namespace {

// Host description of a batch: per-specimen tasks (shifted, with the batch's grid), bond
// parameters and particle ranges.
struct BatchIn {
    std::vector<rf_task> tasks;
    std::vector<rf_ext_params> xs;
    std::vector<uint32_t> p0, n;
    std::vector<double> xoff;
};

// post-peak stop rule of an extended-model specimen: the stress fraction of the peak below
// which it counts as fractured (0: the reference's ZeroStress rule alone)
double keep_fraction(const rf_ext_params& x) { return x.post_peak_drop > 0.0 ? 1.0 - x.post_peak_drop : 0.0; }

void fill_scalars(DevScalars& h, const rf_task& t) {
    std::memset(&h, 0, sizeof(h));
    const rf_compression& K_ = t.Compress;
    h.V = K_.V; h.VLoad = K_.VLoad; h.Top = K_.Top; h.Bottom = K_.Bottom; h.TopR = K_.TopR; h.BottomR = K_.BottomR;
    h.FractureStress = K_.FractureStress; h.FractureStrain = K_.FractureStrain; h.MinStress = K_.MinStress;
    h.ZeroStress = K_.ZeroStress; h.Stress = K_.Stress; h.Strain = K_.Strain; h.MaxStrain = K_.MaxStrain;
    h.Size0 = K_.Size0;
    h.size_d[0] = K_.size_d.x; h.size_d[1] = K_.size_d.y; h.size_d[2] = K_.size_d.z;
    h.center_d[0] = K_.center_d.x; h.center_d[1] = K_.center_d.y; h.center_d[2] = K_.center_d.z;
    h.sz0 = t.sz0 != 0.0 ? t.sz0 : (double)K_.size.z;
    h.center[0] = K_.center.x; h.center[1] = K_.center.y; h.center[2] = K_.center.z;
    h.size[0] = K_.size.x; h.size[1] = K_.size.y; h.size[2] = K_.size.z;
    h.sized2[0] = K_.sized2.x; h.sized2[1] = K_.sized2.y; h.sized2[2] = K_.sized2.z;
    h.RR = K_.RR; h._1d_Area = K_._1d_Area; h.Hd2 = K_.Hd2;
    h.Loading = K_.Loading; h.Fracture = K_.Fracture;
    h.done = (K_.Strain < K_.MaxStrain && !K_.Fracture) ? 0u : 1u;
}

// Rows given in the reference layout (a restored checkpoint) instead of built from the
// positions: the engine sizes its bond records for them.
struct RowsIn {
    const uint_fast32_t* IL;
    const uint8_t* ILtype;
    const float* iL;
    const rf_float3 *Rij, *Oijt, *Mijn, *Mijt;
};

rf_status engine_create_impl(const rf_task* t, const float* h_R, const double* h_Rd, const double* h_rad,
                             const rf_ext_params* x, rf_engine** out, const BatchIn* bin = nullptr,
                             const RowsIn* rows = nullptr) {
    const bool ext = x != nullptr;
    if (!t || !out || t->N == 0 || t->K == 0 || (ext ? (!h_Rd || !h_rad) : !h_R)) {
        set_error("rf_engine_create: bad arguments");
        return RF_ERR_INVALID;
    }
    double rmax = 0.0, rmin = 1e300;
    if (ext) {
        for (uint64_t i = 0; i < t->N; ++i) { rmax = std::max(rmax, h_rad[i]); rmin = std::min(rmin, h_rad[i]); }
        if (x->ref_mode != 0 && x->ref_mode != 1) { set_error("rf_engine_create_ext: ref_mode must be 0 or 1"); return RF_ERR_INVALID; }
        if (x->ref_mode) {
            if (rmin != t->Po.p_r || rmax != t->Po.p_r) {
                set_error("rf_engine_create_ext: ref_mode needs every radius equal to Po.p_r (%g)", t->Po.p_r);
                return RF_ERR_INVALID;
            }
        } else if (!(x->kn > 0.0) || !(x->ks >= 0.0) || !(x->bond_lambda > 0.0) || !(x->weibull_m > 0.0) ||
                   !(x->sigma_c > 0.0) || !(x->tau_c > 0.0)) {
            set_error("rf_engine_create_ext: radii and bond parameters must be positive");
            return RF_ERR_INVALID;
        }
        if (!(rmin > 0.0) || !(x->post_peak_drop >= 0.0 && x->post_peak_drop < 1.0) ||
            !(x->list_gap >= 0.0 && x->list_gap < 1e300)) {
            set_error("rf_engine_create_ext: radii must be positive, post_peak_drop in [0, 1), list_gap >= 0");
            return RF_ERR_INVALID;
        }
        if (!(2.0 * rmax < std::sqrt(t->Po.aa_farcut))) {
            set_error("rf_engine_create_ext: a_farcut (%g) must exceed the largest contact distance 2*r_max (%g)",
                      std::sqrt(t->Po.aa_farcut), 2.0 * rmax);
            return RF_ERR_INVALID;
        }
    }
    if (t->K > 32) { set_error("rf_engine_create: the engine keeps slot masks in 32 bits (K <= 32), got K=%u", t->K); return RF_ERR_INVALID; }
    if (t->N >= 0xFFFFFFFFull) { set_error("rf_engine_create: N too large"); return RF_ERR_INVALID; }
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) { set_error("rf_engine_create: no CUDA device"); return RF_ERR_NO_DEVICE; }
    rf_engine* e = new rf_engine();
    std::memset(&e->d, 0, sizeof(e->d));
    std::memset(&e->c, 0, sizeof(e->c));
    e->task = *t;
    e->graph = nullptr; e->exec = nullptr; e->graph_ok = false; e->staging = nullptr; e->bonds_initial = 0;
    e->stream = nullptr; e->counters_dev = nullptr; e->maxq_dev = nullptr;
    e->fgraph = nullptr; e->fexec = nullptr; e->fire_ready = false;
    cudaGetDevice(&e->device);
    rf_status st = RF_OK;
    auto fail = [&](rf_status s) { rf_engine_destroy(e); return s; };
    if (cudaStreamCreateWithFlags(&e->stream, cudaStreamNonBlocking) != cudaSuccess) return fail(RF_ERR_CUDA);

    const uint32_t N = (uint32_t)t->N, K = t->K;
    Consts& c = e->c;
    c.N = N; c.K = K; c.KC = 64; c.kind = t->kind;
    const rf_potential& P = t->Po;
    c.dt_d = P.dt; c.p_r_d = P.p_r;
    c.bp = BondParams{(float)P.dt, (float)P.m_E, (float)P.m_G, (float)P.b_r, (float)P.m_Ec, (float)P.m_Gc};
    c.cp = ContactParams{(float)P.dt, (float)P.hm_E, (float)P.hm_G, (float)P.p_A, (float)P.p_mu, (float)P.p_mur,
                         (float)P.p_m, (float)P.p_r};
    c.dtm = (float)P.dt_d_m; c.dt = (float)P.dt; c.dtI = (float)P.dt_d_I;
    if (ext) {
        c.ext = 1;
        c.ep = ExtParams{(float)P.dt, (float)P.hm_E, (float)P.hm_G, (float)P.p_A, (float)P.p_mu, (float)P.p_mur};
        c.kn = (float)x->kn; c.ks = (float)x->ks; c.br_lambda = (float)x->bond_lambda;
        c.cmass = (float)(P.p_m / (P.p_r * P.p_r * P.p_r));     // mass = density * 4/3 pi r^3
        c.aa_farcut_d = P.aa_farcut; c.aacut_d = (double)t->aacut;
        c.a_farcut_d = P.a_farcut;
        c.lgap_d = x->list_gap;
        c.lgap_f = (float)x->list_gap;
        c.ref_mode = x->ref_mode;
        c.refE = (float)P.m_E; c.refG = (float)P.m_G; c.ref_br = (float)P.b_r;
    }
    c.aacut = t->aacut; c.aa_farcut = (float)P.aa_farcut;
    c.g.a = t->C.a; c.g.inv_a = t->C._1d_a; c.g.nx = t->C.Nr.x; c.g.ny = t->C.Nr.y; c.g.nz = t->C.Nr.z; c.g.CN = t->C.N;
    c.zcut = (t->kind == RF_TEST_BRAZIL) ? (float)((double)t->S.center.y + (double)t->S.spacesized2.y)
                                         : (float)((double)t->S.center.z + (double)t->S.spacesized2.z);
    c.box_c = t->S.center; c.box_h = t->S.spacesized2; c.hp = t->S.hidenpoint;
    // candidate grid over the cut box, one cell of margin each side; cell >= rc
    const double acut = std::sqrt((double)t->aacut);
    const double skin = 0.1 * acut;
    const double rc = acut + skin;
    c.rc2 = (float)(rc * rc);
    c.disp2 = (float)((0.3 * skin) * (0.3 * skin));   // checked every RF_GRAPH_UNROLL steps
    c.hard2 = (float)((0.5 * skin) * (0.5 * skin));
    c.acut_f = (float)acut;
    c.skin_f = (float)skin;
    const double hcell = rc * 1.0001;
    c.cg_inv_h = (float)(1.0 / hcell);
    c.cg_ox = (float)(t->S.center.x - t->S.spacesized2.x - hcell);
    c.cg_oy = (float)(t->S.center.y - t->S.spacesized2.y - hcell);
    c.cg_oz = (float)(t->S.center.z - t->S.spacesized2.z - hcell);
    c.cg_nx = (uint32_t)std::ceil((2.0 * t->S.spacesized2.x + 2 * hcell) / hcell) + 1;
    c.cg_ny = (uint32_t)std::ceil((2.0 * t->S.spacesized2.y + 2 * hcell) / hcell) + 1;
    c.cg_nz = (uint32_t)std::ceil((2.0 * t->S.spacesized2.z + 2 * hcell) / hcell) + 1;
    const uint64_t cells = (uint64_t)c.cg_nx * c.cg_ny * c.cg_nz;
    if (cells >= 0x7FFFFFFFull) { set_error("rf_engine_create: candidate grid too large"); return fail(RF_ERR_INVALID); }
    c.cg_cells = (uint32_t)cells;
    e->cg_nb = (uint32_t)((cells + 1 + 4095) / 4096);
    const uint32_t nspec = bin ? (uint32_t)bin->tasks.size() : 1u;
    c.curve_cap = nspec == 1 ? (1u << 20) : std::max(4096u, (1u << 20) / nspec);   // records per specimen
    e->nblocks = (N + 127) / 128;
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, e->device);
    e->pw = particles_per_warp(N, sms);
    e->ncta = (N + 4 * e->pw - 1) / (4 * e->pw);
    const size_t nzw = (e->ncta + 31) / 32;

    Dev& d = e->d;
    d.n_particles = N;
    const size_t NK = (size_t)N * K;
    SpecGeom* dgeom = nullptr;
    uint16_t* dblk = nullptr;
    {
        Arrays A;
        for (int b = 0; b < 2; ++b) {
            if (ext) A.add(&d.posd[b], N); else A.add(&d.pos[b], N);
            A.add(&d.vw[b], N);
            A.add(&d.cO[b], 3 * NK);
        }
        A.add(&d.ids, NK); A.add(&d.il, NK);
        A.add(&d.live, N); A.add(&d.bond, N); A.add(&d.cmask, N); A.add(&d.nbq, N); A.add(&d.bmask, N); A.add(&e->maxq_dev, 1);
        A.add(&d.cand, (size_t)c.KC * N); A.add(&d.cand_n, N); A.add(&d.member, N);
        A.add(&d.pos_ref, N); A.add(&d.cmargin, N); A.add(&d.cbound, N); A.add(&d.cg_key, N);
        A.add(&d.cg_count, cells + 1); A.add(&d.cg_start, cells + 1); A.add(&d.cg_fill, cells + 1);
        A.add(&d.cg_bsum, e->cg_nb); A.add(&d.cg_sorted, N); A.add(&d.cg_slot, N); A.add(&d.cg_pos, N);
        A.add(&d.partial, e->ncta); A.add(&d.partial2, e->ncta); A.add(&d.nz, nzw); A.add(&d.nz2, nzw);
        A.add(&d.curve, 3 * (size_t)c.curve_cap * nspec); A.add(&d.sc, 1); A.add(&e->counters_dev, 4);
        A.add(&dgeom, nspec);
        if (nspec > 1) { A.add(&dblk, e->nblocks); A.add(&d.spec, nspec); }
        if ((st = dalloc(e, A))) return fail(st);
    }
    cudaStream_t s = e->stream;
    for (int b = 0; b < 2; ++b) {
        if (cudaMemsetAsync(d.vw[b], 0, N * sizeof(F8), s))
            return fail(cuda_status(cudaGetLastError(), "memset"));
    }
    // specimens: geometry, CTA -> specimen map, per-specimen scalars
    d.nspec = nspec;
    {
        std::vector<SpecGeom> hg(nspec);
        for (uint32_t q = 0; q < nspec; ++q) {
            const rf_task& ts = bin ? bin->tasks[q] : *t;
            SpecGeom& G = hg[q];
            G.zcut = (t->kind == RF_TEST_BRAZIL) ? (float)((double)ts.S.center.y + (double)ts.S.spacesized2.y)
                                                 : (float)((double)ts.S.center.z + (double)ts.S.spacesized2.z);
            G.box_c = ts.S.center; G.box_h = ts.S.spacesized2; G.hp = ts.S.hidenpoint;
            G.p0 = bin ? bin->p0[q] : 0u;
            G.p1 = bin ? bin->p0[q] + bin->n[q] : N;
        }
        if (cudaMemcpyAsync(dgeom, hg.data(), nspec * sizeof(SpecGeom), cudaMemcpyHostToDevice, s)) return fail(RF_ERR_CUDA);
        d.geom = dgeom;
        d.blk_spec = nullptr;
        if (nspec > 1) {
            std::vector<uint16_t> hb(e->nblocks);
            uint32_t q = 0;
            for (uint32_t b = 0; b < e->nblocks; ++b) {
                while (q + 1 < nspec && hg[q].p1 <= b * 128u) ++q;
                hb[b] = (uint16_t)q;
            }
            if (cudaMemcpyAsync(dblk, hb.data(), e->nblocks * sizeof(uint16_t), cudaMemcpyHostToDevice, s))
                return fail(RF_ERR_CUDA);
            d.blk_spec = dblk;
            std::vector<DevScalars> hs(nspec);
            for (uint32_t k = 0; k < nspec; ++k) {
                fill_scalars(hs[k], bin->tasks[k]);
                hs[k].keep_frac = keep_fraction(bin->xs[k]);
            }
            if (cudaMemcpyAsync(d.spec, hs.data(), nspec * sizeof(DevScalars), cudaMemcpyHostToDevice, s))
                return fail(RF_ERR_CUDA);
            e->spec_tasks = bin->tasks;
            e->spec_p0 = bin->p0;
            e->spec_n = bin->n;
            e->spec_xoff = bin->xoff;
        } else {
            d.spec = d.sc;
        }
    }
    // the scalar block is read (step parity) by the row import below: start it at zero
    if (cudaMemsetAsync(d.member, 0, N * sizeof(unsigned long long), s) || cudaMemsetAsync(d.cand_n, 0, N * 4, s) ||
        cudaMemsetAsync(d.cmargin, 0, N * sizeof(float), s) ||
        cudaMemsetAsync(d.nz, 0, nzw * 4, s) || cudaMemsetAsync(d.nz2, 0, nzw * 4, s) ||
        cudaMemsetAsync(d.sc, 0, sizeof(DevScalars), s))
        return fail(RF_ERR_CUDA);

    // Initial rows exactly as the drivers build them (md_calculationbraziltest.cu:132-144): the
    // binning of md_CellDistribution, then lists, bonds and DeleteFarLinks straight into the
    // engine's rows and records; or rows given in the reference layout.
    {
        float* dR = nullptr;
        uint_fast32_t *dCI = nullptr, *dCIs = nullptr, *dpnC = nullptr, *dIL = nullptr;
        uint8_t* dT = nullptr;
        float* dIL_f = nullptr;
        rf_float3* dS = nullptr;
        double *dRd = nullptr, *dRad = nullptr;
        BondSpec* dbs = nullptr;
        char* scratch = nullptr;
        const size_t sb = md_CellDistributionScratchBytes(N, t->C.N);
        Arrays A;
        A.add(&dR, 3 * (size_t)N); A.add(&dCI, N); A.add(&dCIs, 2 * (size_t)N); A.add(&dpnC, 2 * t->C.N);
        A.add(&scratch, sb); A.add(&dbs, nspec);
        if (ext) { A.add(&dRd, 3 * (size_t)N); A.add(&dRad, N); }
        if (rows) { A.add(&dIL, NK); A.add(&dT, NK); A.add(&dIL_f, NK); A.add(&dS, 4 * NK); }
        void* tmp = nullptr;
        cudaError_t ce = A.alloc(&tmp);
        if (!ce && ext) {
            ce = cudaMemcpyAsync(dRd, h_Rd, 3 * (size_t)N * sizeof(double), cudaMemcpyHostToDevice, s);
            if (!ce) ce = cudaMemcpyAsync(dRad, h_rad, (size_t)N * sizeof(double), cudaMemcpyHostToDevice, s);
            if (!ce) { k_posd_from_planar<<<(N + 255) / 256, 256, 0, s>>>(dRd, dRad, N, d.posd[0], dR); ce = cudaGetLastError(); }
        } else if (!ce) {
            ce = cudaMemcpyAsync(dR, h_R, 3 * (size_t)N * sizeof(float), cudaMemcpyHostToDevice, s);
            if (!ce) { k_planar_to_f4<<<(N + 255) / 256, 256, 0, s>>>(dR, N, d.pos[0], 1u); ce = cudaGetLastError(); }
        }
        rf_status st2 = ce ? cuda_status(ce, "engine init buffers") : RF_OK;
        rf_status init_dev = RF_OK;
        if (!st2) {
            rf_status a = md_CellDistribution(dR, N, dCI, dCIs, dpnC, t->C.N, t->C._1d_a, t->C.Nr, scratch, sb, s);
            if (a != RF_OK && a != RF_ERR_CELL_RANGE && a != RF_ERR_ROW_OVERFLOW) st2 = a; else if (a) init_dev = a;
        }
        const bool pair_cut = ext && x->list_gap > 0.0;
        uint32_t qb = 0;
        std::vector<BondSpec> hbs(nspec);
        if (!st2 && rows) {
            ce = cudaMemcpyAsync(dIL, rows->IL, NK * sizeof(uint_fast32_t), cudaMemcpyHostToDevice, s);
            if (!ce) ce = cudaMemcpyAsync(dT, rows->ILtype, NK, cudaMemcpyHostToDevice, s);
            if (!ce) ce = cudaMemcpyAsync(dIL_f, rows->iL, NK * sizeof(float), cudaMemcpyHostToDevice, s);
            const rf_float3* src[4] = {rows->Rij, rows->Oijt, rows->Mijn, rows->Mijt};
            for (int q = 0; q < 4 && !ce; ++q)
                ce = cudaMemcpyAsync(dS + q * NK, src[q], NK * sizeof(rf_float3), cudaMemcpyHostToDevice, s);
            if (!ce) ce = cudaMemsetAsync(e->maxq_dev, 0, sizeof(uint32_t), s);
            if (!ce) { k_count_records<<<148 * 4, 256, 0, s>>>(dIL, dT, dS, N, K, e->maxq_dev); ce = cudaGetLastError(); }
            if (!ce) ce = cudaMemcpyAsync(&qb, e->maxq_dev, sizeof(qb), cudaMemcpyDeviceToHost, s);
            if (!ce) ce = cudaStreamSynchronize(s);
            if (ce) st2 = cuda_status(ce, "engine rows");
        }
        // (with a list gap every listed pair is within its cutoff: nothing to delete)
        const float aa_create = (float)P.b_dd, aa_far = pair_cut ? 0.f : (float)P.aa_farcut;
        if (!st2 && !rows) {
            uint32_t w[2] = {0, 0};                  // status of the lists, most bonds of a row
            for (uint32_t q = 0; q < nspec; ++q) {
                if (!ext) { hbs[q] = BondSpec{}; continue; }
                const rf_ext_params& xq = bin ? bin->xs[q] : *x;
                const rf_task& tq = bin ? bin->tasks[q] : *t;
                hbs[q] = BondSpec{xq.gap_frac, xq.weibull_m, xq.sigma_c, xq.tau_c, xq.seed, bin ? bin->p0[q] : 0u,
                                  bin ? bin->p0[q] + bin->n[q] : N, xq.ref_mode, tq.Po.b_d};
                if (xq.ref_mode) { hbs[q].sig = tq.Po.m_Ec; hbs[q].tau = tq.Po.m_Gc; hbs[q].wm = 1.0; }
            }
            uint32_t* dw = (uint32_t*)e->counters_dev;
            ce = cudaMemcpyAsync(dbs, hbs.data(), nspec * sizeof(BondSpec), cudaMemcpyHostToDevice, s);
            if (!ce) ce = cudaMemsetAsync(dw, 0, 2 * sizeof(uint32_t), s);
            if (!ce) {
                k_rows_list<<<(N + 15) / 16, 128, 0, s>>>(dR, d, c, dCIs, dpnC, P.a_farcut, pair_cut ? x->list_gap : -1.0, dw);
                k_rows_bonds<0><<<(N + 31) / 32, 128, 0, s>>>(dR, d, c, aa_create, aa_far, dbs, nspec, dw + 1);
                ce = cudaGetLastError();
            }
            if (!ce) ce = cudaMemcpyAsync(w, dw, sizeof(w), cudaMemcpyDeviceToHost, s);
            if (!ce) ce = cudaStreamSynchronize(s);
            if (ce) st2 = cuda_status(ce, "engine lists");
            else if (w[0] && !init_dev) init_dev = (rf_status)w[0];
            qb = w[1];
        }
        if (!st2) {
            // bond records: as many per particle as its row holds bonds (bonds are never created later)
            d.QB = qb ? qb : 1u;
            Arrays B;
            B.add(&d.bjk, (size_t)d.QB * N); B.add(&d.rec, (size_t)d.QB * N);
            st2 = dalloc(e, B);
        }
        if (!st2) {
            if (rows)
                k_rows_import<<<(N + 127) / 128, 128, 0, s>>>(dIL, dT, dIL_f, dS, dS + NK, dS + 2 * NK, dS + 3 * NK, d, c);
            else
                k_rows_bonds<1><<<(N + 31) / 32, 128, 0, s>>>(dR, d, c, aa_create, aa_far, dbs, nspec, nullptr);
            ce = cudaGetLastError();
            if (!ce) ce = cudaStreamSynchronize(s);
            if (ce) st2 = cuda_status(ce, "engine init");
        }
        cudaFree(tmp);
        if (st2) return fail(st2);
        st = init_dev;
    }

    // scalar state (with one specimen the global block is also the specimen's)
    DevScalars h;
    fill_scalars(h, *t);
    if (ext) h.keep_frac = keep_fraction(*x);
    if (nspec > 1) {
        h.done = 0;
        for (uint32_t q = 0; q < nspec; ++q) {
            const rf_compression& Kq = bin->tasks[q].Compress;
            if (Kq.Strain < Kq.MaxStrain && !Kq.Fracture) break;
            if (q + 1 == nspec) h.done = 1;
        }
    }
    h.rebuild = 1;
    h.err = (uint32_t)st;
    if (cudaMemcpyAsync(d.sc, &h, sizeof(h), cudaMemcpyHostToDevice, s) || cudaStreamSynchronize(s))
        return fail(RF_ERR_CUDA);

    {
        uint64_t cnt[5];
        if (rf_engine_counters(e, cnt, 5) == RF_OK) e->bonds_initial = cnt[2];
    }
    // graph with device-driven loop; fall back to plain stream launches if unavailable
    if (!getenv("RF_ENGINE_NO_GRAPH")) {
        rf_status gs = build_graph(e);
        if (gs == RF_OK) e->graph_ok = true;
        else { cudaGetLastError(); e->c.use_graph = 0; }
    }
    *out = e;
    return RF_OK;
}

}  // namespace

extern "C" {

rf_status rf_engine_create(const rf_task* t, const float* h_R, rf_engine** out) {
    return engine_create_impl(t, h_R, nullptr, nullptr, nullptr, out);
}

rf_status rf_engine_create_ext(const rf_task* t, const rf_ext_params* x, const double* h_R, const double* h_radius,
                               rf_engine** out) {
    if (!x) { set_error("rf_engine_create_ext: null parameters"); return RF_ERR_INVALID; }
    return engine_create_impl(t, nullptr, h_R, h_radius, x, out);
}

rf_status rf_engine_create_batch(const rf_task* tasks, const rf_ext_params* xs, const double* const* h_R,
                                 const double* const* h_radius, int nspec, rf_engine** out) {
    if (!tasks || !xs || !h_R || !h_radius || !out || nspec < 1 || nspec > 65535) {
        set_error("rf_engine_create_batch: bad arguments");
        return RF_ERR_INVALID;
    }
    const rf_task& t0 = tasks[0];
    uint64_t total = 0;
    for (int q = 0; q < nspec; ++q) {
        const rf_task& tq = tasks[q];
        if (!h_R[q] || !h_radius[q] || tq.N < 128 || tq.kind != t0.kind || tq.K != t0.K || tq.C.a != t0.C.a ||
            tq.aacut != t0.aacut || tq.Po.dt != t0.Po.dt || tq.Po.p_r != t0.Po.p_r ||
            tq.Po.aa_farcut != t0.Po.aa_farcut || tq.Po.hm_E != t0.Po.hm_E || tq.Po.hm_G != t0.Po.hm_G ||
            tq.Po.p_A != t0.Po.p_A || tq.Po.p_mu != t0.Po.p_mu || tq.Po.p_mur != t0.Po.p_mur ||
            tq.Po.p_m != t0.Po.p_m || xs[q].kn != xs[0].kn || xs[q].ks != xs[0].ks ||
            xs[q].bond_lambda != xs[0].bond_lambda || xs[q].list_gap != xs[0].list_gap ||
            xs[q].ref_mode != xs[0].ref_mode ||
            (xs[0].ref_mode && (tq.Po.m_E != t0.Po.m_E || tq.Po.m_G != t0.Po.m_G || tq.Po.b_r != t0.Po.b_r)) ||
            !(xs[q].post_peak_drop >= 0.0 && xs[q].post_peak_drop < 1.0)) {
            set_error("rf_engine_create_batch: specimen %d must have >= 128 particles and the batch's test kind, "
                      "slots, grid cell, material, time step, bond stiffness and list gap, and a post-peak drop in [0, 1)", q);
            return RF_ERR_INVALID;
        }
        total += tq.N;
    }
    if (total >= 0xFFFFFFFFull) { set_error("rf_engine_create_batch: too many particles"); return RF_ERR_INVALID; }
    // lay the specimens out along x, each shifted by a whole number of cells so that its
    // cell-relative geometry (and so its insertion order) is what it would be alone,
    // with two cells between neighbouring boxes (no cross-specimen links)
    const double a = (double)t0.C.a;
    BatchIn bin;
    bin.tasks.resize(nspec); bin.xs.assign(xs, xs + nspec); bin.p0.resize(nspec); bin.n.resize(nspec);
    bin.xoff.resize(nspec);
    double cursor = 0.0, Bx = 0.0, By = 0.0, Bz = 0.0, lo_y = 1e300, lo_z = 1e300, hi_y = -1e300, hi_z = -1e300;
    uint32_t p = 0;
    for (int q = 0; q < nspec; ++q) {
        const rf_sample& S = tasks[q].S;
        const double lo = (double)S.center.x - (double)S.spacesized2.x, hi = (double)S.center.x + (double)S.spacesized2.x;
        const double off = q == 0 ? 0.0 : std::ceil((cursor - lo) / a) * a;
        bin.xoff[q] = off;
        cursor = hi + off + 2.0 * a;
        rf_task tq = tasks[q];
        tq.S.center.x = (float)((double)S.center.x + off);
        tq.S.A.x = (float)((double)S.A.x + off); tq.S.B.x = (float)((double)S.B.x + off);
        tq.S.hidenpoint.x = (float)((double)S.hidenpoint.x + off);
        tq.S.center_real.x += off; tq.S.A_real.x += off; tq.S.B_real.x += off;
        tq.Compress.center_d.x += off;
        tq.Compress.center.x = (float)tq.Compress.center_d.x;
        bin.tasks[q] = tq;
        bin.p0[q] = p; bin.n[q] = (uint32_t)tq.N;
        p += (uint32_t)tq.N;
        Bx = std::max(Bx, (double)tq.S.B.x); By = std::max(By, (double)S.B.y); Bz = std::max(Bz, (double)S.B.z);
        lo_y = std::min(lo_y, (double)S.center.y - (double)S.spacesized2.y);
        hi_y = std::max(hi_y, (double)S.center.y + (double)S.spacesized2.y);
        lo_z = std::min(lo_z, (double)S.center.z - (double)S.spacesized2.z);
        hi_z = std::max(hi_z, (double)S.center.z + (double)S.spacesized2.z);
    }
    // the batch's cell grid covers every box (cell_data::CalculateParameters on the union corner)
    rf_cells C = t0.C;
    C.Nr.x = (unsigned)(std::floor((float)(Bx * (double)C._1d_a)) + 1.0f);
    C.Nr.y = (unsigned)(std::floor((float)(By * (double)C._1d_a)) + 1.0f);
    C.Nr.z = (unsigned)(std::floor((float)(Bz * (double)C._1d_a)) + 3.0f);
    C.N = (uint64_t)C.Nr.x * C.Nr.y * C.Nr.z;
    for (int q = 0; q < nspec; ++q) bin.tasks[q].C = C;
    rf_task tc = bin.tasks[0];
    tc.N = total;
    tc.C = C;
    const double lo_x = (double)bin.tasks[0].S.center.x - (double)bin.tasks[0].S.spacesized2.x;
    const double hi_x = (double)bin.tasks[nspec - 1].S.center.x + (double)bin.tasks[nspec - 1].S.spacesized2.x;
    tc.S.center = rf_float3{(float)(0.5 * (lo_x + hi_x)), (float)(0.5 * (lo_y + hi_y)), (float)(0.5 * (lo_z + hi_z))};
    tc.S.spacesized2 = rf_float3{(float)(0.5 * (hi_x - lo_x)), (float)(0.5 * (hi_y - lo_y)), (float)(0.5 * (hi_z - lo_z))};
    tc.bloks = total / 1024 + 1;
    std::vector<double> R(3 * total), rad(total);
    for (int q = 0; q < nspec; ++q) {
        const uint64_t n = tasks[q].N, p0 = bin.p0[q];
        for (uint64_t i = 0; i < n; ++i) {
            R[p0 + i] = h_R[q][i] + bin.xoff[q];
            R[total + p0 + i] = h_R[q][n + i];
            R[2 * total + p0 + i] = h_R[q][2 * n + i];
            rad[p0 + i] = h_radius[q][i];
        }
    }
    return engine_create_impl(&tc, nullptr, R.data(), rad.data(), &xs[0], out, &bin);
}

rf_status rf_engine_positions_f64(rf_engine* e, double* R) {
    if (!e || !R) { set_error("rf_engine_positions_f64: bad arguments"); return RF_ERR_INVALID; }
    if (!e->c.ext) { set_error("rf_engine_positions_f64: engine keeps float positions"); return RF_ERR_STATE; }
    const uint32_t N = e->c.N;
    cudaStream_t s = e->stream;
    DevScalars h;
    RF_CUDA(cudaStreamSynchronize(s));
    RF_CUDA(cudaMemcpy(&h, e->d.sc, sizeof(h), cudaMemcpyDeviceToHost));
    double* tmp = nullptr;
    RF_CUDA(cudaMalloc(&tmp, 3 * (size_t)N * sizeof(double)));
    k_posd_to_planar<<<(N + 255) / 256, 256, 0, s>>>(e->d.posd[h.steps & 1ull], N, tmp);
    cudaError_t ce = cudaGetLastError();
    if (!ce) ce = cudaMemcpyAsync(R, tmp, 3 * (size_t)N * sizeof(double), cudaMemcpyDeviceToHost, s);
    if (!ce) ce = cudaStreamSynchronize(s);
    cudaFree(tmp);
    if (ce) return cuda_status(ce, "rf_engine_positions_f64");
    return RF_OK;
}

rf_status rf_relax_default_params(rf_relax_params* p, const rf_task* t) {
    if (!p || !t) { set_error("rf_relax_default_params: bad arguments"); return RF_ERR_INVALID; }
    std::memset(p, 0, sizeof(*p));
    p->strain_inc = 2.5e-5;
    p->tol = 1e-6;
    p->dt0 = 0.1;
    p->dt_max = 1.0;
    p->dt_min = 1e-3;
    p->alpha0 = 0.1;
    p->f_inc = 1.1;
    p->f_dec = 0.5;
    p->f_alpha = 0.99;
    p->n_delay = 5;
    p->max_iter = 200000;
    return RF_OK;
}

}  // extern "C"

namespace {
rf_status fire_setup(rf_engine* e) {
    if (e->fire_ready) return RF_OK;
    Dev& d = e->d;
    const uint32_t N = e->c.N;
    const size_t groups = (size_t)d.nspec + e->ncta / FIRE_GROUP + 1;
    rf_status st;
    Arrays A;
    A.add(&d.frc, N); A.add(&d.mom, N); A.add(&d.rot, N); A.add(&d.x0, N); A.add(&d.xax, N);
    A.add(&d.fpart, (size_t)e->ncta * FIRE_SUMS);
    if (d.nspec > 1) A.add(&d.fpart2, (size_t)e->ncta * FIRE_SUMS);
    A.add(&d.fgrp, groups * FIRE_SUMS); A.add(&d.fgrp_n, groups);
    A.add(&d.rec0, (size_t)d.QB * N);
    if ((st = dalloc(e, A))) return st;
    RF_CUDA(cudaMemsetAsync(d.fgrp_n, 0, groups * sizeof(uint32_t), e->stream));
    e->cf = e->c;
    if (!getenv("RF_ENGINE_NO_GRAPH")) {
        if (build_fire_graph(e) != RF_OK) { cudaGetLastError(); e->cf.use_graph = 0; }
    } else {
        e->cf.use_graph = 0;
    }
    k_fire_buffers_init<<<(N + 255) / 256, 256, 0, e->stream>>>(d, e->cf);
    RF_CHECK_LAUNCH("k_fire_buffers_init");
    e->fire_ready = true;
    return RF_OK;
}

// One quasi-static load increment of every specimen of the engine (a batch relaxes its
// specimens together, each on its own FIRE scalars, and a specimen whose relaxation
// stopped stays put until the others stop). r: one result per specimen.
rf_status load_increment(rf_engine* e, const rf_relax_params* p, const float* warm, int ldw, int scaled,
                         rf_relax_result* r) {
    if (!e || !p) { set_error("rf_engine_load_increment: bad arguments"); return RF_ERR_INVALID; }
    if (!e->c.ext) { set_error("rf_engine_load_increment: quasi-static relaxation needs the extended model"); return RF_ERR_STATE; }
    if (e->c.ref_mode) { set_error("rf_engine_load_increment: the reference-constants mode runs explicit steps only"); return RF_ERR_STATE; }
    if (!(p->dt0 > 0) || !(p->dt_max >= p->dt0) || !(p->dt_min > 0) || !(p->dt_min <= p->dt0) || !(p->tol > 0) ||
        p->max_iter == 0 || !(p->alpha0 >= 0 && p->alpha0 < 1) || !(p->f_inc >= 1) || !(p->f_dec > 0 && p->f_dec < 1) ||
        !(p->strain_inc > 0)) {
        set_error("rf_engine_load_increment: bad FIRE parameters");
        return RF_ERR_INVALID;
    }
    cudaStream_t s = e->stream;
    Dev& d = e->d;
    const uint32_t N = e->c.N, ns = d.nspec;
    if (rf_status st = fire_setup(e)) return st;
    // FIRE constants into every specimen's scalar block (host read-modify-write, stream ordered)
    std::vector<DevScalars> hs(ns);
    RF_CUDA(cudaMemcpyAsync(hs.data(), d.spec, ns * sizeof(DevScalars), cudaMemcpyDeviceToHost, s));
    RF_CUDA(cudaStreamSynchronize(s));
    for (DevScalars& h : hs) {
        h.fdt0 = p->dt0; h.fdtmax = p->dt_max; h.fdtmin = p->dt_min; h.falpha0 = p->alpha0; h.finc = p->f_inc;
        h.fdec = p->f_dec; h.fshrink = p->f_alpha; h.fndelay = p->n_delay; h.ftol = p->tol; h.fmax_iter = p->max_iter;
    }
    RF_CUDA(cudaMemcpyAsync(d.spec, hs.data(), ns * sizeof(DevScalars), cudaMemcpyHostToDevice, s));
    // the bond records' state at the start of the increment (FIRE mode computes from it)
    RF_CUDA(cudaMemcpyAsync(d.rec0, d.rec, (size_t)d.QB * N * sizeof(Rec), cudaMemcpyDeviceToDevice, s));
    const unsigned nb = (N + 127) / 128;
    if (e->task.kind == RF_TEST_BRAZIL) {
        k_qs_begin_scalars<RF_TEST_BRAZIL><<<1, 32, 0, s>>>(d, e->cf, p->strain_inc);
        k_qs_begin<RF_TEST_BRAZIL><<<nb, 128, 0, s>>>(d, e->cf, warm, ldw, scaled, p->strain_inc);
    } else {
        k_qs_begin_scalars<RF_TEST_UNIAXIAL><<<1, 32, 0, s>>>(d, e->cf, p->strain_inc);
        k_qs_begin<RF_TEST_UNIAXIAL><<<nb, 128, 0, s>>>(d, e->cf, warm, ldw, scaled, p->strain_inc);
    }
    RF_CHECK_LAUNCH("k_qs_begin");
    if (e->cf.use_graph) RF_CUDA(cudaGraphLaunch(e->fexec, s));
    else if (rf_status st = launch_stream_fire(e, p->max_iter)) return st;
    if (e->task.kind == RF_TEST_BRAZIL) k_fire_bond_state<RF_TEST_BRAZIL><<<nb, 128, 0, s>>>(d, e->cf);
    else k_fire_bond_state<RF_TEST_UNIAXIAL><<<nb, 128, 0, s>>>(d, e->cf);
    RF_CHECK_LAUNCH("k_fire_bond_state");
    DevScalars g;
    RF_CUDA(cudaMemcpyAsync(hs.data(), d.spec, ns * sizeof(DevScalars), cudaMemcpyDeviceToHost, s));
    RF_CUDA(cudaMemcpyAsync(&g, d.sc, sizeof(g), cudaMemcpyDeviceToHost, s));
    RF_CUDA(cudaStreamSynchronize(s));
    if (r) {
        for (uint32_t k = 0; k < ns; ++k) {
            const DevScalars& h = hs[k];
            r[k].iterations = h.fiter;
            r[k].converged = (int32_t)h.fconverged;
            r[k].residual = h.fresidual;
            r[k].mean_force = h.fmean;
            r[k].stress = h.Stress;
            r[k].strain = h.Strain;
            r[k].broken_bonds = g.broken;         // (the engine's total)
            r[k].error = (rf_status)g.err;
        }
    }
    return RF_OK;
}

}  // namespace

extern "C" {

rf_status rf_engine_load_increment(rf_engine* e, const rf_relax_params* p, const float* warm, rf_relax_result* r) {
    if (e && e->d.nspec > 1) { set_error("rf_engine_load_increment: a batch takes rf_engine_load_increment_batch"); return RF_ERR_STATE; }
    return load_increment(e, p, warm, 6, 0, r);
}

rf_status rf_engine_load_increment_batch(rf_engine* e, const rf_relax_params* p, const float* warm, int ldw,
                                         int scaled, rf_relax_result* results) {
    if (warm && ldw < 6) { set_error("rf_engine_load_increment_batch: bad warm-start buffer"); return RF_ERR_INVALID; }
    return load_increment(e, p, warm, ldw, scaled ? 1 : 0, results);
}

rf_status rf_engine_load_increment_pred(rf_engine* e, const rf_relax_params* p, const float* pred, int ldp,
                                        rf_relax_result* r) {
    if (!pred || ldp < 6) { set_error("rf_engine_load_increment_pred: bad prediction buffer"); return RF_ERR_INVALID; }
    if (e && e->d.nspec > 1) { set_error("rf_engine_load_increment_pred: a batch takes rf_engine_load_increment_batch"); return RF_ERR_STATE; }
    return load_increment(e, p, pred, ldp, 1, r);
}

rf_status rf_engine_warm_features(rf_engine* e, double strain_inc, void* feat) {
    if (!e || !feat || !(strain_inc > 0)) { set_error("rf_engine_warm_features: bad arguments"); return RF_ERR_INVALID; }
    if (!e->c.ext) { set_error("rf_engine_warm_features: needs an extended-model engine"); return RF_ERR_STATE; }
    if (rf_status st = fire_setup(e)) return st;
    const uint32_t N = e->c.N, rows = (N + 127) / 128 * 128;
    cudaStream_t s = e->stream;
    if (rows > N) RF_CUDA(cudaMemsetAsync((__nv_bfloat16*)feat + (size_t)N * 64, 0, (size_t)(rows - N) * 64 * 2, s));
    if (e->task.kind == RF_TEST_BRAZIL)
        k_warm_features<RF_TEST_BRAZIL><<<(N + 127) / 128, 128, 0, s>>>(e->d, e->cf, strain_inc, (__nv_bfloat16*)feat);
    else
        k_warm_features<RF_TEST_UNIAXIAL><<<(N + 127) / 128, 128, 0, s>>>(e->d, e->cf, strain_inc, (__nv_bfloat16*)feat);
    RF_CHECK_LAUNCH("k_warm_features");
    return RF_OK;
}

rf_status rf_engine_warm_targets(rf_engine* e, double strain_inc, float* targets) {
    if (!e || !targets || !(strain_inc > 0)) { set_error("rf_engine_warm_targets: bad arguments"); return RF_ERR_INVALID; }
    if (!e->fire_ready) { set_error("rf_engine_warm_targets: no load increment run yet"); return RF_ERR_STATE; }
    cudaStream_t s = e->stream;
    k_warm_targets<<<(e->c.N + 127) / 128, 128, 0, s>>>(e->d, e->cf, strain_inc, targets);
    RF_CHECK_LAUNCH("k_warm_targets");
    return RF_OK;
}

rf_status rf_engine_increment_fields(rf_engine* e, double* x0, double* dx, double* rot) {
    if (!e || !e->fire_ready) { set_error("rf_engine_increment_fields: no load increment run yet"); return RF_ERR_STATE; }
    const uint32_t N = e->c.N;
    cudaStream_t s = e->stream;
    DevScalars h;
    RF_CUDA(cudaMemcpyAsync(&h, e->d.sc, sizeof(h), cudaMemcpyDeviceToHost, s));
    RF_CUDA(cudaStreamSynchronize(s));
    std::vector<double4> a(N), b(N), c(N);
    RF_CUDA(cudaMemcpy(a.data(), e->d.x0, N * sizeof(double4), cudaMemcpyDeviceToHost));
    RF_CUDA(cudaMemcpy(b.data(), e->d.posd[h.steps & 1ull], N * sizeof(double4), cudaMemcpyDeviceToHost));
    RF_CUDA(cudaMemcpy(c.data(), e->d.rot, N * sizeof(double4), cudaMemcpyDeviceToHost));
    for (uint32_t i = 0; i < N; ++i) {
        if (x0) { x0[3 * i] = a[i].x; x0[3 * i + 1] = a[i].y; x0[3 * i + 2] = a[i].z; }
        if (dx) { dx[3 * i] = b[i].x - a[i].x; dx[3 * i + 1] = b[i].y - a[i].y; dx[3 * i + 2] = b[i].z - a[i].z; }
        if (rot) { rot[3 * i] = c[i].x; rot[3 * i + 1] = c[i].y; rot[3 * i + 2] = c[i].z; }
    }
    return RF_OK;
}

rf_status rf_engine_autotune(rf_engine* e, int steps, int* choice, float* ms_out) {
    if (!e || steps <= 0) { set_error("rf_engine_autotune: bad arguments"); return RF_ERR_INVALID; }
    if (!e->c.ext) {
        if (choice) *choice = RF_STEP_MIN_BLOCKS;
        return RF_OK;                                      // the reference-model step has one variant
    }
    cudaStream_t s = e->stream;
    RF_CUDA(cudaStreamSynchronize(s));
    // snapshot the whole device state: the trials advance it and are undone afterwards
    std::vector<void*> backup(e->allocs.size(), nullptr);
    auto release = [&]() { for (void* p : backup) if (p) cudaFree(p); };
    for (size_t q = 0; q < e->allocs.size(); ++q) {
        if (cudaMalloc(&backup[q], e->alloc_bytes[q]) != cudaSuccess) { release(); return cuda_status(cudaGetLastError(), "rf_engine_autotune"); }
        if (cudaMemcpyAsync(backup[q], e->allocs[q], e->alloc_bytes[q], cudaMemcpyDeviceToDevice, s) != cudaSuccess) {
            release();
            return cuda_status(cudaGetLastError(), "rf_engine_autotune");
        }
    }
    auto restore = [&]() -> cudaError_t {
        for (size_t q = 0; q < e->allocs.size(); ++q) {
            cudaError_t ce = cudaMemcpyAsync(e->allocs[q], backup[q], e->alloc_bytes[q], cudaMemcpyDeviceToDevice, s);
            if (ce) return ce;
        }
        return cudaStreamSynchronize(s);
    };
    const int variants[3] = {8, 6, 5};
    const int first = e->pw == 32 ? 0 : 1, last = e->pw == 32 ? 3 : 2;     // (see ext_step_kind)
    float best = 1e30f;
    int pick = e->step_minb;
    float times[3] = {0, 0, 0};
    Dev d = e->d;
    Consts c = e->c;
    c.use_graph = 0;
    void* args[] = {&d, &c};
    cudaEvent_t a0, a1;
    cudaEventCreate(&a0); cudaEventCreate(&a1);
    cudaError_t ce = cudaSuccess;
    for (int v = first; v < last && !ce; ++v) {
        void* fn = ext_step_variant(e, variants[v]);
        for (int rep = 0; rep < 2 && !ce; ++rep) {             // first pass warms up
            ce = restore();
            // candidate lists from the current positions (the engine's first step would build them)
            const unsigned gN = (c.N + 255) / 256, gC = (c.cg_cells + 1 + 255) / 256;
            k_force_rebuild<<<1, 1, 0, s>>>(d.sc);
            k_rb_zero<<<gC, 256, 0, s>>>(d, c);
            k_rb_bin<<<gN, 256, 0, s>>>(d, c);
            k_rb_scan_sums<<<e->cg_nb, 1024, 0, s>>>(d, c);
            k_rb_scan_totals<<<1, 32, 0, s>>>(d, c);
            k_rb_scan_apply<<<e->cg_nb, 1024, 0, s>>>(d, c);
            k_rb_scatter<<<gN, 256, 0, s>>>(d, c);
            k_rb_cand<<<(c.N + RF_RB_CTA - 1) / RF_RB_CTA, RF_RB_CTA, 0, s>>>(d, c);
            k_set_target<<<1, 1, 0, s>>>(d.sc, (unsigned long long)steps);
            cudaEventRecord(a0, s);
            for (int q = 0; q < steps && !ce; ++q)
                ce = cudaLaunchKernel(fn, dim3(e->ncta), dim3(128), args, step_smem(e), s);
            cudaEventRecord(a1, s);
            if (!ce) ce = cudaEventSynchronize(a1);
            float ms = 0.f;
            cudaEventElapsedTime(&ms, a0, a1);
            times[v] = ms;
        }
        if (!ce && times[v] < best) { best = times[v]; pick = variants[v]; }
    }
    if (!ce) ce = restore();
    cudaEventDestroy(a0); cudaEventDestroy(a1);
    release();
    if (ce) return cuda_status(ce, "rf_engine_autotune");
    if (pick != e->step_minb) {
        e->step_minb = pick;
        if (e->graph_ok) {                                     // rebuild the step graph with the choice
            if (e->exec) cudaGraphExecDestroy(e->exec);
            if (e->graph) cudaGraphDestroy(e->graph);
            e->exec = nullptr; e->graph = nullptr; e->graph_ok = false;
            if (build_graph(e) == RF_OK) e->graph_ok = true;
            else { cudaGetLastError(); e->c.use_graph = 0; }
        }
    }
    if (choice) *choice = pick;
    if (ms_out) for (int v = 0; v < 3; ++v) ms_out[v] = times[std::min(std::max(v, first), last - 1)];
    return RF_OK;
}

rf_status rf_engine_destroy(rf_engine* e) {
    if (!e) return RF_OK;
    if (e->stream) cudaStreamSynchronize(e->stream);
    if (e->exec) cudaGraphExecDestroy(e->exec);
    if (e->graph) cudaGraphDestroy(e->graph);
    if (e->fexec) cudaGraphExecDestroy(e->fexec);
    if (e->fgraph) cudaGraphDestroy(e->fgraph);
    for (void* p : e->allocs) cudaFree(p);
    if (e->staging) cudaFree(e->staging);
    if (e->stream) cudaStreamDestroy(e->stream);
    delete e;
    return RF_OK;
}

rf_status rf_engine_step(rf_engine* e, uint64_t nsteps) {
    if (!e) { set_error("rf_engine_step: null engine"); return RF_ERR_INVALID; }
    if (nsteps == 0) return RF_OK;
    k_set_target<<<1, 1, 0, e->stream>>>(e->d.sc, (unsigned long long)nsteps);
    RF_CHECK_LAUNCH("k_set_target");
    if (e->graph_ok) {
        RF_CUDA(cudaGraphLaunch(e->exec, e->stream));
        return RF_OK;
    }
    return launch_stream_steps(e, nsteps);
}

rf_status rf_engine_affine_strain(rf_engine* e, const double strain[3]) {
    if (!e || !strain) { set_error("rf_engine_affine_strain: bad arguments"); return RF_ERR_INVALID; }
    if (e->d.nspec > 1) { set_error("rf_engine_affine_strain: one specimen per engine"); return RF_ERR_STATE; }
    for (int a = 0; a < 3; ++a)
        if (!(strain[a] > -0.5 && strain[a] < 0.5)) {
            set_error("rf_engine_affine_strain: strain components must lie in (-0.5, 0.5)");
            return RF_ERR_INVALID;
        }
    cudaStream_t s = e->stream;
    const uint32_t N = e->c.N;
    k_affine_positions<<<(N + 255) / 256, 256, 0, s>>>(e->d, e->c, strain[0], strain[1], strain[2]);
    RF_CHECK_LAUNCH("k_affine_positions");
    if (e->c.kind == RF_TEST_BRAZIL) k_affine_scalars<RF_TEST_BRAZIL><<<1, 32, 0, s>>>(e->d, e->c, strain[0], strain[1], strain[2]);
    else k_affine_scalars<RF_TEST_UNIAXIAL><<<1, 32, 0, s>>>(e->d, e->c, strain[0], strain[1], strain[2]);
    RF_CHECK_LAUNCH("k_affine_scalars");
    return RF_OK;
}

rf_status rf_engine_step_host(rf_engine* e, const float* h_R_in, uint64_t nsteps, float* h_R_out) {
    if (!e) { set_error("rf_engine_step_host: null engine"); return RF_ERR_INVALID; }
    const uint32_t N = e->c.N;
    cudaStream_t s = e->stream;
    if (!e->staging) RF_CUDA(cudaMalloc(&e->staging, 3 * (size_t)N * sizeof(float)));
    if (h_R_in) {
        RF_CUDA(cudaMemcpyAsync(e->staging, h_R_in, 3 * (size_t)N * sizeof(float), cudaMemcpyHostToDevice, s));
        k_planar_to_cur<<<(N + 255) / 256, 256, 0, s>>>(e->staging, e->d);
        RF_CHECK_LAUNCH("k_planar_to_cur");
    }
    rf_status st = rf_engine_step(e, nsteps);
    if (st) return st;
    if (h_R_out) {
        k_cur_to_planar<<<(N + 255) / 256, 256, 0, s>>>(e->d, e->staging);
        RF_CHECK_LAUNCH("k_cur_to_planar");
        RF_CUDA(cudaMemcpyAsync(h_R_out, e->staging, 3 * (size_t)N * sizeof(float), cudaMemcpyDeviceToHost, s));
        RF_CUDA(cudaStreamSynchronize(s));
    }
    return RF_OK;
}

rf_status rf_engine_sync_spec(rf_engine* e, int spec, rf_task* t_out, rf_run_result* r_out) {
    if (!e || spec < 0 || (uint32_t)spec >= e->d.nspec) { set_error("rf_engine_sync_spec: bad arguments"); return RF_ERR_INVALID; }
    DevScalars h, g;
    RF_CUDA(cudaMemcpyAsync(&h, e->d.spec + spec, sizeof(h), cudaMemcpyDeviceToHost, e->stream));
    RF_CUDA(cudaMemcpyAsync(&g, e->d.sc, sizeof(g), cudaMemcpyDeviceToHost, e->stream));
    RF_CUDA(cudaStreamSynchronize(e->stream));
    if (t_out) {
        *t_out = e->d.nspec > 1 ? e->spec_tasks[spec] : e->task;
        rf_compression& K = t_out->Compress;
        K.V = h.V; K.Top = h.Top; K.Bottom = h.Bottom; K.TopR = h.TopR; K.BottomR = h.BottomR;
        K.FractureStress = h.FractureStress; K.FractureStrain = h.FractureStrain; K.Stress = h.Stress;
        K.Strain = h.Strain; K.Loading = h.Loading; K.Fracture = h.Fracture; K.Hd2 = h.Hd2;
        K.size_d = rf_double3{h.size_d[0], h.size_d[1], h.size_d[2]};
        K.center_d = rf_double3{h.center_d[0], h.center_d[1], h.center_d[2]};
        K.size = rf_float3{h.size[0], h.size[1], h.size[2]};
        K.sized2 = rf_float3{h.sized2[0], h.sized2[1], h.sized2[2]};
        K.center = rf_float3{h.center[0], h.center[1], h.center[2]};
    }
    if (r_out) {
        r_out->steps = h.steps;                  // the specimen's own steps (all steps for one specimen)
        r_out->FractureStress = h.FractureStress; r_out->FractureStrain = h.FractureStrain;
        r_out->Stress = h.Stress; r_out->Strain = h.Strain; r_out->Fracture = h.Fracture;
        r_out->broken_bonds = g.broken;          // of the whole engine
        r_out->bonds_initial = e->bonds_initial;
        r_out->error = (rf_status)g.err;
    }
    return RF_OK;
}

rf_status rf_engine_sync(rf_engine* e, rf_task* t_out, rf_run_result* r_out) {
    if (!e) { set_error("rf_engine_sync: null engine"); return RF_ERR_INVALID; }
    if (rf_status st = rf_engine_sync_spec(e, 0, t_out, r_out)) return st;
    if (r_out && e->d.nspec > 1) {
        DevScalars g;
        RF_CUDA(cudaMemcpy(&g, e->d.sc, sizeof(g), cudaMemcpyDeviceToHost));
        r_out->steps = g.steps;
    }
    return RF_OK;
}

rf_status rf_engine_export(rf_engine* e, float* R, float* V, float* W, uint_fast32_t* IL, uint8_t* ILtype,
                           float* _1d_iL, rf_float3* Rij, rf_float3* Oijt, rf_float3* Mijn, rf_float3* Mijt) {
    if (!e) { set_error("rf_engine_export: null engine"); return RF_ERR_INVALID; }
    const uint32_t N = e->c.N, K = e->c.K;
    const size_t NK = (size_t)N * K;
    cudaStream_t s = e->stream;
    RF_CUDA(cudaStreamSynchronize(s));
    DevScalars h;
    RF_CUDA(cudaMemcpy(&h, e->d.sc, sizeof(h), cudaMemcpyDeviceToHost));
    const int cur = (int)(h.steps & 1ull);
    if (!e->staging) RF_CUDA(cudaMalloc(&e->staging, 3 * (size_t)N * sizeof(float)));
    if (e->c.ext) k_delete_pending_ext<<<(N + 127) / 128, 128, 0, s>>>(e->d, e->c);
    else k_delete_pending<<<(N + 127) / 128, 128, 0, s>>>(e->d, e->c);
    RF_CHECK_LAUNCH("k_delete_pending");
    const float4* vecs[3] = {e->d.pos[cur], &e->d.vw[cur]->a, &e->d.vw[cur]->b};
    float* outs[3] = {R, V, W};
    for (int q = 0; q < 3; ++q) {
        if (!outs[q]) continue;
        if (q == 0 && e->c.ext) k_posd_to_planar_f<<<(N + 255) / 256, 256, 0, s>>>(e->d.posd[cur], N, e->staging);
        else k_f4_to_planar<<<(N + 255) / 256, 256, 0, s>>>(vecs[q], N, e->staging, q ? 2u : 1u);
        RF_CHECK_LAUNCH("k_f4_to_planar");
        RF_CUDA(cudaMemcpyAsync(outs[q], e->staging, 3 * (size_t)N * sizeof(float), cudaMemcpyDeviceToHost, s));
        RF_CUDA(cudaStreamSynchronize(s));
    }
    if (IL || ILtype || _1d_iL || Rij || Oijt || Mijn || Mijt) {
        RowBuffers b;
        cudaError_t ce = b.alloc(NK);
        if (!ce) {
            k_rows_export<<<(N + 127) / 128, 128, 0, s>>>(b.IL, b.type, b.iL, b.S, b.S + NK, b.S + 2 * NK, b.S + 3 * NK, e->d, e->c);
            ce = cudaGetLastError();
        }
        if (!ce && IL) ce = cudaMemcpyAsync(IL, b.IL, NK * sizeof(uint_fast32_t), cudaMemcpyDeviceToHost, s);
        if (!ce && ILtype) ce = cudaMemcpyAsync(ILtype, b.type, NK, cudaMemcpyDeviceToHost, s);
        if (!ce && _1d_iL) ce = cudaMemcpyAsync(_1d_iL, b.iL, NK * sizeof(float), cudaMemcpyDeviceToHost, s);
        rf_float3* outs3[4] = {Rij, Oijt, Mijn, Mijt};
        for (int q = 0; q < 4 && !ce; ++q)
            if (outs3[q]) ce = cudaMemcpyAsync(outs3[q], b.S + q * NK, NK * sizeof(rf_float3), cudaMemcpyDeviceToHost, s);
        if (!ce) ce = cudaStreamSynchronize(s);
        if (ce) return cuda_status(ce, "rf_engine_export");
    }
    return RF_OK;
}

rf_status rf_engine_import(rf_engine* e, const float* R, const float* V, const float* W, const uint_fast32_t* IL,
                           const uint8_t* ILtype, const float* _1d_iL, const rf_float3* Rij, const rf_float3* Oijt,
                           const rf_float3* Mijn, const rf_float3* Mijt) {
    if (!e || !R || !V || !W || !IL || !ILtype || !_1d_iL || !Rij || !Oijt || !Mijn || !Mijt) {
        set_error("rf_engine_import: bad arguments");
        return RF_ERR_INVALID;
    }
    if (e->c.ext) {
        set_error("rf_engine_import: the extended model resumes from its own state only (no reference layout)");
        return RF_ERR_STATE;
    }
    const uint32_t N = e->c.N, K = e->c.K;
    const size_t NK = (size_t)N * K;
    cudaStream_t s = e->stream;
    RF_CUDA(cudaStreamSynchronize(s));
    DevScalars h;
    RF_CUDA(cudaMemcpy(&h, e->d.sc, sizeof(h), cudaMemcpyDeviceToHost));
    const int cur = (int)(h.steps & 1ull);
    if (!e->staging) RF_CUDA(cudaMalloc(&e->staging, 3 * (size_t)N * sizeof(float)));
    const float* ins[3] = {R, V, W};
    float4* vecs[3] = {e->d.pos[cur], &e->d.vw[cur]->a, &e->d.vw[cur]->b};
    for (int q = 0; q < 3; ++q) {
        RF_CUDA(cudaMemcpyAsync(e->staging, ins[q], 3 * (size_t)N * sizeof(float), cudaMemcpyHostToDevice, s));
        k_planar_to_f4<<<(N + 255) / 256, 256, 0, s>>>(e->staging, N, vecs[q], q ? 2u : 1u);
        RF_CHECK_LAUNCH("k_planar_to_f4");
        RF_CUDA(cudaStreamSynchronize(s));
    }
    RowBuffers b;
    cudaError_t ce = b.alloc(NK);
    if (!ce) ce = cudaMemcpyAsync(b.IL, IL, NK * sizeof(uint_fast32_t), cudaMemcpyHostToDevice, s);
    if (!ce) ce = cudaMemcpyAsync(b.type, ILtype, NK, cudaMemcpyHostToDevice, s);
    if (!ce) ce = cudaMemcpyAsync(b.iL, _1d_iL, NK * sizeof(float), cudaMemcpyHostToDevice, s);
    const rf_float3* ins3[4] = {Rij, Oijt, Mijn, Mijt};
    for (int q = 0; q < 4 && !ce; ++q)
        ce = cudaMemcpyAsync(b.S + q * NK, ins3[q], NK * sizeof(rf_float3), cudaMemcpyHostToDevice, s);
    uint32_t qb = 0;
    if (!ce) ce = cudaMemsetAsync(e->maxq_dev, 0, sizeof(uint32_t), s);
    if (!ce) { k_count_records<<<148 * 4, 256, 0, s>>>(b.IL, b.type, b.S, N, K, e->maxq_dev); ce = cudaGetLastError(); }
    if (!ce) ce = cudaMemcpyAsync(&qb, e->maxq_dev, sizeof(qb), cudaMemcpyDeviceToHost, s);
    if (!ce) ce = cudaStreamSynchronize(s);
    if (!ce && qb > e->d.QB) {
        set_error("rf_engine_import: a row holds %u bond records, the engine was sized for %u", qb, e->d.QB);
        return RF_ERR_CAPACITY;
    }
    if (!ce) {
        k_rows_import<<<(N + 127) / 128, 128, 0, s>>>(b.IL, b.type, b.iL, b.S, b.S + NK, b.S + 2 * NK, b.S + 3 * NK, e->d, e->c);
        ce = cudaGetLastError();
    }
    if (!ce) {
        k_force_rebuild<<<1, 1, 0, s>>>(e->d.sc);
        ce = cudaGetLastError();
    }
    if (!ce) ce = cudaStreamSynchronize(s);
    if (ce) return cuda_status(ce, "rf_engine_import");
    return RF_OK;
}

rf_status rf_engine_curve_spec(rf_engine* e, int spec, double* curve, uint64_t cap, uint64_t* n) {
    if (!e || spec < 0 || (uint32_t)spec >= e->d.nspec) { set_error("rf_engine_curve: bad arguments"); return RF_ERR_INVALID; }
    DevScalars h;
    RF_CUDA(cudaStreamSynchronize(e->stream));
    RF_CUDA(cudaMemcpy(&h, e->d.spec + spec, sizeof(h), cudaMemcpyDeviceToHost));
    uint64_t m = h.curve_n < e->c.curve_cap ? h.curve_n : e->c.curve_cap;
    if (n) *n = h.curve_n;
    if (curve && cap) {
        if (m > cap) m = cap;
        RF_CUDA(cudaMemcpy(curve, e->d.curve + 3 * (size_t)spec * e->c.curve_cap, 3 * m * sizeof(double),
                           cudaMemcpyDeviceToHost));
    }
    return RF_OK;
}

}  // extern "C"

// Checkpoint files: header, the rf_task, the SaveAllData payload (rf_io.cpp).
namespace rf {
rf_status io_write_all(std::ostream& f, int id_bytes, const rf_sample* S, uint64_t pn, uint64_t N, uint32_t K,
                       float acut, const float* F, const float* V, const float* R, const float* M, const float* W,
                       const float* Q, const uint_fast32_t* IL, const uint8_t* ILtype, const float* _1d_iL,
                       const rf_float3* Rij, const rf_float3* Oijt, const rf_float3* Fijn, const rf_float3* Fijt,
                       const rf_float3* Mijn, const rf_float3* Mijt, const rf_float3* Mijadd);
rf_status io_read_all(std::istream& f, int id_bytes, rf_sample* S, uint64_t* pn, uint64_t* N_out, uint32_t* K_out,
                      float* acut, float* F, float* V, float* R, float* M, float* W, float* Q, uint_fast32_t* IL,
                      uint8_t* ILtype, float* _1d_iL, rf_float3* Rij, rf_float3* Oijt, rf_float3* Fijn,
                      rf_float3* Fijt, rf_float3* Mijn, rf_float3* Mijt, rf_float3* Mijadd);
}  // namespace rf

namespace {
const char kCkptMagic[8] = {'R', 'F', 'B', '2', 'C', 'K', 'P', 'T'};
struct CkptHeader {
    char magic[8];
    uint32_t version, id_bytes, model, reserved;
    uint64_t task_bytes;
};
}  // namespace

extern "C" {

rf_status rf_engine_checkpoint(rf_engine* e, const char* path) {
    if (!e || !path) { set_error("rf_engine_checkpoint: bad arguments"); return RF_ERR_INVALID; }
    if (e->c.ext) {
        set_error("rf_engine_checkpoint: the reference model only (the extended model has no reference layout)");
        return RF_ERR_STATE;
    }
    rf_task t;
    rf_run_result r;
    TRY(rf_engine_sync(e, &t, &r));
    const uint64_t N = e->c.N, K = e->c.K, NK = N * K;
    std::vector<float> R(3 * N), V(3 * N), W(3 * N), iL(NK);
    std::vector<uint_fast32_t> IL(NK);
    std::vector<uint8_t> ty(NK);
    std::vector<rf_float3> Rij(NK), Oijt(NK), Mijn(NK), Mijt(NK);
    TRY(rf_engine_export(e, R.data(), V.data(), W.data(), IL.data(), ty.data(), iL.data(), Rij.data(), Oijt.data(),
                         Mijn.data(), Mijt.data()));
    std::ofstream f(path, std::ios::out | std::ios::binary | std::ios::trunc);
    if (!f) { set_error("rf_engine_checkpoint: cannot open %s", path); return RF_ERR_INVALID; }
    CkptHeader h;
    std::memcpy(h.magic, kCkptMagic, 8);
    h.version = 1; h.id_bytes = (uint32_t)sizeof(uint_fast32_t); h.model = 0; h.reserved = 0;
    h.task_bytes = sizeof(rf_task);
    f.write((const char*)&h, sizeof(h));
    f.write((const char*)&t, sizeof(t));
    TRY(io_write_all(f, (int)sizeof(uint_fast32_t), &t.S, 0, N, (uint32_t)K, t.acut, nullptr, V.data(), R.data(),
                     nullptr, W.data(), nullptr, IL.data(), ty.data(), iL.data(), Rij.data(), Oijt.data(), nullptr,
                     nullptr, Mijn.data(), Mijt.data(), nullptr));
    f.close();
    if (!f) { set_error("rf_engine_checkpoint: write to %s failed", path); return RF_ERR_INVALID; }
    return RF_OK;
}

rf_status rf_engine_restore(const char* path, rf_engine** out) {
    if (!path || !out) { set_error("rf_engine_restore: bad arguments"); return RF_ERR_INVALID; }
    *out = nullptr;
    std::ifstream f(path, std::ios::in | std::ios::binary);
    if (!f) { set_error("rf_engine_restore: cannot open %s", path); return RF_ERR_INVALID; }
    CkptHeader h;
    f.read((char*)&h, sizeof(h));
    if (!f || std::memcmp(h.magic, kCkptMagic, 8) != 0 || h.version != 1 || h.model != 0 ||
        h.id_bytes != sizeof(uint_fast32_t) || h.task_bytes != sizeof(rf_task)) {
        set_error("rf_engine_restore: %s is not a version-1 checkpoint of this build", path);
        return RF_ERR_INVALID;
    }
    rf_task t;
    f.read((char*)&t, sizeof(t));
    const std::streampos body = f.tellg();
    uint64_t N = 0;
    uint32_t K = 0;
    TRY(io_read_all(f, (int)h.id_bytes, nullptr, nullptr, &N, &K, nullptr, nullptr, nullptr, nullptr, nullptr,
                    nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr,
                    nullptr));
    if (N != t.N || K != t.K) { set_error("rf_engine_restore: the payload does not match the task"); return RF_ERR_INVALID; }
    const uint64_t NK = N * K;
    std::vector<float> R(3 * N), V(3 * N), W(3 * N), iL(NK);
    std::vector<uint_fast32_t> IL(NK);
    std::vector<uint8_t> ty(NK);
    std::vector<rf_float3> Rij(NK), Oijt(NK), Mijn(NK), Mijt(NK);
    f.clear();
    f.seekg(body);
    TRY(io_read_all(f, (int)h.id_bytes, nullptr, nullptr, &N, &K, nullptr, nullptr, V.data(), R.data(), nullptr,
                    W.data(), nullptr, IL.data(), ty.data(), iL.data(), Rij.data(), Oijt.data(), nullptr, nullptr,
                    Mijn.data(), Mijt.data(), nullptr));
    RowsIn rows{IL.data(), ty.data(), iL.data(), Rij.data(), Oijt.data(), Mijn.data(), Mijt.data()};
    rf_engine* e = nullptr;
    TRY(engine_create_impl(&t, R.data(), nullptr, nullptr, nullptr, &e, nullptr, &rows));
    const rf_status st = rf_engine_import(e, R.data(), V.data(), W.data(), IL.data(), ty.data(), iL.data(), Rij.data(),
                                          Oijt.data(), Mijn.data(), Mijt.data());
    if (st != RF_OK) { rf_engine_destroy(e); return st; }
    *out = e;
    return RF_OK;
}

rf_status rf_engine_curve(rf_engine* e, double* curve, uint64_t cap, uint64_t* n) {
    return rf_engine_curve_spec(e, 0, curve, cap, n);
}

int rf_engine_batch_size(rf_engine* e) { return e ? (int)e->d.nspec : 0; }

rf_status rf_engine_spec_info(rf_engine* e, int spec, uint64_t* first, uint64_t* count, double* x_offset,
                              rf_task* task) {
    if (!e || spec < 0 || (uint32_t)spec >= e->d.nspec) { set_error("rf_engine_spec_info: bad arguments"); return RF_ERR_INVALID; }
    const bool b = e->d.nspec > 1;
    if (first) *first = b ? e->spec_p0[spec] : 0;
    if (count) *count = b ? e->spec_n[spec] : e->c.N;
    if (x_offset) *x_offset = b ? e->spec_xoff[spec] : 0.0;
    if (task) *task = b ? e->spec_tasks[spec] : e->task;
    return RF_OK;
}

rf_status rf_engine_counters(rf_engine* e, uint64_t* out, int n) {
    if (!e || !out || n <= 0) { set_error("rf_engine_counters: bad arguments"); return RF_ERR_INVALID; }
    cudaStream_t s = e->stream;
    RF_CUDA(cudaMemsetAsync(e->counters_dev, 0, 4 * sizeof(unsigned long long), s));
    k_counters<<<148 * 4, 256, 0, s>>>(e->d, e->c, e->counters_dev);
    RF_CHECK_LAUNCH("k_counters");
    unsigned long long cnt[4];
    DevScalars h;
    RF_CUDA(cudaMemcpyAsync(cnt, e->counters_dev, sizeof(cnt), cudaMemcpyDeviceToHost, s));
    RF_CUDA(cudaMemcpyAsync(&h, e->d.sc, sizeof(h), cudaMemcpyDeviceToHost, s));
    RF_CUDA(cudaStreamSynchronize(s));
    const uint64_t v[5] = {h.steps, h.rebuilds, cnt[0], cnt[1], cnt[2]};
    for (int q = 0; q < n && q < 5; ++q) out[q] = v[q];
    return RF_OK;
}

int rf_engine_launches_per_step(void) { return 1; }
rf_stream rf_engine_stream(rf_engine* e) { return e ? (rf_stream)e->stream : nullptr; }
int rf_engine_uses_graph(rf_engine* e) { return (e && e->graph_ok) ? 1 : 0; }

}  // extern "C"
