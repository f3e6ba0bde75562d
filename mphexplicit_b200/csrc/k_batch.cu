// k_batch.cu — the batched form: many independent MPH-WC scenes of one
// dimension stepped together on sm_100a (mph_batch_* in mph_b200.h).
//
// All scenes share one set of particle arrays; scene s owns the slots
// [pbase[s], pbase[s+1]), kept sorted by the scene's own cell id (the CellId of
// main.cpp:96-100; wall and fluid particles share one cell range here).  One
// step of every scene is
//   move     convection (main.cpp:1605-1615), periodic wrap (2306-2317) and the
//            rebuild test of neighborCalculation (1086-1108), per scene;
//   rebuild  a stable counting sort by cell of the scenes whose test fired
//            (histogram, per-scene scan, place, rank + gather, commit); each
//            of these kernels returns at once when no scene asked for it, so
//            the host never waits on the decision;
//   sweep A  DensityP, DivergenceP (+ DensityA, GravityCenter with surface
//            tension) and the PressureP / PressureA values (1631-1662,
//            1665-1740, 1831-1906);
//   sweep B  PressureP, PressureA, DiffuseInterface and ViscosityV forces,
//            gravity, acceleration (1742-2010).
// The sweeps come in two forms.  By default a neighbour table per particle,
// built on the device when a scene is sorted (k_bt_table) and walked by a thread
// per particle (k_bt_a, k_bt_b).  Where a tile shape is asked for, or the table
// does not fit in memory, they are persistent kernels: every CTA takes (scene,
// cell tile) items from a queue, stages the tile and its one-cell halo in shared
// memory and evaluates the tile's pairs from there, no list stored.  Both visit a
// particle's pairs in the same order with the same expressions; the table form
// takes its displacements from the FP64 positions, those of the pressure forces
// rounded as a tile of the default shape rounds them, so that a batch gives the
// same flow in both.  Staged
// positions are tile-relative, split into a part on a power-of-two grid and
// an FP32 remainder, so x_j - x_i is the true displacement rounded once to
// FP32.  The density sweep's DensityP / DivergenceP pairs are evaluated in
// FP64 on that displacement (the pressure is a bulk modulus times a small
// difference of two numbers near N0p), every other pair term in FP32 with
// the mixed form's formulas (Kahan-compensated short-range force sums);
// positions and velocities are integrated in FP64.  A tile whose halo does not fit in
// shared memory is split in two until it does.  mph_batch_step replays K steps
// as one CUDA graph; mph_batch_autotune times the candidate tile shapes on the
// batch itself and keeps the fastest.
#include <algorithm>
#include <array>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>
#include <nvtx3/nvToolsExt.h>
#include "mph_internal.h"
#include "mph_pair32.cuh"

namespace mph {
namespace {

constexpr int kStack = 64;         // pending sub-tiles per CTA
constexpr int kMaxThreads = 256;   // CTA size bound of the sweeps
constexpr int kGraphSteps = MPH_BATCH_GRAPH_STEPS;  // steps per captured graph

enum : int {
    BERR_CAPACITY = 1,   // a one-cell tile did not fit in shared memory
    BERR_NONFINITE = 2,  // NaN/Inf velocity
};

// Per-scene constants: FP64 values for the integration, FP32 values for the
// pair terms (field names follow MixConst so the shared pair helpers apply).
struct alignas(16) BScene {
    int n, pbase, cbase, tot;
    int cc[3], tile[3];
    int has_st, ratio_all_one, uniform_mu;
    int nfl, fbase;                     // fluid particles, first entry of the scene in flist
    int pad0[3];
    double dmin[3], width[3], inv_width[3], cell_width[3], half_width[3];
    double dt, shift_thr, grid, inv_grid, vol_d, n0p_d;
    double rp2_d, inv_rp_d, cp_d, cp_m2_d;  // FP64 density pairs
    double gravity[3];
    double density[MPH_TYPE_COUNT], bulk_modulus_d[MPH_TYPE_COUNT], bulk_viscosity_d[MPH_TYPE_COUNT];
    int ttile[3];                       // table form: the default tile, whose rounding it follows
    int hw_hi[3], pad1[2];              // high word of half_width
    double rgrid, inv_rgrid;            // table form: grid of that tile's hi parts
    float cw32[3];                      // table form: cell width, for the lists
    float list_r2, lists_r2;            // table form: cut-offs of the two lists
    float pad2[3];
    float cut2_a, cut2_b, short_r2;
    float rp2_pre;                      // RP^2 a little widened: FP32 pre-filter of the FP64 density pairs
    float ra2, rp2, rv2, rg2;
    float inv_ra, inv_rp, inv_rv, inv_rg;
    float ca, cp, cg, cv;
    float cp_m2, cg_m2, ca_inv;
    float p_a, p_b, v_a, v_b;
    float vol, vol_over_l0, n0a, n0p, inv_r2g_rg, l0;
    float visc_mu[MPH_TYPE_COUNT][MPH_TYPE_COUNT];
    float ratio[MPH_TYPE_COUNT][MPH_TYPE_COUNT];
    float a_k[MPH_TYPE_COUNT], cof_a[MPH_TYPE_COUNT];
};
static_assert(sizeof(BScene) % 16 == 0, "BScene is copied as 16-byte words");

// Kernel arguments (by value): sizes and device pointers, fixed between
// set-ups so that captured graphs stay valid.
struct BatchDev {
    int n, S, n_items, cap;
    int hmax, ncol;               // halo cells / interior columns of the largest tile
    const BScene* scenes;
    const int* sid;               // scene of every slot
    const int4* items;            // (scene, x0, y0, z0) of every tile, largest first
    double4* pos;                 // x, y, z, (double)type
    double4* vel;
    double4* snap;                // positions at the scene's last sort
    int* pidx;                    // index in the scene's input order
    double4* pos_t;
    double4* vel_t;
    int* pidx_t;
    int* key;                     // global cell of a re-sorted particle
    int* slot;
    int* tmp;
    int* counts;                  // [cells], zero between sorts
    int* start;                   // [cells + 1]: first slot of every cell
    float4* vp;                   // sweep A -> B: 2-D (vx, vy, P, type), 3-D (vx, vy, vz, P)
    float4* gc;                   // sweep A -> B: (GravityCenter, PressureA)
    int* flags;                   // [S]: the scene's rebuild test fired
    // table form
    int table, cells, tcap, tcap_s;   // on; cells of all scenes; entries per particle of the two lists
    const int* cell_scene;        // scene of every cell
    int* home;                    // cell of the particle at the last sort (10 bits per axis)
    float4* rel;                  // position in that cell at the last sort, type (the lists are built from it)
    float4* v32;                  // (vx, vy, vz, type)
    float4* tile2;                // 2-D: position in its default tile, hi.xy and lo.xy
    int* cfluid;                  // [cells]: the cell holds fluid
    int* fcount;                  // [S]: fluid slots listed so far
    int* flist;                   // slots of the fluid particles, scene by scene
    uint4* tab;                   // [tcap / 4][n]: entries in candidate order
    uint4* tab_s;                 // [tcap_s / 4][n]: those within RadiusP + 2 MARGIN
    int* tcnt;
    int* tcnt_s;
    const int2* items_a;          // (scene, first slot) of every block of sweep A
    const int2* items_b;          // (scene, first entry of flist) of every block of sweep B
    int* ctl;                     // [8] see below
};
// ctl: 0 any scene to sort, 1 error bits, 2/3 sweep A queue head/done,
// 4/5 sweep B queue head/done, 6 scene sorts so far, 7 tile splits so far.

__device__ __forceinline__ double bmod(double x, double w) { return x - w * floor(x / w); }
__device__ __forceinline__ double bmod_fast(double x, double w) {
    return (x >= 0.0 && x < 0.75 * w) ? x : bmod(x, w);
}
__device__ __forceinline__ int wrapi(int v, int m) { return ((v % m) + m) % m; }

__device__ __forceinline__ void cell_of(const BScene& c, const double4& p, int& cx, int& cy, int& cz) {
    cx = wrapi((int)floor((p.x - c.dmin[0]) / c.cell_width[0]), c.cc[0]);
    cy = wrapi((int)floor((p.y - c.dmin[1]) / c.cell_width[1]), c.cc[1]);
    cz = wrapi((int)floor((p.z - c.dmin[2]) / c.cell_width[2]), c.cc[2]);
}

__device__ __forceinline__ double drint(double x) {  // rint for |x| < 2^51, two additions
    const double m = 6755399441055744.0;  // 1.5 * 2^52
    return __dadd_rn(__dadd_rn(x, m), -m);
}

// Origin of the default tile of cell coordinate c on axis k (one halo cell below).
__device__ __forceinline__ double tile_origin(const BScene& s, int k, int c) {
    return s.dmin[k] + (double)(c / s.ttile[k] * s.ttile[k] - 1) * s.cell_width[k];
}
// A tile-relative coordinate's part on the tile's grid, in steps, and the rest.
__device__ __forceinline__ void tile_split(const BScene& s, double d, double& hq, float& lo) {
    hq = drint(d * s.inv_rgrid);
    lo = (float)(d - hq * s.rgrid);
}
// 2-D: a particle's position in the default tile of its home cell, hi.xy and lo.xy.
__device__ __forceinline__ float4 tile_pos(const BScene& s, const double4& p, int h) {
    const double x[2] = {p.x, p.y};
    float hi[2], lo[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int c = (h >> (10 * k)) & 1023;
        const double ec = ((double)(c - c / s.ttile[k] * s.ttile[k] + 1) + 0.5) * s.cell_width[k];
        double d = x[k] - tile_origin(s, k, c), hq;
        d -= s.width[k] * rint((d - ec) * s.inv_width[k]);
        tile_split(s, d, hq, lo[k]);
        hi[k] = (float)(hq * s.rgrid);
    }
    return make_float4(hi[0], hi[1], lo[0], lo[1]);
}

// ---- per step: move -----------------------------------------------------------

template <bool TABLE>
__global__ void __launch_bounds__(256) k_bt_move(BatchDev b) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= b.n) return;
    const int s = b.sid[i];
    const BScene& c = b.scenes[s];
    double4 p = b.pos[i];
    const double4 v = b.vel[i];
    if ((int)p.w < 2) {
        p.x += v.x * c.dt;
        p.y += v.y * c.dt;
        p.z += v.z * c.dt;
    }
    p.x = bmod_fast(p.x - c.dmin[0], c.width[0]) + c.dmin[0];
    p.y = bmod_fast(p.y - c.dmin[1], c.width[1]) + c.dmin[1];
    p.z = bmod_fast(p.z - c.dmin[2], c.width[2]) + c.dmin[2];
    b.pos[i] = p;
    if (TABLE) {
        b.v32[i] = make_float4((float)v.x, (float)v.y, (float)v.z, __int_as_float((int)p.w));
        if (b.tile2) b.tile2[i] = tile_pos(c, p, b.home[i]);
    }
    const double4 q = b.snap[i];
    const double d0 = bmod_fast(p.x - q.x + c.half_width[0], c.width[0]) - c.half_width[0];
    const double d1 = bmod_fast(p.y - q.y + c.half_width[1], c.width[1]) - c.half_width[1];
    const double d2 = bmod_fast(p.z - q.z + c.half_width[2], c.width[2]) - c.half_width[2];
    if (d0 * d0 + d1 * d1 + d2 * d2 > c.shift_thr) {
        b.flags[s] = 1;
        b.ctl[0] = 1;
    }
}

// ---- rebuild: stable counting sort of the flagged scenes ----------------------

__global__ void __launch_bounds__(256) k_bt_hist(BatchDev b) {
    if (b.ctl[0] == 0) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= b.n) return;
    const int s = b.sid[i];
    if (!b.flags[s]) return;
    const BScene& c = b.scenes[s];
    int cx, cy, cz;
    cell_of(c, b.pos[i], cx, cy, cz);
    const int key = c.cbase + (cx * c.cc[1] + cy) * c.cc[2] + cz;
    b.key[i] = key;
    b.slot[i] = atomicAdd(&b.counts[key], 1);
}

// One block per scene: exclusive scan of the scene's cell counts into start
// (offset by the scene's first slot), counts reset to zero.
__global__ void __launch_bounds__(1024) k_bt_scan(BatchDev b) {
    if (b.ctl[0] == 0) return;
    const int s = blockIdx.x;
    if (!b.flags[s]) return;
    __shared__ int part[1024];
    const BScene& c = b.scenes[s];
    int* counts = b.counts + c.cbase;
    int* out = b.start + c.cbase;
    const int m = c.tot, t = threadIdx.x;
    const int chunk = (m + blockDim.x - 1) / blockDim.x;
    const int lo = min(m, t * chunk), hi = min(m, lo + chunk);
    int sum = 0;
    for (int k = lo; k < hi; ++k) sum += counts[k];
    part[t] = sum;
    __syncthreads();
    for (int off = 1; off < (int)blockDim.x; off <<= 1) {  // Hillis-Steele inclusive scan
        const int v = t >= off ? part[t - off] : 0;
        __syncthreads();
        part[t] += v;
        __syncthreads();
    }
    int run = c.pbase + part[t] - sum;
    for (int k = lo; k < hi; ++k) {
        out[k] = run;
        run += counts[k];
        counts[k] = 0;
        if (b.table) b.cfluid[c.cbase + k] = 0;
    }
    if (b.table && t == 0) b.fcount[s] = 0;
}

__global__ void __launch_bounds__(256) k_bt_place(BatchDev b) {
    if (b.ctl[0] == 0) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= b.n || !b.flags[b.sid[i]]) return;
    b.tmp[b.start[b.key[i]] + b.slot[i]] = i;
}

// Order each cell's particles by their previous slot (a stable sort) and
// gather the state into the temporaries.
__global__ void __launch_bounds__(256) k_bt_gather(BatchDev b) {
    if (b.ctl[0] == 0) return;
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= b.n || !b.flags[b.sid[p]]) return;
    const int i = b.tmp[p];
    const int key = b.key[i];
    const int lo = b.start[key], hi = b.start[key + 1];
    int rank = 0;
    for (int q = lo; q < hi; ++q) rank += b.tmp[q] < i;
    const int dst = lo + rank;
    b.pos_t[dst] = b.pos[i];
    b.vel_t[dst] = b.vel[i];
    b.pidx_t[dst] = b.pidx[i];
}

// What the table form keeps per particle of a sorted scene: its home cell, its
// FP32 position in it, and, for the fluid, the cell's mark and a place in the
// scene's fluid list (any order: a particle's result does not depend on it; warp
// by warp, so that neighbouring lanes of sweep B are neighbouring slots).  All
// lanes take part.
__device__ __forceinline__ void table_home(const BatchDev& b, bool on, int p, int s, const double4& x,
                                           const double4& v) {
    bool fluid = false;
    if (on) {
        const BScene& c = b.scenes[s];
        int cx, cy, cz;
        cell_of(c, x, cx, cy, cz);
        b.home[p] = cx | (cy << 10) | (cz << 20);
        const int hc[3] = {cx, cy, cz};
        const double xd[3] = {x.x, x.y, x.z};
        float r[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            double d = xd[k] - (c.dmin[k] + (double)hc[k] * c.cell_width[k]);
            if (d > c.half_width[k]) d -= c.width[k];  // minimum image from the home cell
            if (d < -c.half_width[k]) d += c.width[k];
            r[k] = (float)d;
        }
        const float type = __int_as_float((int)x.w);
        b.rel[p] = make_float4(r[0], r[1], r[2], type);
        b.v32[p] = make_float4((float)v.x, (float)v.y, (float)v.z, type);
        if (b.tile2) b.tile2[p] = tile_pos(c, x, b.home[p]);
        fluid = (int)x.w < 2;
        if (fluid) b.cfluid[c.cbase + (cx * c.cc[1] + cy) * c.cc[2] + cz] = 1;
    }
    const unsigned same = __match_any_sync(0xffffffffu, fluid ? s : -1);
    if (fluid) {
        const int lane = threadIdx.x & 31, lead = __ffs(same) - 1;
        int at = 0;
        if (lane == lead) at = atomicAdd(&b.fcount[s], __popc(same));
        at = __shfl_sync(same, at, lead);
        b.flist[b.scenes[s].fbase + at + __popc(same & ((1u << lane) - 1u))] = p;
    }
}

template <bool TABLE>
__global__ void __launch_bounds__(256) k_bt_commit(BatchDev b) {
    if (b.ctl[0] == 0) return;
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    const int s = p < b.n ? b.sid[p] : 0;
    const bool on = p < b.n && b.flags[s] != 0;
    double4 x = make_double4(0, 0, 0, 0), v = x;
    if (on) {
        x = b.pos_t[p];
        v = b.vel_t[p];
        b.pos[p] = x;
        b.snap[p] = x;
        b.vel[p] = v;
        b.pidx[p] = b.pidx_t[p];
    }
    if (TABLE) table_home(b, on, p, s, x, v);
}

// The same from the positions of the last sort, for a batch that turns to the
// table form between sorts (its cells and slots are those of that sort).
__global__ void __launch_bounds__(256) k_bt_home(BatchDev b) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    const bool on = p < b.n;
    double4 x = make_double4(0, 0, 0, 0), v = x;
    if (on) {
        x = b.snap[p];
        v = b.vel[p];
    }
    table_home(b, on, p, on ? b.sid[p] : 0, x, v);
}

// ---- the neighbour table ---------------------------------------------------------

constexpr int kCross = 64;                       // k_bt_table: a stencil cell of another tile
constexpr unsigned kEntryCross = 0x80000000u;    // ... and its entries (2-D)
constexpr int kTabWarps = 4;
constexpr int kTabLanes = 4;                 // lanes per particle
constexpr int kTabParts = 32 / kTabLanes;    // particles per warp

// The lists of the flagged scenes (all: every scene).  One block per cell, cells
// dealt over a fixed grid, so that a step without a sort costs one short launch;
// a warp takes eight of the cell's particles at a time, four lanes each: a step
// mostly sorts a few scenes of the batch, and with a lane per particle their
// cells left most of the GPU idle behind long serial candidate loops.
// The candidates of the 3^D cells come 32 at a time, those near the box around
// the warp's particles are compacted in order into shared memory, each lane tests
// every fourth of them in FP32, and a ballot numbers the hits in candidate order.
// An entry is the neighbour's slot, in 2-D with the top bit set where its default
// tile is another one (tile2 is then not in this particle's tile); the particle
// itself is left out.  A list longer than its table is counted and the
// sweeps walk the cells for that particle.  Without surface tension only the fluid
// needs the whole list (sweep B), and a wall with no fluid in reach needs none:
// nothing reads its pressure.
template <int DIM>
__global__ void __launch_bounds__(32 * kTabWarps, 8) k_bt_table(BatchDev b, int all) {
    if (!all && b.ctl[0] == 0) return;
    __shared__ float4 cand[kTabWarps][32];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int sub = lane & (kTabLanes - 1), part = lane / kTabLanes;
    const size_t n = (size_t)b.n;
    const float kInf = __int_as_float(0x7f800000);
    constexpr int NST = DIM == 3 ? 27 : 9;
    float4* cw = cand[wib];
    unsigned* const tab = reinterpret_cast<unsigned*>(b.tab);
    unsigned* const tab_s = reinterpret_cast<unsigned*>(b.tab_s);
    for (int cell = blockIdx.x; cell < b.cells; cell += gridDim.x) {
        const int s = b.cell_scene[cell];
        if (!all && !b.flags[s]) continue;
        const int hb = b.start[cell], he = b.start[cell + 1];
        if (hb + wib * kTabParts >= he) continue;
        const BScene& c = b.scenes[s];
        const int lc = cell - c.cbase;
        const int ix = lc / (c.cc[1] * c.cc[2]), iy = (lc / c.cc[2]) % c.cc[1], iz = lc % c.cc[2];
        int st_b = 0, st_e = 0, st_code = 0;  // lane q: slots of stencil cell q, its code
        bool fl = false;
        if (lane < NST) {
            const int ax = DIM == 3 ? lane / 9 : lane / 3, ay = DIM == 3 ? (lane / 3) % 3 : lane % 3,
                      az = DIM == 3 ? lane % 3 : 1;
            const int k = c.cbase + (wrapi(ix + ax - 1, c.cc[0]) * c.cc[1] + wrapi(iy + ay - 1, c.cc[1])) * c.cc[2] +
                          (DIM == 3 ? wrapi(iz + az - 1, c.cc[2]) : 0);
            st_b = b.start[k];
            st_e = b.start[k + 1];
            st_code = ax * 9 + ay * 3 + az;
            fl = b.cfluid[k] != 0;
            if (DIM == 2) {  // the stencil cell's tile, beyond a periodic face another one
                const int jx = ix + ax - 1, jy = iy + ay - 1;
                const bool cross = jx < 0 || jx >= c.cc[0] || jy < 0 || jy >= c.cc[1] ||
                                   jx / c.ttile[0] != ix / c.ttile[0] || jy / c.ttile[1] != iy / c.ttile[1];
                if (cross) st_code |= kCross;
            }
        }
        const bool near_fluid = __any_sync(0xffffffffu, fl);
        const float list_r2 = c.list_r2, lists_r2 = c.lists_r2;
        const float cwx = c.cw32[0], cwy = c.cw32[1], cwz = c.cw32[2];
        for (int h0 = hb + wib * kTabParts; h0 < he; h0 += kTabWarps * kTabParts) {
            const int i = h0 + part;
            const bool active = i < he;
            if (!near_fluid) {  // walls out of reach of the fluid
                if (active && sub == 0) b.tcnt[i] = b.tcnt_s[i] = 0;
                continue;
            }
            const float4 pi = b.rel[active ? i : hb];
            const bool is_wall = __float_as_int(pi.w) >= 2;
            const bool whole = !is_wall || c.has_st;
            float b0x = active ? pi.x : kInf, b0y = active ? pi.y : kInf, b0z = active ? pi.z : kInf;
            float b1x = active ? pi.x : -kInf, b1y = active ? pi.y : -kInf, b1z = active ? pi.z : -kInf;
            for (int o = 16; o >= kTabLanes; o >>= 1) {
                b0x = fminf(b0x, __shfl_xor_sync(0xffffffffu, b0x, o));
                b0y = fminf(b0y, __shfl_xor_sync(0xffffffffu, b0y, o));
                b1x = fmaxf(b1x, __shfl_xor_sync(0xffffffffu, b1x, o));
                b1y = fmaxf(b1y, __shfl_xor_sync(0xffffffffu, b1y, o));
                if (DIM == 3) {
                    b0z = fminf(b0z, __shfl_xor_sync(0xffffffffu, b0z, o));
                    b1z = fmaxf(b1z, __shfl_xor_sync(0xffffffffu, b1z, o));
                }
            }
            int cs = 0, cl = 0;
            bool any_fluid = !is_wall;
            const int self = active ? i : -1;
            for (int q = 0; q < NST; ++q) {
                const int cb0 = __shfl_sync(0xffffffffu, st_b, q), ce = __shfl_sync(0xffffffffu, st_e, q);
                const int code_x = __shfl_sync(0xffffffffu, st_code, q), code = code_x & 31;
                const unsigned cross = DIM == 2 && (code_x & kCross) ? kEntryCross : 0u;
                const float gx = (float)(code / 9 - 1) * cwx, gy = (float)((code / 3) % 3 - 1) * cwy,
                            gz = DIM == 3 ? (float)(code % 3 - 1) * cwz : 0.f;
                const float ox = gx - pi.x, oy = gy - pi.y, oz = DIM == 3 ? gz - pi.z : 0.f;
                for (int cb = cb0; cb < ce; cb += 32) {
                    bool near = false;
                    float4 qc = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (cb + lane < ce) {
                        qc = b.rel[cb + lane];
                        const float ax = qc.x + gx, ay = qc.y + gy, az = DIM == 3 ? qc.z + gz : 0.f;
                        const float ex = fmaxf(0.f, fmaxf(b0x - ax, ax - b1x));
                        const float ey = fmaxf(0.f, fmaxf(b0y - ay, ay - b1y));
                        const float ez = DIM == 3 ? fmaxf(0.f, fmaxf(b0z - az, az - b1z)) : 0.f;
                        near = ex * ex + ey * ey + ez * ez < list_r2;
                    }
                    const unsigned kept = __ballot_sync(0xffffffffu, near);
                    __syncwarp();
                    if (near) {  // .w: slot, sign bit for a wall
                        const bool wall = __float_as_int(qc.w) >= 2;
                        qc.w = __int_as_float((cb + lane) | (wall ? (int)0x80000000 : 0));
                        cw[__popc(kept & ((1u << lane) - 1u))] = qc;
                    }
                    __syncwarp();
                    const int mm = __popc(kept);
                    for (int t0 = 0; t0 < mm; t0 += kTabLanes) {
                        const float4 qq = cw[min(t0 + sub, mm - 1)];
                        const float dx = qq.x + ox, dy = qq.y + oy, dz = DIM == 3 ? qq.z + oz : 0.f;
                        const float r2 = dx * dx + dy * dy + dz * dz;
                        const int jw = __float_as_int(qq.w), j = jw & 0x7fffffff;
                        const bool hit = active && t0 + sub < mm && r2 < list_r2 && j != self;
                        const unsigned entry = (unsigned)j | cross;
                        const unsigned group = ((1u << kTabLanes) - 1u) << (part * kTabLanes);
                        const unsigned below = group & ((1u << lane) - 1u);
                        const unsigned hits = __ballot_sync(0xffffffffu, hit);
                        if (hits == 0u) continue;
                        const unsigned near_s = __ballot_sync(0xffffffffu, hit && r2 < lists_r2);
                        any_fluid |= (__ballot_sync(0xffffffffu, hit && jw >= 0) & group) != 0u;
                        if (hit && whole) {
                            const int at = cl + __popc(hits & below);
                            if (at < b.tcap) tab[((size_t)(at >> 2) * n + i) * 4 + (at & 3)] = entry;
                        }
                        cl += __popc(hits & group);
                        if (hit && r2 < lists_r2) {
                            const int at = cs + __popc(near_s & below);
                            if (at < b.tcap_s) tab_s[((size_t)(at >> 2) * n + i) * 4 + (at & 3)] = entry;
                        }
                        cs += __popc(near_s & group);
                    }
                }
            }
            if (active && sub == 0) {
                b.tcnt_s[i] = any_fluid ? cs : 0;
                b.tcnt[i] = any_fluid && whole ? cl : 0;
            }
        }
    }
}

// ---- the sweeps over the table ----------------------------------------------------

__device__ __forceinline__ void load_scene(const BatchDev& b, int s, BScene& sc) {
    const int4* src = reinterpret_cast<const int4*>(b.scenes + s);
    int4* dst = reinterpret_cast<int4*>(&sc);
    for (int k = threadIdx.x; k < (int)(sizeof(BScene) / 16); k += blockDim.x) dst[k] = src[k];
    __syncthreads();
}

// The pairs' displacements.  A pair's positions in i's default tile give, as in the
// tile sweeps, x_j - x_i as the exact difference of the hi parts plus that of the
// lo parts.
// 2-D: a particle's tile2, which serves every pair inside one tile; for a pair
// across tiles (a flagged entry, 1 in 5 to 10) j's position is split in i's tile.
template <int DIM>
struct Rec;
template <>
struct Rec<2> {
    float4 t;    // tile2, or (flagged) the 16 bytes of the FP64 x and y: one load either way
    bool cross;
    __device__ __forceinline__ void load(const BatchDev& b, unsigned e) {
        const int j = (int)(e & ~kEntryCross);
        cross = (e & kEntryCross) != 0u;
        t = __ldg(cross ? reinterpret_cast<const float4*>(b.pos + j) : b.tile2 + j);
    }
    // the position in the tile of ti with origin (ox, oy)
    __device__ __forceinline__ float4 in_tile(const BScene& sc, double ox, double oy, const float4& ti) const {
        if (!cross) return t;
        const double x = __hiloint2double(__float_as_int(t.y), __float_as_int(t.x));
        const double y = __hiloint2double(__float_as_int(t.w), __float_as_int(t.z));
        double d[2] = {x - ox, y - oy}, hq;
        const double c[2] = {(double)ti.x, (double)ti.y};
        float hi[2], lo[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            if (d[k] - c[k] > sc.half_width[k]) d[k] -= sc.width[k];
            else if (d[k] - c[k] < -sc.half_width[k]) d[k] += sc.width[k];
            tile_split(sc, d[k], hq, lo[k]);
            hi[k] = (float)(hq * sc.rgrid);
        }
        return make_float4(hi[0], hi[1], lo[0], lo[1]);
    }
};
// 3-D: FP64 positions; a tile of the default shape holds so few cells that most
// pairs cross one.
template <>
struct Rec<3> {
    double x[3], t;
    __device__ __forceinline__ void load(const BatchDev& b, unsigned j) {
        asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
            : "=d"(x[0]), "=d"(x[1]), "=d"(x[2]), "=d"(t)
            : "l"(b.pos + j));
    }
};

template <int DIM>
struct Frame;
template <>
struct Frame<2> {
    float4 t;       // tile2
    double ox, oy;  // the tile's origin
    __device__ __forceinline__ void set(const BatchDev& b, const BScene& sc, int i) {
        t = __ldg(b.tile2 + i);
        const int h = b.home[i];
        ox = tile_origin(sc, 0, h & 1023);
        oy = tile_origin(sc, 1, (h >> 10) & 1023);
    }
    __device__ __forceinline__ void disp32(const BScene& sc, const Rec<2>& r, float* d) const {
        const float4 j = r.in_tile(sc, ox, oy, t);
        d[0] = (j.x - t.x) + (j.z - t.z);
        d[1] = (j.y - t.y) + (j.w - t.w);
        d[2] = 0.0f;
    }
    __device__ __forceinline__ void disp_tile(const BScene& sc, const Rec<2>& r, float* d) const { disp32(sc, r, d); }
    __device__ __forceinline__ void disp64(const BScene& sc, const Rec<2>& r, double* d) const {
        const float4 j = r.in_tile(sc, ox, oy, t);
        d[0] = (double)(j.x - t.x) + ((double)j.z - (double)t.z);
        d[1] = (double)(j.y - t.y) + ((double)j.w - (double)t.w);
        d[2] = 0.0;
    }
};
template <>
struct Frame<3> {
    double x[3], o[3], q[3];  // position (the image nearest the home cell), tile origin, hi part in grid steps
    float l[3];               // lo part
    __device__ __forceinline__ void set(const BatchDev& b, const BScene& sc, int i) {
        Rec<3> p;
        p.load(b, (unsigned)i);
        const int h = b.home[i];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int c = (h >> (10 * k)) & 1023;
            o[k] = tile_origin(sc, k, c);
            const double ec = ((double)(c - c / sc.ttile[k] * sc.ttile[k] + 1) + 0.5) * sc.cell_width[k];
            double d = p.x[k] - o[k];
            const double r = rint((d - ec) * sc.inv_width[k]);  // 0, or +-1 across a periodic face
            d -= sc.width[k] * r;
            x[k] = p.x[k] - sc.width[k] * r;
            tile_split(sc, d, q[k], l[k]);
        }
    }
    // minimum image (no listed pair is near half a domain apart, so the high words
    // decide); one branch for a pair that crosses no face
    __device__ __forceinline__ void disp64(const BScene& sc, const Rec<3>& r, double* d) const {
        bool far = false;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            d[k] = r.x[k] - x[k];
            far |= (__double2hiint(d[k]) & 0x7fffffff) >= sc.hw_hi[k];
        }
        if (far) {
#pragma unroll
            for (int k = 0; k < 3; ++k)
                if ((__double2hiint(d[k]) & 0x7fffffff) >= sc.hw_hi[k]) d[k] += d[k] < 0.0 ? sc.width[k] : -sc.width[k];
        }
    }
    __device__ __forceinline__ void disp32(const BScene& sc, const Rec<3>& r, float* d) const {
        double e[3];
        disp64(sc, r, e);
#pragma unroll
        for (int k = 0; k < 3; ++k) d[k] = (float)e[k];
    }
    __device__ __forceinline__ void disp_tile(const BScene& sc, const Rec<3>& r, float* d) const {
        double e[3];
        disp64(sc, r, e);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const double raw = r.x[k] - x[k];
            double t = r.x[k] - o[k], hq;
            float lo;
            if (raw != e[k]) t += raw < 0.0 ? sc.width[k] : -sc.width[k];
            tile_split(sc, t, hq, lo);
            d[k] = (float)((hq - q[k]) * sc.rgrid) + (lo - l[k]);
        }
    }
};

// Visits the entries of slot i's list in order: visit(load(entry)), rows of four
// entries loaded one row ahead and records one entry ahead.  A list that outgrew
// its table is walked from the cells instead: every other particle of the 3^D
// cells around the home cell in the order the table is built in (the pairs beyond
// the cut-offs add nothing).
template <int DIM, class Load, class Visit>
__device__ __forceinline__ void walk_table(const BatchDev& b, const BScene& sc, const uint4* __restrict__ tab, int cnt,
                                           int cap, int i, Load&& load, Visit&& visit) {
    if (cnt > cap) {
        const int h = b.home[i];
        const int ix = h & 1023, iy = (h >> 10) & 1023, iz = (h >> 20) & 1023;
        for (int q = 0; q < (DIM == 3 ? 27 : 9); ++q) {
            const int ax = DIM == 3 ? q / 9 : q / 3, ay = DIM == 3 ? (q / 3) % 3 : q % 3, az = DIM == 3 ? q % 3 : 1;
            const int k = sc.cbase +
                          (wrapi(ix + ax - 1, sc.cc[0]) * sc.cc[1] + wrapi(iy + ay - 1, sc.cc[1])) * sc.cc[2] +
                          (DIM == 3 ? wrapi(iz + az - 1, sc.cc[2]) : 0);
            for (int j = b.start[k]; j < b.start[k + 1]; ++j)
                if (j != i) visit(load((unsigned)j | (DIM == 2 ? kEntryCross : 0u)));
        }
        return;
    }
    if (cnt <= 0) return;
    const size_t n = (size_t)b.n;
    const uint4* row = tab + i;
    uint4 q = __ldg(row);
    auto r0 = load(q.x);
    for (int k = 0;; k += 4) {
        uint4 qn = q;
        row += n;
        if (k + 4 < cnt) qn = __ldg(row);
        auto r1 = load(k + 1 < cnt ? q.y : q.x);  // past the end: a record again, not visited
        visit(r0);
        if (k + 1 >= cnt) break;
        r0 = load(k + 2 < cnt ? q.z : q.x);
        visit(r1);
        if (k + 2 >= cnt) break;
        r1 = load(k + 3 < cnt ? q.w : q.x);
        visit(r0);
        if (k + 3 >= cnt) break;
        r0 = load(qn.x);
        visit(r1);
        if (k + 4 >= cnt) break;
        q = qn;
    }
}

// Resident 128-thread blocks per SM the table sweeps are compiled for.  Their
// gathers' latency and the instruction count bound them (L1 data pipe 41-59 %,
// issue 51-55 %).  64 droplets (371,729 particles): sweep A 96 us at 7 blocks, 110 at
// 6, 107 at 10; sweep B 142 us at 5, 148 at 6, 161 at 8 (tile sweeps: 145 and 189).  24
// dam breaks (391,426 particles, 75,970 fluid): 38 and 127 us (tile sweeps: 563 and 969,
// whose 96-cell halos hold six times the tile and mostly had to be split).
constexpr int kTabMinA = 7, kTabMinB = 5;

// Sweep A: the tile sweep's sums over the table, the FP64 density pairs over
// the short list, the surface-tension sums over the whole one.
template <int DIM, bool ST>
__global__ void __launch_bounds__(128, kTabMinA) k_bt_a(BatchDev b) {
    __shared__ BScene sc;
    const int2 it = b.items_a[blockIdx.x];
    if (blockIdx.x == 0) {  // the sorts of this step are done: clear the requests
        for (int s = threadIdx.x; s < b.S; s += blockDim.x)
            if (b.flags[s]) {
                atomicAdd(&b.ctl[6], 1);
                b.flags[s] = 0;
            }
        if (threadIdx.x == 0) b.ctl[0] = 0;
    }
    load_scene(b, it.x, sc);
    const int i = it.y + threadIdx.x;
    if (i >= sc.pbase + sc.n) return;
    Frame<DIM> f;
    f.set(b, sc, i);
    const float4 vi = b.v32[i];
    const int ti = __float_as_int(vi.w);
    double spd = 0.0, sdd = 0.0;  // DensityP, DivergenceP: FP64 pairs
    struct RV {
        Rec<DIM> p;
        float4 v;
    };
    walk_table<DIM>(b, sc, b.tab_s, b.tcnt_s[i], b.tcap_s, i,
                    [&](unsigned e) {
                        RV r;
                        r.p.load(b, e);
                        r.v = __ldg(b.v32 + (DIM == 2 ? e & ~kEntryCross : e));
                        return r;
                    },
                    [&](const RV& rj) {
        double dd[3];
        f.disp64(sc, rj.p, dd);
        const double r2d = dd[0] * dd[0] + dd[1] * dd[1] + dd[2] * dd[2];
        if (!(r2d <= sc.rp2_d)) return;
        const double y = rsqrt_dnr(r2d);
        const double q = 1.0 - r2d * y * sc.inv_rp_d;
        spd += sc.cp_d * q * q;  // wp
        const double dw = sc.cp_m2_d * q;
        double ue = ((double)rj.v.x - (double)vi.x) * dd[0] + ((double)rj.v.y - (double)vi.y) * dd[1];
        if (DIM == 3) ue += ((double)rj.v.z - (double)vi.z) * dd[2];
        sdd -= ue * y * dw;
    });
    float sa = 0.f, cak = 0.f, g0 = 0.f, g1 = 0.f, g2 = 0.f;
    const bool st = ST && sc.has_st;
    if (st) {
        const bool ratio1 = sc.ratio_all_one;
        struct RT {
            Rec<DIM> p;
            int t;
        };
        walk_table<DIM>(b, sc, b.tab, b.tcnt[i], b.tcap, i,
                        [&](unsigned e) {
                            RT r;
                            r.p.load(b, e);
                            r.t = ratio1 ? 0 : __float_as_int(__ldg(&b.v32[DIM == 2 ? e & ~kEntryCross : e].w));
                            return r;
                        },
                        [&](const RT& rj) {
            float d[3];
            f.disp_tile(sc, rj.p, d);
            const float r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
            if (!(r2 < sc.cut2_a)) return;
            const float rr = r2 * rsqrt_nr(r2);
            if (ratio1) st_density<false>(sc, ti, rj.t, r2, rr, d[0], d[1], d[2], sa, cak, g0, g1, g2);
            else st_density<true>(sc, ti, rj.t, r2, rr, d[0], d[1], d[2], sa, cak, g0, g1, g2);
        });
    }
    const double strain = spd - sc.n0p_d;
    double kappa = sc.bulk_modulus_d[ti];
    if (strain < 0.0) kappa = 0.0;
    const double pp = -sc.bulk_viscosity_d[ti] * sdd + kappa * strain;
    if (ST) {
        float pa = 0.0f;
        if (st) {
            const float dens = sa - cak;
            pa = sc.cof_a[ti] * (dens - sc.n0a) / sc.l0;
            if (sc.n0a <= dens) pa = 0.0f;
        }
        b.gc[i] = make_float4(g0, g1, g2, pa);
    }
    b.vp[i] = DIM == 2 ? make_float4(vi.x, vi.y, (float)pp, vi.w) : make_float4(vi.x, vi.y, vi.z, (float)pp);
}

// Sweep B: the tile sweep's force sums, fluid particles only.  2-D: one walk of the
// whole list.  3-D: two walks, the pairs within RadiusP + MARGIN with their tile
// displacement (Kahan sums; all of them are in the short list, which reaches a
// margin further at the sort), then the rest with the FP64 displacement rounded
// once (plain sums); both walks tell the two apart by the same rounded distance.
template <int DIM, bool ST>
__global__ void __launch_bounds__(128, kTabMinB) k_bt_b(BatchDev b) {
    __shared__ BScene sc;
    const int2 it = b.items_b[blockIdx.x];
    load_scene(b, it.x, sc);
    const int k = it.y + threadIdx.x;
    if (k >= sc.fbase + sc.nfl) return;
    const int i = b.flist[k];
    Frame<DIM> f;
    f.set(b, sc, i);
    const float4 vi = __ldg(b.vp + i);
    const int ti = DIM == 2 ? __float_as_int(vi.w) : __float_as_int(b.v32[i].w);
    const bool st = ST && sc.has_st;
    const bool ratio1 = sc.ratio_all_one;
    const float Pi = DIM == 2 ? vi.z : vi.w;
    const float4 gi = st ? __ldg(b.gc + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    const float ai = sc.a_k[ti];
    const float mu_u = sc.visc_mu[ti][ti];
    struct RB {
        Rec<DIM> p;
        float4 v, g;
    };
    auto load = [&](unsigned e) {
        const int j = (int)(DIM == 2 ? e & ~kEntryCross : e);
        RB r;
        r.p.load(b, e);
        r.v = __ldg(b.vp + j);
        if (ST) r.g = __ldg(b.gc + j);
        return r;
    };
    // a pair's terms: radial part s, tangential part t
    auto terms = [&](const RB& rj, const float* d, float r2, float& s, float3& t) {
        const float rinv = rsqrt_nr(r2);
        const float rr = r2 * rinv;
        int tj;
        if constexpr (DIM == 2) tj = __float_as_int(rj.v.w);
        else tj = (int)rj.p.t;
        if (r2 < sc.rp2) s += (Pi + (DIM == 2 ? rj.v.z : rj.v.w)) * fmaf(sc.p_b, rr, sc.p_a) * rinv;
        if (r2 < sc.rv2) {
            const float mu = sc.uniform_mu ? mu_u : sc.visc_mu[ti][tj];
            float ud = (rj.v.x - vi.x) * d[0] + (rj.v.y - vi.y) * d[1];
            if (DIM == 3) ud += (rj.v.z - vi.z) * d[2];
            s += mu * ud * fmaf(sc.v_b, rr, sc.v_a) * (rinv * rinv * rinv);
        }
        if (ST && st) {
            if (ratio1) s += st_terms<false, DIM>(sc, ti, tj, r2, rr, rinv, d[0], d[1], d[2], gi, rj.g, ai, t);
            else s += st_terms<true, DIM>(sc, ti, tj, r2, rr, rinv, d[0], d[1], d[2], gi, rj.g, ai, t);
        }
    };
    float fx = 0.f, fy = 0.f, fz = 0.f, cx = 0.f, cy = 0.f, cz = 0.f;  // short range, Kahan
    float gx = 0.f, gy = 0.f, gz = 0.f;                                // long range
    auto add_short = [&](float s, const float* d, const float3& t) {
        kahan_add(fx, cx, fmaf(s, d[0], t.x));
        kahan_add(fy, cy, fmaf(s, d[1], t.y));
        if (DIM == 3) kahan_add(fz, cz, fmaf(s, d[2], t.z));
    };
    auto add_long = [&](float s, const float* d, const float3& t) {
        gx += fmaf(s, d[0], t.x);
        gy += fmaf(s, d[1], t.y);
        if (DIM == 3) gz += fmaf(s, d[2], t.z);
    };
    if (DIM == 3) {
        walk_table<DIM>(b, sc, b.tab_s, b.tcnt_s[i], b.tcap_s, i, load, [&](const RB& rj) {
            float d[3];
            f.disp32(sc, rj.p, d);
            if (!(d[0] * d[0] + d[1] * d[1] + d[2] * d[2] < sc.short_r2)) return;
            f.disp_tile(sc, rj.p, d);
            const float r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
            if (!(r2 < sc.cut2_b)) return;
            float s = 0.0f;
            float3 t = make_float3(0.f, 0.f, 0.f);
            terms(rj, d, r2, s, t);
            add_short(s, d, t);
        });
    }
    walk_table<DIM>(b, sc, b.tab, b.tcnt[i], b.tcap, i, load, [&](const RB& rj) {
        float d[3];
        f.disp32(sc, rj.p, d);
        const float r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
        if (!(r2 < sc.cut2_b) || (DIM == 3 && r2 < sc.short_r2)) return;
        float s = 0.0f;
        float3 t = make_float3(0.f, 0.f, 0.f);
        terms(rj, d, r2, s, t);
        if (DIM == 2 && r2 < sc.short_r2) add_short(s, d, t);
        else add_long(s, d, t);
    });
    double F0 = ((double)fx - (double)cx) + (double)gx;
    double F1 = ((double)fy - (double)cy) + (double)gy;
    double F2 = ((double)fz - (double)cz) + (double)gz;
    const double mass = sc.density[ti] * sc.vol_d;
    F0 += mass * sc.gravity[0];
    F1 += mass * sc.gravity[1];
    F2 += mass * sc.gravity[2];
    double4 v = b.vel[i];
    v.x += F0 / mass * sc.dt;
    v.y += F1 / mass * sc.dt;
    v.z += F2 / mass * sc.dt;
    if (!(isfinite(v.x) && isfinite(v.y) && isfinite(v.z))) atomicOr(&b.ctl[1], BERR_NONFINITE);
    b.vel[i] = v;
}

// Positions and velocities of every scene in its input order, packed.
__global__ void __launch_bounds__(256) k_bt_state(BatchDev b, double* __restrict__ xyz, double* __restrict__ vel) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= b.n) return;
    const size_t o = 3 * ((size_t)b.scenes[b.sid[p]].pbase + b.pidx[p]);
    const double4 x = b.pos[p], v = b.vel[p];
    xyz[o] = x.x;
    xyz[o + 1] = x.y;
    xyz[o + 2] = x.z;
    vel[o] = v.x;
    vel[o + 1] = v.y;
    vel[o + 2] = v.z;
}

// ---- the tile sweeps -----------------------------------------------------------

template <int DIM, int SWEEP, bool ST>
struct Smem {
    // staged per particle: P (2-D hi.xy lo.xy; 3-D hi.xyz type), L (3-D lo.xyz),
    // V (sweep A: velocity; sweep B: vp), G (sweep B with surface tension: gc)
    static constexpr int kL = DIM == 3 ? 1 : 0;
    static constexpr int kG = (SWEEP == 1 && ST) ? 1 : 0;
    static constexpr int kVec = 2 + kL + kG;
    static size_t bytes(int cap, int hmax, int ncol) {
        return (size_t)cap * 16 * kVec + (size_t)(2 * hmax + 1 + ncol + 1) * 4 + (size_t)cap * 2 + 16;
    }
};

template <int DIM, int SWEEP, bool ST>
__global__ void __launch_bounds__(kMaxThreads) k_bt_sweep(BatchDev b) {
    using SM = Smem<DIM, SWEEP, ST>;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ BScene sc;
    __shared__ int4 stack[kStack];
    __shared__ int s_item, s_sp;
    const int cap = b.cap, tid = threadIdx.x, bd = blockDim.x, lane = tid & 31, warp = tid >> 5;
    float4* sP = reinterpret_cast<float4*>(smem);
    float4* sL = sP + cap;
    float4* sV = sL + (size_t)cap * SM::kL;
    float4* sG = sV + cap;
    int* hb = reinterpret_cast<int*>(sG + (size_t)cap * SM::kG);  // [hmax + 1] staged begin of each halo cell
    int* hsrc = hb + b.hmax + 1;                                   // [hmax] first slot of each halo cell
    int* col = hsrc + b.hmax;                                      // [ncol + 1] interior prefix per column
    unsigned short* sH = reinterpret_cast<unsigned short*>(col + b.ncol + 1);
    int* qhead = b.ctl + (SWEEP == 0 ? 2 : 4);

    if (SWEEP == 0 && blockIdx.x == 0) {  // the sorts of this step are done: clear the requests
        for (int s = tid; s < b.S; s += bd)
            if (b.flags[s]) {
                atomicAdd(&b.ctl[6], 1);
                b.flags[s] = 0;
            }
        if (tid == 0) b.ctl[0] = 0;
    }
    int cur = -1;
    for (;;) {
        __syncthreads();
        if (tid == 0) s_item = atomicAdd(qhead, 1);
        __syncthreads();
        const int item = s_item;
        if (item >= b.n_items) break;
        const int4 it = b.items[item];
        if (it.x != cur) {
            const int4* src = reinterpret_cast<const int4*>(b.scenes + it.x);
            int4* dst = reinterpret_cast<int4*>(&sc);
            for (int k = tid; k < (int)(sizeof(BScene) / 16); k += bd) dst[k] = src[k];
            cur = it.x;
            __syncthreads();
        }
        if (tid == 0) {
            const int t0 = min(sc.tile[0], sc.cc[0] - it.y), t1 = min(sc.tile[1], sc.cc[1] - it.z);
            const int t2 = DIM == 3 ? min(sc.tile[2], sc.cc[2] - it.w) : 1;
            stack[0] = make_int4(it.y, it.z, it.w, t0 | (t1 << 8) | (t2 << 16));
            s_sp = 1;
        }
        for (;;) {
            __syncthreads();
            if (s_sp == 0) break;
            const int4 e = stack[s_sp - 1];
            __syncthreads();
            if (tid == 0) --s_sp;
            const int x0 = e.x, y0 = e.y, z0 = e.z;
            const int t0 = e.w & 255, t1 = (e.w >> 8) & 255, t2 = (e.w >> 16) & 255;
            const int H1 = t1 + 2, H2 = DIM == 3 ? t2 + 2 : 1, H = (t0 + 2) * H1 * H2;
            // halo cells: first slot and count
            for (int h = tid; h < H; h += bd) {
                const int a = h / (H1 * H2), bb = (h / H2) % H1, cz = h % H2;
                const int cx = wrapi(x0 - 1 + a, sc.cc[0]), cy = wrapi(y0 - 1 + bb, sc.cc[1]);
                const int czz = DIM == 3 ? wrapi(z0 - 1 + cz, sc.cc[2]) : 0;
                const int key = sc.cbase + (cx * sc.cc[1] + cy) * sc.cc[2] + czz;
                const int s0 = b.start[key];
                hsrc[h] = s0;
                hb[h] = b.start[key + 1] - s0;
            }
            __syncthreads();
            if (warp == 0) {  // exclusive scan of the counts, hb[H] = total
                int run = 0;
                for (int base = 0; base < H; base += 32) {
                    const int v = base + lane < H ? hb[base + lane] : 0;
                    int x = v;
                    for (int o = 1; o < 32; o <<= 1) {
                        const int y = __shfl_up_sync(0xffffffffu, x, o);
                        if (lane >= o) x += y;
                    }
                    if (base + lane < H) hb[base + lane] = run + x - v;
                    run += __shfl_sync(0xffffffffu, x, 31);
                }
                if (lane == 0) hb[H] = run;
            }
            __syncthreads();
            const int total = hb[H];
            if (total > cap) {  // split the tile along its longest axis
                if (tid == 0) {
                    const int ax = (DIM == 3 && t2 >= t0 && t2 >= t1) ? 2 : (t1 > t0 ? 1 : 0);
                    const int len = ax == 0 ? t0 : ax == 1 ? t1 : t2;
                    if (len <= 1 || s_sp + 2 > kStack) {
                        atomicOr(&b.ctl[1], BERR_CAPACITY);
                    } else {
                        const int h0 = len / 2, h1 = len - h0;
                        int4 lo = e, hi = e;
                        const int sh = 8 * ax;
                        lo.w = (e.w & ~(255 << sh)) | (h0 << sh);
                        hi.w = (e.w & ~(255 << sh)) | (h1 << sh);
                        if (ax == 0) hi.x += h0;
                        else if (ax == 1) hi.y += h0;
                        else hi.z += h0;
                        stack[s_sp] = lo;
                        stack[s_sp + 1] = hi;
                        s_sp += 2;
                        atomicAdd(&b.ctl[7], 1);
                    }
                }
                continue;
            }
            if (total == 0) continue;
            // interior columns: (a in 1..t0) in 2-D, (a, b) in 1..t0 x 1..t1 in 3-D
            const int ncol = DIM == 3 ? t0 * t1 : t0;
            auto col_begin = [&](int k, int& lo, int& hi) {
                const int a = DIM == 3 ? 1 + k / t1 : 1 + k, bb = DIM == 3 ? 1 + k % t1 : 1;
                if (DIM == 3) {
                    const int base = (a * H1 + bb) * H2;
                    lo = hb[base + 1];
                    hi = hb[base + t2 + 1];
                } else {
                    lo = hb[a * H1 + 1];
                    hi = hb[a * H1 + t1 + 1];
                }
            };
            if (warp == 0) {
                int run = 0;
                for (int base = 0; base < ncol; base += 32) {
                    int v = 0;
                    if (base + lane < ncol) {
                        int lo, hi;
                        col_begin(base + lane, lo, hi);
                        v = hi - lo;
                    }
                    int x = v;
                    for (int o = 1; o < 32; o <<= 1) {
                        const int y = __shfl_up_sync(0xffffffffu, x, o);
                        if (lane >= o) x += y;
                    }
                    if (base + lane < ncol) col[base + lane] = run + x - v;
                    run += __shfl_sync(0xffffffffu, x, 31);
                }
                if (lane == 0) col[ncol] = run;
            }
            // stage every halo particle: tile-relative hi/lo coordinates
            const double ox = sc.dmin[0] + (double)(x0 - 1) * sc.cell_width[0];
            const double oy = sc.dmin[1] + (double)(y0 - 1) * sc.cell_width[1];
            const double oz = sc.dmin[2] + (double)(z0 - 1) * sc.cell_width[2];
            for (int q = tid; q < total; q += bd) {
                int lo = 0, hi = H;  // largest h with hb[h] <= q (skips empty cells)
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (hb[mid] <= q) lo = mid;
                    else hi = mid - 1;
                }
                const int h = lo;
                const int g = hsrc[h] + (q - hb[h]);
                const int a = h / (H1 * H2), bb = (h / H2) % H1, cz = h % H2;
                const double4 p = b.pos[g];
                double d[3] = {p.x - ox, p.y - oy, p.z - oz};
                const int hc[3] = {a, bb, cz};
                float fh[3], fl[3];
#pragma unroll
                for (int k = 0; k < DIM; ++k) {
                    const double ec = ((double)hc[k] + 0.5) * sc.cell_width[k];
                    d[k] -= sc.width[k] * rint((d[k] - ec) * sc.inv_width[k]);
                    const double qh = rint(d[k] * sc.inv_grid) * sc.grid;
                    fh[k] = (float)qh;
                    fl[k] = (float)(d[k] - qh);
                }
                const int type = (int)p.w;
                if (DIM == 2) {
                    sP[q] = make_float4(fh[0], fh[1], fl[0], fl[1]);
                } else {
                    sP[q] = make_float4(fh[0], fh[1], fh[2], __int_as_float(type));
                    sL[q] = make_float4(fl[0], fl[1], fl[2], 0.0f);
                }
                if (SWEEP == 0) {
                    const double4 v = b.vel[g];
                    sV[q] = DIM == 2 ? make_float4((float)v.x, (float)v.y, 0.0f, __int_as_float(type))
                                     : make_float4((float)v.x, (float)v.y, (float)v.z, 0.0f);
                } else {
                    sV[q] = b.vp[g];
                    if (ST) sG[q] = b.gc[g];
                }
                sH[q] = (unsigned short)h;
            }
            __syncthreads();
            const int nin = col[ncol];
            for (int k = tid; k < nin; k += bd) {
                int lo = 0, hi = ncol;  // column of interior particle k
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (col[mid] <= k) lo = mid;
                    else hi = mid - 1;
                }
                int cb, ce;
                col_begin(lo, cb, ce);
                const int si = cb + (k - col[lo]);
                const int h = sH[si];
                const int a = h / (H1 * H2), bb = (h / H2) % H1, cz = h % H2;
                const int g = hsrc[h] + (si - hb[h]);
                const float4 pi = sP[si];
                float4 li = make_float4(0.f, 0.f, 0.f, 0.f);
                if (DIM == 3) li = sL[si];
                const float4 vi = sV[si];
                const int ti = DIM == 2 ? __float_as_int(vi.w) : __float_as_int(pi.w);
                if (SWEEP == 1 && ti >= 2) continue;  // walls never accelerate
                // runs of three cells along the last axis: 3 in 2-D, 9 in 3-D
                auto run_of = [&](int r, int& rb, int& re) {
                    if (DIM == 2) {
                        const int base = (a + r - 1) * H1 + bb;
                        rb = hb[base - 1];
                        re = hb[base + 2];
                    } else {
                        const int base = ((a + r / 3 - 1) * H1 + (bb + r % 3 - 1)) * H2 + cz;
                        rb = hb[base - 1];
                        re = hb[base + 2];
                    }
                };
                auto disp = [&](int j, float& dx, float& dy, float& dz) {
                    const float4 pj = sP[j];
                    if (DIM == 2) {
                        dx = (pj.x - pi.x) + (pj.z - pi.z);
                        dy = (pj.y - pi.y) + (pj.w - pi.w);
                        dz = 0.0f;
                    } else {
                        const float4 lj = sL[j];
                        dx = (pj.x - pi.x) + (lj.x - li.x);
                        dy = (pj.y - pi.y) + (lj.y - li.y);
                        dz = (pj.z - pi.z) + (lj.z - li.z);
                    }
                };
                auto type_of = [&](int j) {
                    return DIM == 2 ? __float_as_int(sV[j].w) : __float_as_int(sP[j].w);
                };
                const bool st = ST && sc.has_st;
                const bool ratio1 = sc.ratio_all_one;
                // Pairs within sqrt(cut2) in the runs' order: each chunk of up to 64
                // candidates is filtered into a bit mask first, then only the set
                // bits are visited, so the lanes of a warp run the pair terms
                // together instead of under divergent distance tests.
                auto for_near = [&](float cut2, auto&& visit) {
                    for (int r = 0; r < (DIM == 2 ? 3 : 9); ++r) {
                        int rb, re;
                        run_of(r, rb, re);
                        for (int base = rb; base < re; base += 64) {
                            const int cnt = min(64, re - base);
                            unsigned long long m = 0ull;
                            for (int q = 0; q < cnt; ++q) {
                                float dx, dy, dz;
                                disp(base + q, dx, dy, dz);
                                if (dx * dx + dy * dy + dz * dz < cut2) m |= 1ull << q;
                            }
                            if (si >= base && si < base + cnt) m &= ~(1ull << (si - base));
                            while (m != 0ull) {
                                const int j = base + __ffsll((long long)m) - 1;
                                m &= m - 1ull;
                                float dx, dy, dz;
                                disp(j, dx, dy, dz);
                                visit(j, dx, dy, dz, dx * dx + dy * dy + dz * dz);
                            }
                        }
                    }
                };
                if (SWEEP == 0) {
                    double spd = 0.0, sdd = 0.0;  // DensityP, DivergenceP: FP64 pairs
                    float sa = 0.f, cak = 0.f, g0 = 0.f, g1 = 0.f, g2 = 0.f;
                    for_near(sc.cut2_a, [&](int j, float dx, float dy, float dz, float r2) {
                            const float rinv = rsqrt_nr(r2);
                            const float rr = r2 * rinv;
                            if (r2 <= sc.rp2_pre) {
                                // FP64 displacement: the hi parts' difference is exact in FP32,
                                // the lo parts carry the rest
                                const float4 pj = sP[j];
                                double dd[3];
                                if (DIM == 2) {
                                    dd[0] = (double)(pj.x - pi.x) + ((double)pj.z - (double)pi.z);
                                    dd[1] = (double)(pj.y - pi.y) + ((double)pj.w - (double)pi.w);
                                    dd[2] = 0.0;
                                } else {
                                    const float4 lj = sL[j];
                                    dd[0] = (double)(pj.x - pi.x) + ((double)lj.x - (double)li.x);
                                    dd[1] = (double)(pj.y - pi.y) + ((double)lj.y - (double)li.y);
                                    dd[2] = (double)(pj.z - pi.z) + ((double)lj.z - (double)li.z);
                                }
                                const double r2d = dd[0] * dd[0] + dd[1] * dd[1] + dd[2] * dd[2];
                                if (r2d <= sc.rp2_d) {
                                    const double y = rsqrt_dnr(r2d);
                                    const double q = 1.0 - r2d * y * sc.inv_rp_d;
                                    spd += sc.cp_d * q * q;  // wp
                                    const double dw = sc.cp_m2_d * q;
                                    const float4 vj = sV[j];
                                    double ue = ((double)vj.x - (double)vi.x) * dd[0] +
                                                ((double)vj.y - (double)vi.y) * dd[1];
                                    if (DIM == 3) ue += ((double)vj.z - (double)vi.z) * dd[2];
                                    sdd -= ue * y * dw;
                                }
                            }
                            if (ST && st) {
                                const int tj = type_of(j);
                                if (ratio1) st_density<false>(sc, ti, tj, r2, rr, dx, dy, dz, sa, cak, g0, g1, g2);
                                else st_density<true>(sc, ti, tj, r2, rr, dx, dy, dz, sa, cak, g0, g1, g2);
                            }
                    });
                    const double strain = spd - sc.n0p_d;
                    const double div = sdd;
                    double kappa = sc.bulk_modulus_d[ti];
                    if (strain < 0.0) kappa = 0.0;
                    const double pp = -sc.bulk_viscosity_d[ti] * div + kappa * strain;
                    if (ST) {
                        float pa = 0.0f;
                        if (st) {
                            const float dens = sa - cak;
                            pa = sc.cof_a[ti] * (dens - sc.n0a) / sc.l0;
                            if (sc.n0a <= dens) pa = 0.0f;
                        }
                        b.gc[g] = make_float4(g0, g1, g2, pa);
                    }
                    b.vp[g] = DIM == 2 ? make_float4(vi.x, vi.y, (float)pp, vi.w)
                                       : make_float4(vi.x, vi.y, vi.z, (float)pp);
                } else {
                    const float Pi = DIM == 2 ? vi.z : vi.w;
                    float4 gi = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (ST) gi = sG[si];
                    const float ai = sc.a_k[ti];
                    const float mu_u = sc.visc_mu[ti][ti];
                    float fx = 0.f, fy = 0.f, fz = 0.f, cx = 0.f, cy = 0.f, cz2 = 0.f;  // short range, Kahan
                    float gx = 0.f, gy = 0.f, gz = 0.f;                                  // long range
                    for_near(sc.cut2_b, [&](int j, float dx, float dy, float dz, float r2) {
                            const float rinv = rsqrt_nr(r2);
                            const float rr = r2 * rinv;
                            const float4 vj = sV[j];
                            const float Pj = DIM == 2 ? vj.z : vj.w;
                            const int tj = (sc.uniform_mu && ratio1 && !st) ? ti : type_of(j);
                            float s = 0.0f;
                            if (r2 < sc.rp2) s += (Pi + Pj) * fmaf(sc.p_b, rr, sc.p_a) * rinv;
                            if (r2 < sc.rv2) {
                                const float mu = sc.uniform_mu ? mu_u : sc.visc_mu[ti][tj];
                                float ud = (vj.x - vi.x) * dx + (vj.y - vi.y) * dy;
                                if (DIM == 3) ud += (vj.z - vi.z) * dz;
                                s += mu * ud * fmaf(sc.v_b, rr, sc.v_a) * (rinv * rinv * rinv);
                            }
                            float3 t = make_float3(0.f, 0.f, 0.f);
                            if (ST && st) {
                                if (ratio1) s += st_terms<false>(sc, ti, tj, r2, rr, rinv, dx, dy, dz, gi, sG[j], ai, t);
                                else s += st_terms<true>(sc, ti, tj, r2, rr, rinv, dx, dy, dz, gi, sG[j], ai, t);
                            }
                            if (r2 < sc.short_r2) {
                                kahan_add(fx, cx, fmaf(s, dx, t.x));
                                kahan_add(fy, cy, fmaf(s, dy, t.y));
                                if (DIM == 3) kahan_add(fz, cz2, fmaf(s, dz, t.z));
                            } else {
                                gx += fmaf(s, dx, t.x);
                                gy += fmaf(s, dy, t.y);
                                if (DIM == 3) gz += fmaf(s, dz, t.z);
                            }
                    });
                    double F0 = ((double)fx - (double)cx) + (double)gx;
                    double F1 = ((double)fy - (double)cy) + (double)gy;
                    double F2 = ((double)fz - (double)cz2) + (double)gz;
                    const double mass = sc.density[ti] * sc.vol_d;
                    F0 += mass * sc.gravity[0];
                    F1 += mass * sc.gravity[1];
                    F2 += mass * sc.gravity[2];
                    double4 v = b.vel[g];
                    v.x += F0 / mass * sc.dt;
                    v.y += F1 / mass * sc.dt;
                    v.z += F2 / mass * sc.dt;
                    if (!(isfinite(v.x) && isfinite(v.y) && isfinite(v.z))) atomicOr(&b.ctl[1], BERR_NONFINITE);
                    b.vel[g] = v;
                }
            }
        }
    }
    // every CTA has drawn past the end of the queue: the last one resets it
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        if (atomicAdd(qhead + 1, 1) == (int)gridDim.x - 1) {
            qhead[0] = 0;
            qhead[1] = 0;
            __threadfence();
        }
    }
}

inline int nblocks(long long n, int t) { return (int)((n + t - 1) / t); }

using SweepFn = void (*)(BatchDev);

template <int DIM>
SweepFn sweep_fn(int sweep, bool st) {
    if (sweep == 0) return st ? k_bt_sweep<DIM, 0, true> : k_bt_sweep<DIM, 0, false>;
    return st ? k_bt_sweep<DIM, 1, true> : k_bt_sweep<DIM, 1, false>;
}

size_t sweep_smem(int dim, int sweep, bool st, int cap, int hmax, int ncol) {
    if (dim == 2) {
        if (sweep == 0) return st ? Smem<2, 0, true>::bytes(cap, hmax, ncol) : Smem<2, 0, false>::bytes(cap, hmax, ncol);
        return st ? Smem<2, 1, true>::bytes(cap, hmax, ncol) : Smem<2, 1, false>::bytes(cap, hmax, ncol);
    }
    if (sweep == 0) return st ? Smem<3, 0, true>::bytes(cap, hmax, ncol) : Smem<3, 0, false>::bytes(cap, hmax, ncol);
    return st ? Smem<3, 1, true>::bytes(cap, hmax, ncol) : Smem<3, 1, false>::bytes(cap, hmax, ncol);
}

}  // namespace
}  // namespace mph

using mph::BatchDev;
using mph::BScene;

// ---------------------------------------------------------------------------
// host side

struct BatchProfile {
    bool on = false;
    std::vector<std::string> names;
    std::vector<long long> launches;
    std::vector<double> ms;
    struct Pending {
        int id, count;
        cudaEvent_t a, b;
    };
    std::vector<Pending> pending;
};

struct mph_batch {
    int dim = 2, S = 0, n = 0, n_fluid = 0, cells = 0;
    int tile[3] = {8, 8, 1}, threads = 256, occ = 2;
    int cap = 0, hmax = 0, ncol = 0, n_items = 0, grid_a = 0, grid_b = 0, sms = 0;
    size_t smem_a = 0, smem_b = 0;
    bool has_st = false;
    std::vector<BScene> hs;
    std::vector<int> pbase;
    std::vector<std::vector<int>> cell_count;  // per scene: particles per cell at creation
    cudaStream_t stream = nullptr;
    BatchDev d{};
    BScene* d_scenes = nullptr;
    int4* d_items = nullptr;
    int* d_sid = nullptr;
    int2* d_items_t = nullptr;         // table form: sweep A's blocks, then sweep B's
    char* slab = nullptr;              // the arrays of d, d_scenes and d_sid
    int table_cta = 0;                 // block size its items are cut for
    bool table_ok = false;             // the table fits: allocated at creation
    bool sorted = false;               // the initial sort is done
    bool table_valid = false;          // the table holds the lists of the current sort
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    long long steps = 0, launches = 0;
    int* h_ctl = nullptr;  // pinned [8]
    BatchProfile prof;
    std::string err;
};

static thread_local std::string g_batch_err;

static int bfail(mph_batch* b, int code, const std::string& msg) {
    if (b) b->err = msg;
    g_batch_err = msg;
    return code;
}

#define BTRY(b, expr)                                                                        \
    do {                                                                                     \
        cudaError_t e_ = (expr);                                                             \
        if (e_ != cudaSuccess)                                                               \
            return bfail(b, MPH_ERR_CUDA, std::string(#expr ": ") + cudaGetErrorString(e_)); \
    } while (0)

// Device arrays that live as long as their batch, in one allocation (thirty of
// their own cost a batch 0.5 to 4 ms: 64 droplets 20-31 ms to create, now 19-21; 24 dam
// breaks 31, now 21-27).
class Slab {
public:
    template <class T>
    void want(T** p, size_t n) {
        list_.push_back({(void**)p, bytes_});
        bytes_ += ((n ? n : 1) * sizeof(T) + 255) / 256 * 256;
    }
    cudaError_t alloc(char** base) {
        const cudaError_t e = cudaMalloc((void**)base, bytes_);
        if (e == cudaSuccess)
            for (const auto& w : list_) *w.first = *base + w.second;
        return e;
    }

private:
    std::vector<std::pair<void**, size_t>> list_;
    size_t bytes_ = 0;
};

template <class T>
static cudaError_t balloc(T** p, size_t n) {
    *p = nullptr;
    return cudaMalloc((void**)p, (n ? n : 1) * sizeof(T));
}

static void free_graph(mph_batch* b) {
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->graph) cudaGraphDestroy(b->graph);
    b->exec = nullptr;
    b->graph = nullptr;
}

extern "C" void mph_batch_destroy(mph_batch* b) {
    if (!b) return;
    if (b->stream) cudaStreamSynchronize(b->stream);
    free_graph(b);
    void* ptrs[] = {b->d_items_t, b->d_items, b->slab};
    for (void* p : ptrs)
        if (p) cudaFree(p);
    for (auto& pe : b->prof.pending) {
        cudaEventDestroy(pe.a);
        cudaEventDestroy(pe.b);
    }
    if (b->h_ctl) cudaFreeHost(b->h_ctl);
    if (b->stream) cudaStreamDestroy(b->stream);
    delete b;
}

// The default tiles (cells per axis).
static constexpr int kTile2D[3] = {8, 8, 1}, kTile3D[3] = {2, 2, 4};

// Pair constants of one scene (the mixed form's, from the FP64 values).
static void fill_bscene(BScene& s, const mph::SimConst& c, const mph_constants& k) {
    std::memset(&s, 0, sizeof(s));
    s.n = c.n;
    s.tot = c.tot;
    for (int d = 0; d < 3; ++d) {
        s.cc[d] = c.cc[d];
        s.dmin[d] = c.dmin[d];
        s.width[d] = c.width[d];
        s.inv_width[d] = 1.0 / c.width[d];
        s.cell_width[d] = c.cell_width[d];
        s.half_width[d] = c.half_width[d];
        s.gravity[d] = c.gravity[d];
    }
    s.has_st = c.has_st;
    s.ratio_all_one = c.ratio_all_one;
    s.uniform_mu = 1;
    for (int t = 0; t < MPH_TYPE_COUNT; ++t)
        for (int u = 0; u < MPH_TYPE_COUNT; ++u)
            if (c.visc_mu[t][u] != c.visc_mu[0][0]) s.uniform_mu = 0;
    s.dt = c.dt;
    s.shift_thr = c.shift_thr;
    s.vol_d = c.vol;
    for (int t = 0; t < MPH_TYPE_COUNT; ++t) {
        s.density[t] = c.density[t];
        s.bulk_modulus_d[t] = c.bulk_modulus[t];
        s.bulk_viscosity_d[t] = c.bulk_viscosity[t];
        s.a_k[t] = (float)c.a_k[t];
        s.cof_a[t] = (float)c.cof_a[t];
        for (int u = 0; u < MPH_TYPE_COUNT; ++u) {
            s.visc_mu[t][u] = (float)c.visc_mu[t][u];
            s.ratio[t][u] = (float)c.ratio[t][u];
        }
    }
    const double margin = 0.1 * c.l0, rs = k.radius_p + margin;
    s.short_r2 = (float)(rs * rs);
    // table form: the default tile and its hi grid (configure's), and the lists'
    // cut-offs, with room for the FP32 rounding of cell-relative coordinates (below
    // 2 cell widths: three of 2^-24 * 2 cell widths, and as much again)
    double cwmax = 0.0, ext = 0.0;
    for (int d = 0; d < 3; ++d) {
        const int t = c.dim == 2 ? kTile2D[d] : kTile3D[d];
        s.ttile[d] = d < c.dim ? std::max(1, std::min(t, c.cc[d] - 2)) : 1;
        s.cw32[d] = (float)c.cell_width[d];
        if (d >= c.dim) continue;
        cwmax = std::max(cwmax, c.cell_width[d]);
        ext = std::max(ext, (s.ttile[d] + 2.5) * c.cell_width[d]);
    }
    s.rgrid = std::ldexp(1.0, (int)std::ceil(std::log2(ext)) - 23);
    s.inv_rgrid = 1.0 / s.rgrid;
    for (int d = 0; d < 3; ++d) {
        long long bits;
        std::memcpy(&bits, &s.half_width[d], sizeof(bits));
        s.hw_hi[d] = (int)(bits >> 32);
    }
    const double slack = 32.0 * std::ldexp(cwmax, -24);
    const double rl = k.max_radius + margin + slack, rsl = rs + margin + slack;
    s.list_r2 = std::nextafter((float)(rl * rl), INFINITY);
    s.lists_r2 = std::nextafter((float)(rsl * rsl), INFINITY);
    s.ra2 = (float)c.ra2;
    s.rp2 = (float)c.rp2;
    s.rv2 = (float)c.rv2;
    s.rg2 = (float)c.rg2;
    // the density sums take r^2 <= R^2 (main.cpp:1684), the forces r^2 < R^2:
    // pairs are selected by r^2 < cut2 in FP32, so cut2_a lies a little above
    // (the FP64 test r^2 <= RP^2 decides the pressure pairs)
    s.rp2_pre = (float)(c.rp2 * (1.0 + 1e-5));
    s.cut2_a = std::nextafter(c.has_st ? std::max(s.rp2_pre, std::max(s.ra2, s.rg2)) : s.rp2_pre, INFINITY);
    s.cut2_b = std::max(s.rp2, s.rv2);
    if (c.has_st) s.cut2_b = std::max(s.cut2_b, std::max(s.ra2, s.rg2));
    s.inv_ra = (float)(1.0 / c.ra);
    s.inv_rp = (float)(1.0 / c.rp);
    s.inv_rv = (float)(1.0 / c.rv);
    s.inv_rg = (float)(1.0 / c.rg);
    s.ca = (float)c.ca;
    s.cp = (float)c.cp;
    s.cg = (float)c.cg;
    s.cv = (float)c.cv;
    s.cp_m2 = (float)(c.cp * c.m2_rp);
    s.cg_m2 = (float)(c.cg * c.m2_rg);
    s.ca_inv = (float)(c.ca * c.inv_ra);
    s.p_a = (float)(c.cp * c.m2_rp * c.vol);
    s.p_b = (float)(-c.cp * c.m2_rp * c.vol / c.rp);
    s.v_a = (float)(-c.cv * c.m2_rv * c.vol);
    s.v_b = (float)(c.cv * c.m2_rv * c.vol / c.rv);
    s.vol = (float)c.vol;
    s.vol_over_l0 = (float)c.vol_over_l0;
    s.n0a = (float)c.n0a;
    s.n0p = (float)c.n0p;
    s.n0p_d = c.n0p;
    s.rp2_d = c.rp2;
    s.inv_rp_d = 1.0 / c.rp;
    s.cp_d = c.cp;
    s.cp_m2_d = c.cp * c.m2_rp;
    s.inv_r2g_rg = (float)(c.rg / c.r2g);
    s.l0 = (float)c.l0;
}

// The table form (a tile of one cell): blocks of `threads` slots (sweep A) and
// of `threads` fluid particles (sweep B), scene by scene.  Here and in configure() the
// batch changes only once nothing can fail any more: after an error it steps on as it was.
static int configure_table(mph_batch* b, int threads, int ctas_per_sm) {
    const int cta = std::min(threads, 128);  // the kernels' bound; the asked-for size is reported back
    std::vector<int2> ia, ib;
    for (int s = 0; s < b->S; ++s) {
        const BScene& sc = b->hs[s];
        for (int k = 0; k < sc.n; k += cta) ia.push_back(make_int2(s, sc.pbase + k));
        for (int k = 0; k < sc.nfl; k += cta) ib.push_back(make_int2(s, sc.fbase + k));
    }
    int2* items = nullptr;
    BTRY(b, balloc(&items, ia.size() + ib.size()));
    cudaError_t e = cudaMemcpyAsync(items, ia.data(), ia.size() * sizeof(int2), cudaMemcpyHostToDevice, b->stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(items + ia.size(), ib.data(), ib.size() * sizeof(int2), cudaMemcpyHostToDevice, b->stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(b->d_scenes, b->hs.data(), b->hs.size() * sizeof(BScene), cudaMemcpyHostToDevice, b->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(b->stream);  // the vectors go out of scope
    if (e != cudaSuccess) {
        cudaFree(items);
        return bfail(b, MPH_ERR_CUDA, std::string("table form: ") + cudaGetErrorString(e));
    }
    if (b->d_items_t) cudaFree(b->d_items_t);
    b->d_items_t = items;
    BatchDev& d = b->d;
    d.table = 1;
    d.items_a = b->d_items_t;
    d.items_b = b->d_items_t + ia.size();
    for (int k = 0; k < 3; ++k) b->tile[k] = 1;
    b->threads = threads;
    b->table_cta = cta;
    b->occ = std::max(1, std::min(ctas_per_sm, 8));
    b->cap = d.tcap;
    b->n_items = b->grid_a = (int)ia.size();
    b->grid_b = (int)ib.size();
    free_graph(b);
    return MPH_OK;
}

// Tiles, items (largest first by the particle count at creation), staging
// capacity, shared memory and persistent grid sizes for tile t and CTA size.
static int configure(mph_batch* b, const int t[3], int threads, int ctas_per_sm = 2) {
    const int dim = b->dim;
    if (threads < 64 || threads > mph::kMaxThreads || threads % 32 != 0)
        return bfail(b, MPH_ERR_ARG, "threads must be a multiple of 32 in [64, 256]");
    for (int d = 0; d < dim; ++d)
        if (t[d] < 1 || t[d] > 64) return bfail(b, MPH_ERR_ARG, "tile sides must be in [1, 64]");
    if (b->table_ok && t[0] == 1 && t[1] == 1 && (dim == 2 || t[2] == 1)) return configure_table(b, threads, ctas_per_sm);
    int tmax[3] = {1, 1, 1};
    struct Item {
        int4 v;
        long long cost;
    };
    std::vector<Item> items;
    std::vector<BScene> hs = b->hs;
    long long max_halo = 0;
    for (int s = 0; s < b->S; ++s) {
        BScene& sc = hs[s];
        for (int d = 0; d < 3; ++d) sc.tile[d] = 1;
        for (int d = 0; d < dim; ++d) sc.tile[d] = std::max(1, std::min(t[d], sc.cc[d] - 2));  // distinct halo cells
        for (int d = 0; d < 3; ++d) tmax[d] = std::max(tmax[d], sc.tile[d]);
        const std::vector<int>& cnt = b->cell_count[s];
        auto cell_n = [&](int x, int y, int z) {
            x = (x % sc.cc[0] + sc.cc[0]) % sc.cc[0];
            y = (y % sc.cc[1] + sc.cc[1]) % sc.cc[1];
            z = (z % sc.cc[2] + sc.cc[2]) % sc.cc[2];
            return (long long)cnt[((size_t)x * sc.cc[1] + y) * sc.cc[2] + z];
        };
        const int zc = dim == 3 ? sc.cc[2] : 1;
        for (int x0 = 0; x0 < sc.cc[0]; x0 += sc.tile[0])
            for (int y0 = 0; y0 < sc.cc[1]; y0 += sc.tile[1])
                for (int z0 = 0; z0 < zc; z0 += sc.tile[2]) {
                    const int t0 = std::min(sc.tile[0], sc.cc[0] - x0), t1 = std::min(sc.tile[1], sc.cc[1] - y0);
                    const int t2 = dim == 3 ? std::min(sc.tile[2], sc.cc[2] - z0) : 1;
                    long long in = 0, halo = 0;
                    const int hz0 = dim == 3 ? -1 : 0, hz1 = dim == 3 ? t2 + 1 : 1;
                    for (int a = -1; a <= t0; ++a)
                        for (int c = -1; c <= t1; ++c)
                            for (int z = hz0; z < hz1; ++z) {
                                const long long v = cell_n(x0 + a, y0 + c, z0 + z);
                                halo += v;
                                if (a >= 0 && a < t0 && c >= 0 && c < t1 && (dim == 2 || (z >= 0 && z < t2))) in += v;
                            }
                    max_halo = std::max(max_halo, halo);
                    items.push_back({make_int4(s, x0, y0, z0), in});
                }
        // the grid of the hi parts: |tile-relative coordinate| < 2^24 grid
        double ext = 0.0;
        for (int d = 0; d < dim; ++d) ext = std::max(ext, (sc.tile[d] + 2.5) * sc.cell_width[d]);
        sc.grid = std::ldexp(1.0, (int)std::ceil(std::log2(ext)) - 23);
        sc.inv_grid = 1.0 / sc.grid;
    }
    std::stable_sort(items.begin(), items.end(), [](const Item& x, const Item& y) { return x.cost > y.cost; });
    const int hmax = (tmax[0] + 2) * (tmax[1] + 2) * (dim == 3 ? tmax[2] + 2 : 1);
    const int ncol = dim == 3 ? tmax[0] * tmax[1] : tmax[0];
    if (hmax > 65535) return bfail(b, MPH_ERR_ARG, "tile too large");
    // staging capacity: the largest halo at creation with head room, bounded by
    // the shared memory of two resident CTAs per SM
    int dev = 0;
    cudaGetDevice(&dev);
    int smem_optin = 0;
    cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    // shared memory for ctas_per_sm resident CTAs (228 KB per SM, 1 KB reserved per CTA)
    const int occ = std::max(1, std::min(ctas_per_sm, 8));
    const size_t budget = std::min<size_t>((size_t)smem_optin, (size_t)228 * 1024 / occ - 1024) - sizeof(BScene) - 2048;
    int cap = (int)std::min<long long>(max_halo + max_halo / 8 + 32, 1 << 20);
    while (cap > 64 && std::max(mph::sweep_smem(dim, 0, b->has_st, cap, hmax, ncol),
                                mph::sweep_smem(dim, 1, b->has_st, cap, hmax, ncol)) > budget)
        cap -= 32;
    const size_t smem[2] = {mph::sweep_smem(dim, 0, b->has_st, cap, hmax, ncol),
                            mph::sweep_smem(dim, 1, b->has_st, cap, hmax, ncol)};
    int g[2];
    for (int sw = 0; sw < 2; ++sw) {
        mph::SweepFn f = dim == 2 ? mph::sweep_fn<2>(sw, b->has_st) : mph::sweep_fn<3>(sw, b->has_st);
        cudaFuncAttributes fa{};
        BTRY(b, cudaFuncGetAttributes(&fa, f));
        if (smem[sw] + fa.sharedSizeBytes > (size_t)smem_optin)
            return bfail(b, MPH_ERR_ARG, "sweep kernel does not fit on an SM with this tile");
        // the limit belongs to the kernel: never below what another batch asked for
        if ((int)smem[sw] > fa.maxDynamicSharedSizeBytes)
            BTRY(b, cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem[sw]));
        int per = 0;
        BTRY(b, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, f, threads, smem[sw]));
        if (per < 1) return bfail(b, MPH_ERR_ARG, "sweep kernel does not fit on an SM with this tile");
        g[sw] = std::max(1, std::min(per * b->sms, (int)items.size()));
    }
    std::vector<int4> hv(items.size());
    for (size_t k = 0; k < items.size(); ++k) hv[k] = items[k].v;
    int4* d_items = nullptr;
    BTRY(b, balloc(&d_items, hv.size()));
    cudaError_t e = cudaMemcpyAsync(d_items, hv.data(), hv.size() * sizeof(int4), cudaMemcpyHostToDevice, b->stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(b->d_scenes, hs.data(), hs.size() * sizeof(BScene), cudaMemcpyHostToDevice, b->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(b->stream);  // the vectors go out of scope
    if (e != cudaSuccess) {
        cudaFree(d_items);
        return bfail(b, MPH_ERR_CUDA, std::string("tile items: ") + cudaGetErrorString(e));
    }
    if (b->d_items) cudaFree(b->d_items);
    b->d_items = d_items;
    b->hs = std::move(hs);
    for (int d = 0; d < 3; ++d) b->tile[d] = t[d];
    if (dim == 2) b->tile[2] = 1;
    b->threads = threads;
    b->occ = occ;
    b->cap = cap;
    b->hmax = hmax;
    b->ncol = ncol;
    b->n_items = (int)hv.size();
    b->smem_a = smem[0];
    b->smem_b = smem[1];
    b->grid_a = g[0];
    b->grid_b = g[1];
    BatchDev& d = b->d;
    d.n_items = b->n_items;
    d.cap = cap;
    d.hmax = hmax;
    d.ncol = ncol;
    d.items = b->d_items;
    d.table = 0;
    free_graph(b);
    return MPH_OK;
}

// Launch groups: an NVTX range each, and CUDA events around them when
// profiling is enabled (direct launches).
struct BLaunch {
    mph_batch* b;
    int id = -1, count;
    cudaEvent_t a = nullptr;
    BLaunch(mph_batch* bb, const char* name, int c) : b(bb), count(c) {
        nvtxRangePushA(name);
        BatchProfile& p = b->prof;
        if (!p.on) return;
        for (size_t k = 0; k < p.names.size(); ++k)
            if (p.names[k] == name) id = (int)k;
        if (id < 0) {
            id = (int)p.names.size();
            p.names.push_back(name);
            p.launches.push_back(0);
            p.ms.push_back(0.0);
        }
        cudaEventCreate(&a);
        cudaEventRecord(a, b->stream);
    }
    ~BLaunch() {
        nvtxRangePop();
        b->launches += count;
        if (id < 0) return;
        cudaEvent_t e = nullptr;
        cudaEventCreate(&e);
        cudaEventRecord(e, b->stream);
        b->prof.pending.push_back({id, count, a, e});
    }
};

static void launch_table(mph_batch* b, int all) {
    const int nb = std::max(1, std::min(8 * b->sms, b->cells));
    if (b->dim == 2) mph::k_bt_table<2><<<nb, 32 * mph::kTabWarps, 0, b->stream>>>(b->d, all);
    else mph::k_bt_table<3><<<nb, 32 * mph::kTabWarps, 0, b->stream>>>(b->d, all);
}

static int rebuild_launches(const mph_batch* b) { return b->d.table ? 6 : 5; }

static void launch_rebuild(mph_batch* b) {
    const BatchDev& d = b->d;
    const int nb = mph::nblocks(b->n, 256);
    mph::k_bt_hist<<<nb, 256, 0, b->stream>>>(d);
    mph::k_bt_scan<<<b->S, 1024, 0, b->stream>>>(d);
    mph::k_bt_place<<<nb, 256, 0, b->stream>>>(d);
    mph::k_bt_gather<<<nb, 256, 0, b->stream>>>(d);
    if (!d.table) {
        mph::k_bt_commit<false><<<nb, 256, 0, b->stream>>>(d);
        return;
    }
    mph::k_bt_commit<true><<<nb, 256, 0, b->stream>>>(d);
    launch_table(b, 0);
}

// The table of the current sort, from its positions (snap): after steps of the
// tile form, which keeps none, or after the autotuner put the state back.
static int refresh_table(mph_batch* b) {
    if (!b->d.table || b->table_valid || !b->sorted) return MPH_OK;
    BTRY(b, cudaMemsetAsync(b->d.cfluid, 0, (size_t)b->cells * sizeof(int), b->stream));
    BTRY(b, cudaMemsetAsync(b->d.fcount, 0, (size_t)b->S * sizeof(int), b->stream));
    const int nb = mph::nblocks(b->n, 256);
    mph::k_bt_home<<<nb, 256, 0, b->stream>>>(b->d);
    launch_table(b, 1);
    BTRY(b, cudaGetLastError());
    b->launches += 2;
    b->table_valid = true;
    return MPH_OK;
}

static void launch_move(mph_batch* b) {
    const int nb = mph::nblocks(b->n, 256);
    if (b->d.table) mph::k_bt_move<true><<<nb, 256, 0, b->stream>>>(b->d);
    else mph::k_bt_move<false><<<nb, 256, 0, b->stream>>>(b->d);
}

static void launch_sweep(mph_batch* b, int sw) {
    if (b->d.table) {
        const int nb = sw == 0 ? b->grid_a : b->grid_b;
        if (nb == 0) return;  // no fluid
        const int cta = b->table_cta;
#define TABLE_SWEEP(DIM, ST)                                                     \
    if (sw == 0) mph::k_bt_a<DIM, ST><<<nb, cta, 0, b->stream>>>(b->d);   \
    else mph::k_bt_b<DIM, ST><<<nb, cta, 0, b->stream>>>(b->d)
        if (b->dim == 2) {
            if (b->has_st) { TABLE_SWEEP(2, true); } else { TABLE_SWEEP(2, false); }
        } else {
            if (b->has_st) { TABLE_SWEEP(3, true); } else { TABLE_SWEEP(3, false); }
        }
#undef TABLE_SWEEP
        return;
    }
    mph::SweepFn f = b->dim == 2 ? mph::sweep_fn<2>(sw, b->has_st) : mph::sweep_fn<3>(sw, b->has_st);
    f<<<sw == 0 ? b->grid_a : b->grid_b, b->threads, sw == 0 ? b->smem_a : b->smem_b, b->stream>>>(b->d);
}

// One step as direct launches: move, the (usually empty) sort kernels, with
// the table form the table's, sweep A, sweep B.
static void launch_step(mph_batch* b) {
    {
        BLaunch l(b, "batch_move", 1);
        launch_move(b);
    }
    {
        BLaunch l(b, "batch_rebuild", rebuild_launches(b));
        launch_rebuild(b);
    }
    {
        BLaunch l(b, "batch_sweep_a", 1);
        launch_sweep(b, 0);
    }
    {
        BLaunch l(b, "batch_sweep_b", 1);
        launch_sweep(b, 1);
    }
}

static int ensure_graph(mph_batch* b) {
    if (b->exec) return MPH_OK;
    BTRY(b, cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
    const long long before = b->launches;
    for (int k = 0; k < mph::kGraphSteps; ++k) launch_step(b);
    b->launches = before;
    cudaGraph_t g = nullptr;
    BTRY(b, cudaStreamEndCapture(b->stream, &g));
    b->graph = g;
    BTRY(b, cudaGraphInstantiate(&b->exec, g, 0));
    return MPH_OK;
}

static int check_ctl(mph_batch* b) {
    BTRY(b, cudaMemcpyAsync(b->h_ctl, b->d.ctl, 8 * sizeof(int), cudaMemcpyDeviceToHost, b->stream));
    BTRY(b, cudaStreamSynchronize(b->stream));
    const int e = b->h_ctl[1];
    if (e & mph::BERR_CAPACITY)
        return bfail(b, MPH_ERR_CAPACITY, "a one-cell tile and its halo exceed the staging capacity");
    if (e & mph::BERR_NONFINITE) return bfail(b, MPH_ERR_NONFINITE, "non-finite velocity");
    return MPH_OK;
}

// Lattice points within radius r (in spacings) of a lattice point.
static int lattice_count(int dim, double r) {
    const int m = (int)r + 1, zm = dim == 2 ? 0 : m;
    int cnt = 0;
    for (int x = -m; x <= m; ++x)
        for (int y = -m; y <= m; ++y)
            for (int z = -zm; z <= zm; ++z)
                if (x * x + y * y + z * z <= r * r) ++cnt;
    return cnt - 1;
}

// The table form's arrays: lists with a quarter and eight entries of head room
// over the lattice's (longer ones are walked from the cells).  They cost 0.3 KB a
// particle in 2-D and 1.3 KB in 3-D; where that is more than half of the free
// memory the batch runs the tile sweeps.
static cudaError_t want_table(mph_batch* b, int lat_l, int lat_s, Slab& slab) {
    BatchDev& d = b->d;
    const size_t n = (size_t)b->n, cells = (size_t)b->cells;
    d.tcap = ((int)(lat_l * 1.25) + 8 + 3) / 4 * 4;
    d.tcap_s = ((int)(lat_s * 1.25) + 8 + 3) / 4 * 4;
    d.cells = b->cells;
    size_t free_b = 0, total_b = 0;
    cudaError_t e = cudaMemGetInfo(&free_b, &total_b);
    if (e != cudaSuccess) return e;
    if (n * ((size_t)(d.tcap + d.tcap_s) * 4 + 80) + cells * 8 > free_b / 2) {
        b->table_ok = false;
        return cudaSuccess;
    }
    slab.want(&d.cell_scene, cells);
    slab.want(&d.home, n);
    slab.want(&d.rel, n);
    slab.want(&d.v32, n);
    if (b->dim == 2) slab.want(&d.tile2, n);
    slab.want(&d.cfluid, cells);
    slab.want(&d.fcount, (size_t)b->S);
    slab.want(&d.flist, (size_t)b->n_fluid);
    slab.want(&d.tab, n * (size_t)(d.tcap / 4));
    slab.want(&d.tab_s, n * (size_t)(d.tcap_s / 4));
    slab.want(&d.tcnt, n);
    slab.want(&d.tcnt_s, n);
    return cudaSuccess;
}

extern "C" int mph_batch_create(int n_scenes, const mph_params* params, const mph_grid_header* headers, int dim,
                                const int* type, const double* xyz, const double* vel, mph_batch** out) {
    if (!out) return bfail(nullptr, MPH_ERR_ARG, "out is NULL");
    *out = nullptr;
    if (n_scenes < 1 || !params || !headers || !type || !xyz || !vel || (dim != 2 && dim != 3))
        return bfail(nullptr, MPH_ERR_ARG, "bad arguments");
    mph_batch* b = new mph_batch();
    b->dim = dim;
    b->S = n_scenes;
    b->hs.resize(n_scenes);
    b->pbase.assign(n_scenes + 1, 0);
    b->cell_count.resize(n_scenes);
    long long ntot = 0, ctot = 0;
    b->table_ok = true;
    int tab_l = 0, tab_s = 0;  // lattice neighbours within the two lists' radii
    for (int s = 0; s < n_scenes; ++s) {
        const mph_params& p = params[s];
        const mph_grid_header& h = headers[s];
        if (h.particle_count < 1) {
            mph_batch_destroy(b);
            return bfail(nullptr, MPH_ERR_ARG, "every scene needs particles");
        }
        for (int t = 2; t < MPH_TYPE_COUNT; ++t)
            for (int k = 0; k < 3; ++k)
                if (p.wall_velocity[t][k] != 0.0 || p.wall_omega[t][k] != 0.0) {
                    mph_batch_destroy(b);
                    return bfail(nullptr, MPH_ERR_ARG, "the batched form takes static walls only");
                }
        mph_constants k{};
        int st = mph_compute_constants(&p, &h, dim, &k);
        mph::SimConst sc{};
        std::string msg;
        if (st == MPH_OK) st = mph::make_simconst(p, h, k, dim, h.particle_count, sc, msg);
        else msg = "scene constants";
        if (st == MPH_OK && (sc.cc[0] < 3 || sc.cc[1] < 3 || (dim == 3 && sc.cc[2] < 3))) {
            st = MPH_ERR_GEOMETRY;
            msg = "the batched form needs at least 3 cells per axis";
        }
        if (st != MPH_OK) {
            mph_batch_destroy(b);
            return bfail(nullptr, st, "scene " + std::to_string(s) + ": " + msg);
        }
        BScene& bs = b->hs[s];
        fill_bscene(bs, sc, k);
        bs.pbase = (int)ntot;
        bs.cbase = (int)ctot;
        b->pbase[s] = (int)ntot;
        if (sc.has_st) b->has_st = true;
        // table form: home cells are packed with 10 bits per axis
        if (sc.cc[0] > 1024 || sc.cc[1] > 1024 || sc.cc[2] > 1024) b->table_ok = false;
        const double margin = 0.1 * sc.l0;
        tab_l = std::max(tab_l, lattice_count(dim, (k.max_radius + margin) / sc.l0));
        tab_s = std::max(tab_s, lattice_count(dim, (k.radius_p + 2.0 * margin) / sc.l0));
        ntot += h.particle_count;
        ctot += sc.tot;
        if (ntot > (1LL << 30) || ctot > (1LL << 30)) {
            mph_batch_destroy(b);
            return bfail(nullptr, MPH_ERR_ARG, "batch too large");
        }
    }
    b->pbase[n_scenes] = (int)ntot;
    b->n = (int)ntot;
    b->cells = (int)ctot;
    std::vector<double4> hp(ntot), hvv(ntot);
    std::vector<int> hpi(ntot), hsid(ntot), hflags(n_scenes, 1);
    for (int s = 0; s < n_scenes; ++s) {
        b->hs[s].fbase = b->n_fluid;  // of the scenes before
        const BScene& sc = b->hs[s];
        std::vector<int>& cnt = b->cell_count[s];
        cnt.assign((size_t)sc.tot, 0);
        for (int q = 0; q < headers[s].particle_count; ++q) {
            const long long i = (long long)sc.pbase + q;
            const int t = type[i];
            if (t < 0 || t >= MPH_TYPE_COUNT) {
                mph_batch_destroy(b);
                return bfail(nullptr, MPH_ERR_ARG, "particle type out of range");
            }
            for (int k = 0; k < 3; ++k)
                if (!std::isfinite(xyz[3 * i + k]) || !std::isfinite(vel[3 * i + k])) {
                    mph_batch_destroy(b);
                    return bfail(nullptr, MPH_ERR_ARG, "non-finite input");
                }
            hp[i] = make_double4(xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2], (double)t);
            const bool wall = t >= 2;  // static walls: calculateWall gives them zero velocity (main.cpp:2013-2053)
            hvv[i] = wall ? make_double4(0, 0, 0, 0) : make_double4(vel[3 * i], vel[3 * i + 1], vel[3 * i + 2], 0);
            hpi[i] = q;
            hsid[i] = s;
            if (t < 2) {
                ++b->n_fluid;
                ++b->hs[s].nfl;
            }
            int c3[3];
            const double x3[3] = {xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2]};
            for (int k = 0; k < 3; ++k) {
                const double w = sc.width[k];
                double xr = x3[k] - sc.dmin[k];
                xr -= w * std::floor(xr / w);
                c3[k] = std::min(sc.cc[k] - 1, std::max(0, (int)std::floor(xr / sc.cell_width[k])));
            }
            ++cnt[((size_t)c3[0] * sc.cc[1] + c3[1]) * sc.cc[2] + c3[2]];
        }
    }
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&b->sms, cudaDevAttrMultiProcessorCount, dev);
    cudaError_t e = cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking);
    BatchDev& d = b->d;
    const size_t n = (size_t)ntot;
    Slab slab;
    slab.want(&b->d_scenes, (size_t)n_scenes);
    slab.want(&b->d_sid, n);
    slab.want(&d.pos, n);
    slab.want(&d.vel, n);
    slab.want(&d.snap, n);
    slab.want(&d.pidx, n);
    slab.want(&d.pos_t, n);
    slab.want(&d.vel_t, n);
    slab.want(&d.pidx_t, n);
    slab.want(&d.key, n);
    slab.want(&d.slot, n);
    slab.want(&d.tmp, n);
    slab.want(&d.counts, (size_t)ctot);
    slab.want(&d.start, (size_t)ctot + 1);
    slab.want(&d.vp, n);
    slab.want(&d.gc, n);
    slab.want(&d.flags, (size_t)n_scenes);
    slab.want(&d.ctl, 8);
    if (e == cudaSuccess && b->table_ok) e = want_table(b, tab_l, tab_s, slab);
    if (e == cudaSuccess) e = slab.alloc(&b->slab);
    if (e == cudaSuccess) e = cudaMallocHost((void**)&b->h_ctl, 8 * sizeof(int));
    if (e != cudaSuccess) {
        const std::string m = std::string("batch allocation: ") + cudaGetErrorString(e);
        mph_batch_destroy(b);
        return bfail(nullptr, MPH_ERR_NOMEM, m);
    }
    d.n = b->n;
    d.S = n_scenes;
    d.scenes = b->d_scenes;
    d.sid = b->d_sid;
    const int end = (int)ntot;
    const int ctl0[8] = {1, 0, 0, 0, 0, 0, 0, 0};  // sort every scene once
    cudaStream_t st = b->stream;
    e = cudaSuccess;
    if (e == cudaSuccess) e = cudaMemcpyAsync(d.pos, hp.data(), n * sizeof(double4), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d.vel, hvv.data(), n * sizeof(double4), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d.pidx, hpi.data(), n * sizeof(int), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(b->d_sid, hsid.data(), n * sizeof(int), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(d.counts, 0, (size_t)ctot * sizeof(int), st);
    if (e == cudaSuccess) e = cudaMemsetAsync(d.vp, 0, n * sizeof(float4), st);
    if (e == cudaSuccess) e = cudaMemsetAsync(d.gc, 0, n * sizeof(float4), st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d.start + ctot, &end, sizeof(int), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(d.flags, hflags.data(), hflags.size() * sizeof(int), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d.ctl, ctl0, sizeof(ctl0), cudaMemcpyHostToDevice, st);
    std::vector<int> hcs;
    if (b->table_ok) {
        hcs.resize((size_t)ctot);
        for (int s = 0; s < n_scenes; ++s)
            std::fill(hcs.begin() + b->hs[s].cbase, hcs.begin() + b->hs[s].cbase + b->hs[s].tot, s);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync((void*)d.cell_scene, hcs.data(), hcs.size() * sizeof(int), cudaMemcpyHostToDevice, st);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);  // host vectors go out of scope below
    if (e != cudaSuccess) {
        const std::string m = std::string("batch upload: ") + cudaGetErrorString(e);
        mph_batch_destroy(b);
        return bfail(nullptr, MPH_ERR_CUDA, m);
    }
    // the table where it fits, else these tiles, until mph_batch_autotune / set_tiles
    const int t1[3] = {1, 1, 1};
    int rc = b->table_ok ? configure(b, t1, 128) : configure(b, dim == 2 ? kTile2D : kTile3D, 256);
    if (rc == MPH_OK) {
        // the initial sort of every scene (the reference's start-up neighbour
        // build, main.cpp:357-359)
        launch_rebuild(b);
        b->launches += rebuild_launches(b);
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemsetAsync(d.flags, 0, (size_t)n_scenes * sizeof(int), st);
        if (e == cudaSuccess) e = cudaMemsetAsync(d.ctl, 0, 8 * sizeof(int), st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) rc = bfail(b, MPH_ERR_CUDA, std::string("initial sort: ") + cudaGetErrorString(e));
        b->sorted = true;
        b->table_valid = d.table != 0;
    }
    if (rc != MPH_OK) {
        const std::string m = b->err;
        mph_batch_destroy(b);
        return bfail(nullptr, rc, m);
    }
    *out = b;
    return MPH_OK;
}

extern "C" int mph_batch_step(mph_batch* b, int nsteps) {
    if (!b || nsteps < 0) return bfail(b, MPH_ERR_ARG, "bad arguments");
    if (nsteps > 0) {
        const int rc = refresh_table(b);
        if (rc != MPH_OK) return rc;
        if (!b->d.table) b->table_valid = false;
    }
    if (b->prof.on) {
        for (int k = 0; k < nsteps; ++k) launch_step(b);
    } else {
        int left = nsteps;
        if (left >= mph::kGraphSteps) {
            const int rc = ensure_graph(b);
            if (rc != MPH_OK) return rc;
            for (; left >= mph::kGraphSteps; left -= mph::kGraphSteps) {
                BTRY(b, cudaGraphLaunch(b->exec, b->stream));
                b->launches += (3LL + rebuild_launches(b)) * mph::kGraphSteps;
            }
        }
        for (; left > 0; --left) launch_step(b);
    }
    BTRY(b, cudaGetLastError());
    b->steps += nsteps;
    return MPH_OK;
}

extern "C" int mph_batch_synchronize(mph_batch* b) {
    if (!b) return bfail(nullptr, MPH_ERR_ARG, "batch is NULL");
    return check_ctl(b);
}

extern "C" int mph_batch_get_state(mph_batch* b, double* xyz, double* vel) {
    if (!b || !xyz || !vel) return bfail(b, MPH_ERR_ARG, "bad arguments");
    const int rc = check_ctl(b);
    if (rc != MPH_OK) return rc;
    // packed in input order on the device, in the sort's buffers
    const size_t bytes = 3 * (size_t)b->n * sizeof(double);
    double* dx = reinterpret_cast<double*>(b->d.pos_t);
    double* dv = reinterpret_cast<double*>(b->d.vel_t);
    mph::k_bt_state<<<mph::nblocks(b->n, 256), 256, 0, b->stream>>>(b->d, dx, dv);
    ++b->launches;
    BTRY(b, cudaGetLastError());
    BTRY(b, cudaMemcpyAsync(xyz, dx, bytes, cudaMemcpyDeviceToHost, b->stream));
    BTRY(b, cudaMemcpyAsync(vel, dv, bytes, cudaMemcpyDeviceToHost, b->stream));
    BTRY(b, cudaStreamSynchronize(b->stream));
    return MPH_OK;
}

extern "C" int mph_batch_set_tiles(mph_batch* b, int tx, int ty, int tz, int threads, int ctas_per_sm) {
    if (!b) return bfail(nullptr, MPH_ERR_ARG, "batch is NULL");
    if (ctas_per_sm < 0 || ctas_per_sm > 8) return bfail(b, MPH_ERR_ARG, "ctas_per_sm must be in [0, 8]");
    BTRY(b, cudaStreamSynchronize(b->stream));
    const int t[3] = {tx, ty, b->dim == 3 ? tz : 1};
    return configure(b, t, threads, ctas_per_sm > 0 ? ctas_per_sm : b->occ);
}

extern "C" int mph_batch_get_info(mph_batch* b, mph_batch_info* info) {
    if (!b || !info) return bfail(b, MPH_ERR_ARG, "bad arguments");
    const int rc = check_ctl(b);
    if (rc != MPH_OK) return rc;
    std::memset(info, 0, sizeof(*info));
    info->dim = b->dim;
    info->scenes = b->S;
    info->particles = b->n;
    info->fluid_particles = b->n_fluid;
    for (int d = 0; d < 3; ++d) info->tile[d] = b->tile[d];
    info->threads = b->threads;
    info->ctas_per_sm = b->occ;
    info->items = b->n_items;
    info->capacity = b->cap;
    info->grid_a = b->grid_a;
    info->grid_b = b->grid_b;
    info->graph_steps = mph::kGraphSteps;
    info->steps = b->steps;
    info->scene_rebuilds = b->h_ctl[6];
    info->tile_splits = b->h_ctl[7];
    info->launches = b->launches;
    return MPH_OK;
}

// Device state a trial may change: saved before the autotuner's trials and
// put back after each.
struct BatchBackup {
    double4 *pos = nullptr, *vel = nullptr, *snap = nullptr;
    int *pidx = nullptr, *start = nullptr, *flags = nullptr, *ctl = nullptr;
};

static int backup_copy(mph_batch* b, BatchBackup& k, bool save) {
    const size_t n = (size_t)b->n;
    auto cp = [&](void* bk, void* live, size_t bytes) {
        return save ? cudaMemcpyAsync(bk, live, bytes, cudaMemcpyDeviceToDevice, b->stream)
                    : cudaMemcpyAsync(live, bk, bytes, cudaMemcpyDeviceToDevice, b->stream);
    };
    BTRY(b, cp(k.pos, b->d.pos, n * sizeof(double4)));
    BTRY(b, cp(k.vel, b->d.vel, n * sizeof(double4)));
    BTRY(b, cp(k.snap, b->d.snap, n * sizeof(double4)));
    BTRY(b, cp(k.pidx, b->d.pidx, n * sizeof(int)));
    BTRY(b, cp(k.start, b->d.start, ((size_t)b->cells + 1) * sizeof(int)));
    BTRY(b, cp(k.flags, b->d.flags, (size_t)b->S * sizeof(int)));
    BTRY(b, cp(k.ctl, b->d.ctl, 8 * sizeof(int)));
    return MPH_OK;
}

extern "C" int mph_batch_autotune(mph_batch* b, int steps, mph_batch_trial* trials, int capacity, int* count) {
    if (!b || steps < 1) return bfail(b, MPH_ERR_ARG, "bad arguments");
    int rc = check_ctl(b);
    if (rc != MPH_OK) return rc;
    std::vector<std::array<int, 5>> cand;  // tile x, y, z, CTA size, CTAs per SM the staging is sized for
    if (b->table_ok)
        for (int th : {64, 128}) cand.push_back({1, 1, 1, th, 2});
    if (b->dim == 2) {
        const int ts[][2] = {{4, 4}, {4, 8}, {8, 4}, {8, 8}, {8, 16}, {16, 8}, {12, 12}, {16, 16}};
        for (auto& t : ts)
            for (int th : {128, 256})
                for (int oc : {2, 3, 4}) cand.push_back({t[0], t[1], 1, th, oc});
    } else {
        const int ts[][3] = {{1, 2, 2}, {2, 2, 2}, {2, 2, 4}, {2, 4, 4}, {4, 4, 4}, {1, 1, 4}, {1, 2, 4}};
        for (auto& t : ts)
            for (int th : {128, 256})
                for (int oc : {1, 2}) cand.push_back({t[0], t[1], t[2], th, oc});
    }
    const bool prof = b->prof.on;
    b->prof.on = false;
    const long long steps0 = b->steps, launches0 = b->launches;
    const int keep[3] = {b->tile[0], b->tile[1], b->tile[2]}, keep_threads = b->threads, keep_occ = b->occ;
    BatchBackup k;
    const size_t n = (size_t)b->n;
    cudaError_t e = cudaSuccess;
    if (e == cudaSuccess) e = balloc(&k.pos, n);
    if (e == cudaSuccess) e = balloc(&k.vel, n);
    if (e == cudaSuccess) e = balloc(&k.snap, n);
    if (e == cudaSuccess) e = balloc(&k.pidx, n);
    if (e == cudaSuccess) e = balloc(&k.start, (size_t)b->cells + 1);
    if (e == cudaSuccess) e = balloc(&k.flags, (size_t)b->S);
    if (e == cudaSuccess) e = balloc(&k.ctl, 8);
    auto release = [&]() {
        void* ptrs[] = {k.pos, k.vel, k.snap, k.pidx, k.start, k.flags, k.ctl};
        for (void* p : ptrs)
            if (p) cudaFree(p);
    };
    if (e != cudaSuccess) {
        release();
        return bfail(b, MPH_ERR_NOMEM, std::string("autotune backup: ") + cudaGetErrorString(e));
    }
    rc = backup_copy(b, k, true);
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    double best = 1e300;
    int best_i = -1, nt = 0;
    const int rounds = std::max(1, (steps + mph::kGraphSteps - 1) / mph::kGraphSteps);
    for (size_t ci = 0; ci < cand.size() && rc == MPH_OK; ++ci) {
        const int t[3] = {cand[ci][0], cand[ci][1], cand[ci][2]};
        rc = configure(b, t, cand[ci][3], cand[ci][4]);
        if (rc != MPH_OK) {  // a shape this GPU cannot hold: skip it
            cudaGetLastError();
            rc = MPH_OK;
            continue;
        }
        rc = backup_copy(b, k, false);
        b->table_valid = false;
        if (rc == MPH_OK) rc = mph_batch_step(b, mph::kGraphSteps);  // warm-up, builds the graph
        if (rc != MPH_OK) break;
        cudaEventRecord(e0, b->stream);
        for (int r = 0; r < rounds && rc == MPH_OK; ++r) rc = mph_batch_step(b, mph::kGraphSteps);
        cudaEventRecord(e1, b->stream);
        if (rc == MPH_OK) rc = check_ctl(b);
        if (rc != MPH_OK) break;
        float ms = 0.f;
        cudaEventElapsedTime(&ms, e0, e1);
        const double per = ms / (rounds * mph::kGraphSteps);
        if (trials && nt < capacity) {
            trials[nt].tile[0] = b->tile[0];
            trials[nt].tile[1] = b->tile[1];
            trials[nt].tile[2] = b->tile[2];
            trials[nt].threads = b->threads;
            trials[nt].ctas_per_sm = b->occ;
            trials[nt].capacity = b->cap;
            trials[nt].ms_per_step = per;
        }
        ++nt;
        if (per < best) {
            best = per;
            best_i = (int)ci;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (rc == MPH_OK) rc = backup_copy(b, k, false);
    b->table_valid = false;
    if (rc == MPH_OK) {
        if (best_i >= 0) {
            const int t[3] = {cand[best_i][0], cand[best_i][1], cand[best_i][2]};
            rc = configure(b, t, cand[best_i][3], cand[best_i][4]);
        } else {
            rc = configure(b, keep, keep_threads, keep_occ);
        }
    }
    if (rc == MPH_OK) {
        e = cudaStreamSynchronize(b->stream);
        if (e != cudaSuccess) rc = bfail(b, MPH_ERR_CUDA, cudaGetErrorString(e));
    }
    release();
    b->steps = steps0;
    b->launches = launches0;
    b->prof.on = prof;
    if (count) *count = nt;
    return rc;
}

extern "C" void* mph_batch_stream(mph_batch* b) { return b ? (void*)b->stream : nullptr; }

extern "C" int mph_batch_profile_enable(mph_batch* b, int enable) {
    if (!b) return bfail(nullptr, MPH_ERR_ARG, "batch is NULL");
    BTRY(b, cudaStreamSynchronize(b->stream));
    for (auto& pe : b->prof.pending) {
        cudaEventDestroy(pe.a);
        cudaEventDestroy(pe.b);
    }
    b->prof = BatchProfile();
    b->prof.on = enable != 0;
    return MPH_OK;
}

extern "C" int mph_batch_profile_read(mph_batch* b, mph_kernel_stat* out, int capacity, int* count) {
    if (!b) return bfail(nullptr, MPH_ERR_ARG, "batch is NULL");
    BTRY(b, cudaStreamSynchronize(b->stream));
    BatchProfile& p = b->prof;
    for (auto& pe : p.pending) {
        float ms = 0.f;
        cudaEventElapsedTime(&ms, pe.a, pe.b);
        p.ms[pe.id] += ms;
        p.launches[pe.id] += pe.count;
        cudaEventDestroy(pe.a);
        cudaEventDestroy(pe.b);
    }
    p.pending.clear();
    const int nn = (int)p.names.size();
    for (int k = 0; k < nn && k < capacity && out; ++k) {
        std::memset(out[k].name, 0, sizeof(out[k].name));
        std::strncpy(out[k].name, p.names[k].c_str(), sizeof(out[k].name) - 1);
        out[k].launches = p.launches[k];
        out[k].total_ms = p.ms[k];
    }
    if (count) *count = nn;
    return MPH_OK;
}

extern "C" int mph_batch_last_error(mph_batch* b, char* buf, int len) {
    const std::string& m = b ? b->err : g_batch_err;
    if (buf && len > 0) {
        std::strncpy(buf, m.c_str(), (size_t)len - 1);
        buf[len - 1] = 0;
    }
    return (int)m.size();
}
