// k_mixed.cu — the mixed-precision MPH-WC step on sm_100a.
//
// Same physics and step order as the reference loop (main.cpp:386-431), with
//   * a stable counting sort by cell (histogram -> scan -> scatter -> in-cell
//     ordering by previous index) instead of the bitonic network;
//   * FP32 pair arithmetic on cell-relative coordinates: each particle keeps
//     its FP32 offset from the origin of its home cell (the cell of the last
//     list build), and every list entry packs the neighbour index with a 5-bit
//     code of the neighbouring cell's offset, so x_j - x_i = (o_j - o_i) +
//     D[code] never subtracts two large FP32 coordinates;
//   * one neighbour table, entries within RP+margin first, so the density
//     sweep walks the short part only; the force sweep runs for fluid
//     particles only (walls never accelerate);
//   * Kahan-compensated FP32 per-particle sums; FP64 position/velocity
//     integration, FP64 global sums.
// Quantities the reference computes for output only (DensityA without surface
// tension, wall forces) are computed when the state is read back.
#include <algorithm>
#include <cstdlib>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>
#include "mph_mixed.h"
#include "mph_pair32.cuh"

namespace mph {

namespace {

constexpr int kCodeBits = 5;  // 27 neighbour-cell offsets

// Resident 128-thread blocks per SM the force sweep is compiled for (register
// cap 65536 / (128 * blocks)); set by measurement on the full dam break.
#ifndef MPH_MIXB_MINB_FUSED
#define MPH_MIXB_MINB_FUSED 8
#endif
// ... and of its surface-tension variants (more live values per pair), bound by latency:
// us a launch at 4 / 5 / 6 / 7 / 8 blocks on the 592,704-particle two-fluid column
// 728 / 703 / 730 / 794 / 947, on the 830,584-particle one 1031 / 969 / 1025 / 1126 / 1308.
#ifndef MPH_MIXB_MINB_ST
#define MPH_MIXB_MINB_ST 5
#endif
// Resident 128-thread blocks per SM of the table-free force sweep.
#ifndef MPH_WALK_MINB
#define MPH_WALK_MINB 6
#endif

struct MixConst {
    int n, tot, dim, has_st, ratio_all_one, uniform_mu;
    int cap_s;                         // table rows of the short part; the long part follows
    int cc[3], range[3];
    double grid, inv_grid;             // hi-part grid (a power of two, metres)
    float dhi[27][4];                  // cell-origin offset per code: hi part (on the grid)
    float dlo[27][4];                  //                              lo part
    float half_cell[3];                // half of dhi's step of one cell
    float list_r2, short_r2;           // (MaxRadius+m)^2, (RP+m)^2
    float walk_r2, walk_short2;        // cell walk: (largest force radius + s)^2, (RP + s)^2, s = 8 grid steps
    float ra2, rp2, rv2, rg2;
    float inv_ra, inv_rp, inv_rv, inv_rg;
    float ca, cp, cg, cv;              // (1/Sw)/h^D
    float cp_m2, cg_m2, cv_m2, ca_inv; // c*(-2/h); ca/h
    float p_a, p_b;                    // pressure:  cp*(-2/rp)*vol * (1 - r/rp) = p_a + p_b*r
    float v_a, v_b;                    // viscosity: -cv*(-2/rv)*vol * (1 - r/rv) = v_a + v_b*r
    float vol, vol_over_l0, n0a, n0p, inv_r2g_rg, l0;
    double p_a_d, p_b_d, v_a_d, v_b_d, cp_d, cp_m2_d, inv_rp_d, n0p_d;  // FP64 pressure core
    float inv_rp_lo, cp_lo;            // 1/RP and Cp as FP32 pairs: (inv_rp, inv_rp_lo), (cp, cp_lo)
    float visc_mu[MPH_TYPE_COUNT][MPH_TYPE_COUNT];
    float ratio[MPH_TYPE_COUNT][MPH_TYPE_COUNT];
    float a_k[MPH_TYPE_COUNT], cof_a[MPH_TYPE_COUNT];
    float bulk_modulus[MPH_TYPE_COUNT], bulk_viscosity[MPH_TYPE_COUNT];
};

__device__ __forceinline__ double omod(double x, double w) { return x - w * floor(x / w); }
__device__ __forceinline__ double omod_fast(double x, double w) {
    return (x >= 0.0 && x < 0.75 * w) ? x : omod(x, w);
}

__device__ __forceinline__ int pack_cell(int x, int y, int z) { return x | (y << 10) | (z << 20); }

// A particle's 32-byte record {hi position + type, velocity + PressureP} in
// one 256-bit read-only load: one L1 sector per neighbour instead of two.
__device__ __forceinline__ void ldg_pv(const float4* __restrict__ pv, int j, float4& p, float4& v) {
    asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=f"(p.x), "=f"(p.y), "=f"(p.z), "=f"(p.w), "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
        : "l"(pv + 2 * (size_t)j));
}

// Cell-relative position in two FP32 words.  hi lies on a power-of-two grid g
// with |hi| < 2^24 g, so hi_j - hi_i + Dhi (also on the grid) is computed
// exactly; lo = x - hi (|lo| <= g/2) carries the rest.  The pair
// displacement ((hi_j - hi_i) + Dhi) + ((lo_j - lo_i) + Dlo) is then the true
// displacement rounded once to FP32, independent of where the cell sits.
__device__ __forceinline__ void rel32(const SimConst& c, const MixConst& m, const double4& p, int h, float4& hi,
                                      float4& lo) {
    const int hx = h & 1023, hy = (h >> 10) & 1023, hz = (h >> 20) & 1023;
    double d[3] = {p.x - (c.dmin[0] + (double)hx * c.cell_width[0]), p.y - (c.dmin[1] + (double)hy * c.cell_width[1]),
                   p.z - (c.dmin[2] + (double)hz * c.cell_width[2])};
    float h3[3], l3[3];
    for (int k = 0; k < 3; ++k) {
        if (d[k] > c.half_width[k]) d[k] -= c.width[k];  // minimum image from the home cell
        if (d[k] < -c.half_width[k]) d[k] += c.width[k];
        const double q = rint(d[k] * m.inv_grid) * m.grid;
        h3[k] = (float)q;
        l3[k] = (float)(d[k] - q);
    }
    hi = make_float4(h3[0], h3[1], h3[2], __int_as_float((int)p.w));
    lo = make_float4(l3[0], l3[1], l3[2], 0.0f);
}

// The neighbour table holds entries in rows of four: entries 4r..4r+3 of
// particle i are one uint4 at row r, column i (tab[r * n + i]), so a lane
// writes 16 bytes at a time when the table is built and the lanes of a warp
// read consecutive uint4 when it is swept.  Visits entries [0, cnt) in order.
template <class F>
__device__ __forceinline__ void for_entries(const uint4* __restrict__ tab, size_t n, int cnt, F&& f) {
    for (int k = 0; k < cnt; k += 4) {
        const uint4 q = __ldg(tab + (size_t)(k >> 2) * n);
        f(q.x);
        if (k + 1 < cnt) f(q.y);
        if (k + 2 < cnt) f(q.z);
        if (k + 3 < cnt) f(q.w);
    }
}

// The warp's stage of the sweeps with G lanes per particle: one float4 a lane, a
// particle's G behind one another and the particles one more apart, so that the lanes
// which sum different particles' terms meet different banks.
template <int G>
struct LaneStage {
    float4 v[32 + 32 / G];
    __device__ __forceinline__ static int slot(int lane) { return lane + lane / G; }
};

// Walks a list by G lanes per particle, G entries a trip: lane sub evaluates
// entry k0 + sub (eval(record): it stages the terms), then add(m) adds the first m
// of the G staged entries in list order.  tab: the list's first row; self: an entry that names the
// particle, loaded where the list has ended.  Entries are loaded two trips ahead and
// records one.  All lanes of the warp take part; cnt is the particle's.
template <int G, class Load, class Eval, class Add>
__device__ __forceinline__ void lane_walk(const unsigned* __restrict__ tab, size_t n, int i, int cnt, unsigned self,
                                          Load&& load, Eval&& eval, Add&& add) {
    const int sub = threadIdx.x & (G - 1);
    const int most = __reduce_max_sync(0xffffffffu, cnt);
    auto entry = [&](int k) { return k < cnt ? __ldg(tab + ((size_t)(k >> 2) * n + i) * 4 + (k & 3)) : self; };
    unsigned eb = entry(sub + G);
    auto a = load(entry(sub));
    for (int k0 = 0; k0 < most; k0 += G) {
        const unsigned ec = entry(k0 + 2 * G + sub);
        const auto b = load(eb);
        const int m = min(G, max(0, cnt - k0));
        eval(a, sub < m);
        add(m);
        __syncwarp();
        eb = ec;
        a = b;
    }
}

// ---- counting sort by cell ------------------------------------------------

// Cell key of main.cpp:1115-1133 (walls offset by TotalCellCount), its slot in
// the cell (atomic, order fixed later), the cell histogram.
__global__ void k_mix_cellkey(SimConst c, const double4* __restrict__ pos, int* __restrict__ keys,
                              int* __restrict__ slot, int* __restrict__ counts) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    const double4 p = pos[i];
    const int cx = ((int)floor((p.x - c.dmin[0]) / c.cell_width[0])) % c.cc[0];
    const int cy = ((int)floor((p.y - c.dmin[1]) / c.cell_width[1])) % c.cc[1];
    const int cz = ((int)floor((p.z - c.dmin[2]) / c.cell_width[2])) % c.cc[2];
    int id = ((cx % c.cc[0] + c.cc[0]) % c.cc[0]) * c.cc[1] * c.cc[2] +
             ((cy % c.cc[1] + c.cc[1]) % c.cc[1]) * c.cc[2] + ((cz % c.cc[2] + c.cc[2]) % c.cc[2]);
    const int t = (int)p.w;
    if (t >= 2 && t < 4) id += c.tot;
    keys[i] = id;
    slot[i] = atomicAdd(&counts[id], 1);
}

// Exclusive scan of counts[0..m) into out[0..m] (out[m] = total).  Two launches,
// 4096 keys a block: the blocks' sums, then every block adds up the sums before its
// own and scans its keys.  (One block scanning all keys was a serial chain of 130
// loads a thread: 179 us a build at 130,000 keys, 1,526,488 particles; now 10 us.)
constexpr int kScanThreads = 1024, kScanKeys = 4096;

__device__ __forceinline__ int block_scan(int v, int* part, int& total) {  // exclusive
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int x = v;
    for (int o = 1; o < 32; o <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += a;
    }
    if (lane == 31) part[w] = x;
    __syncthreads();
    int before = 0;
    total = 0;
    for (int k = 0; k < kScanThreads / 32; ++k) {
        const int q = part[k];
        if (k < w) before += q;
        total += q;
    }
    __syncthreads();
    return before + x - v;
}

__global__ void __launch_bounds__(kScanThreads) k_mix_scan_sums(const int* __restrict__ counts, int m,
                                                                int* __restrict__ sums) {
    __shared__ int part[kScanThreads / 32];
    int v = 0, total;
    for (int q = 0; q < kScanKeys / kScanThreads; ++q) {
        const int k = blockIdx.x * kScanKeys + q * kScanThreads + threadIdx.x;
        if (k < m) v += counts[k];
    }
    block_scan(v, part, total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kScanThreads)
k_mix_scan(const int* __restrict__ counts, int m, const int* __restrict__ sums, int* __restrict__ out) {
    __shared__ int part[kScanThreads / 32];
    int before = 0, total;
    for (int k = threadIdx.x; k < (int)blockIdx.x; k += kScanThreads) before += sums[k];
    block_scan(before, part, total);
    constexpr int kEach = kScanKeys / kScanThreads;
    const int k0 = blockIdx.x * kScanKeys + threadIdx.x * kEach;
    int cnt[kEach], v = 0;
#pragma unroll
    for (int q = 0; q < kEach; ++q) {
        cnt[q] = k0 + q < m ? counts[k0 + q] : 0;
        v += cnt[q];
    }
    before = total;
    int run = before + block_scan(v, part, total);
#pragma unroll
    for (int q = 0; q < kEach; ++q) {
        if (k0 + q <= m) out[k0 + q] = run;  // the last key's end is the total
        run += cnt[q];
    }
}

__global__ void k_mix_place(int n, const int* __restrict__ keys, const int* __restrict__ slot,
                            const int* __restrict__ start, int* __restrict__ tmp) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    tmp[start[keys[i]] + slot[i]] = i;
}

// Order each cell's particles by their previous index (a stable sort overall).
__global__ void k_mix_rank(int n, const int* __restrict__ keys, const int* __restrict__ start,
                           const int* __restrict__ tmp, int* __restrict__ perm, int* __restrict__ sorted_keys) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const int i = tmp[p];
    const int key = keys[i];
    const int b = start[key], e = start[key + 1];
    int rank = 0;
    for (int q = b; q < e; ++q) rank += tmp[q] < i;
    perm[b + rank] = i;
    sorted_keys[b + rank] = key;
}

// ---- list build -------------------------------------------------------------

// Home cell and FP32 positions after a sort (sorted order).
__global__ void k_mix_home(SimConst c, MixConst m, const double4* __restrict__ pos, const int* __restrict__ keys,
                           const double4* __restrict__ vel, int* __restrict__ home, float4* __restrict__ phl,
                           float4* __restrict__ p32, float4* __restrict__ v32) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    int k = keys[i];
    if (k >= c.tot) k -= c.tot;
    const int h = pack_cell(k / (c.cc[1] * c.cc[2]), (k / c.cc[2]) % c.cc[1], k % c.cc[2]);
    home[i] = h;
    float4 hi, lo;
    rel32(c, m, pos[i], h, hi, lo);
    phl[2 * (size_t)i] = hi;
    phl[2 * (size_t)i + 1] = lo;
    p32[i] = hi;
    const double4 v = vel[i];
    v32[i] = make_float4((float)v.x, (float)v.y, (float)v.z, 0.0f);
}

// Neighbour table.  The particles of one key (a cell's fluid, or its walls) share
// their 3^D stencil and its visiting order (main.cpp:1356-1392); a warp walks it with
// eight of them at a time, taken octant by octant of the cell so that the box
// around them is small.  Each candidate range is read 32 records at a time (one
// coalesced record per lane); those near the box are queued in order in shared
// memory, and every full queue is tested with a candidate per lane against one of
// the eight after the other, in FP32 on the cell-relative hi parts; a ballot
// numbers the hits.  Entries are (j << 5 | code): pairs within RP+margin go to
// rows [0, cap_s), the rest within MaxRadius+margin to rows [cap_s, cap_s +
// cap_l), each part in stencil order, self excluded.  Walls without a fluid
// neighbour get no list (their pressure is never used), and a wall key with no
// fluid in its 3^D cells is not walked at all.
//
// What bounds it: the instruction count.  With a lane per particle, every kept
// candidate tested by every lane and the hits pushed one by one, half of the lanes
// idled in the pushes and in part-filled warps, and a small scene's few warps ran one
// long chain: us a build at 1,526,488 particles (3-D dam) 2447 -> 2049, 258,392 441 -> 347,
// 21,924 324 -> 83, 592,704 (3-D column) 1111 -> 1076, 39,304 316 -> 115, in 2-D 90,000
// 73 -> 62, 3,600 30 -> 14.
constexpr int kMixListParts = 8;     // particles per group
constexpr int kMixListSorted = 128;  // home particles that are taken octant by octant (more: in slot order)

__global__ void __launch_bounds__(32 * kListWarps, 8)
k_mix_list(SimConst c, MixConst m, const float4* __restrict__ p32, const int* __restrict__ cellstart,
           unsigned* __restrict__ list, int cap_l, int* __restrict__ cnt_short, int* __restrict__ cnt_all,
           StepScalars* __restrict__ scal, int key_warps) {
    __shared__ float4 queue_[kListWarps][64];  // candidates near the box, in order (a ring)
    __shared__ float4 home_[kListWarps][kMixListParts];
    __shared__ unsigned char order_[kListWarps][kMixListSorted];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int gw = blockIdx.x * kListWarps + wib;
    const int key = gw / key_warps;  // key_warps warps share a key
    if (key >= 2 * c.tot) return;    // whole warp
    const int hb = cellstart[key], nh = cellstart[key + 1] - hb, first = (gw % key_warps) * kMixListParts;
    if (first >= nh) return;
    const bool is_wall = key >= c.tot;
    const int ci = is_wall ? key - c.tot : key;
    const int ic[3] = {ci / (c.cc[1] * c.cc[2]), (ci / c.cc[2]) % c.cc[1], ci % c.cc[2]};
    int jmin[3], w[3];
    for (int d = 0; d < 3; ++d) {
        const int r = c.range[d];
        w[d] = 2 * r + 1;
        const int b = (2 * r) - (ic[d] + r) % c.cc[d];
        jmin[d] = b > 0 ? b : 0;
    }
    // lane s < w0*w1*w2 holds stencil slot s of the visiting order (x outer, z
    // inner): its fluid's and walls' ranges and its offset code
    const int nsl = w[0] * w[1] * w[2];  // at most 27: range <= 1 on every axis
    int st_b[2] = {0, 0}, st_e[2] = {0, 0}, st_code = 0;
    if (lane < nsl) {
        const int ax = (jmin[0] + lane / (w[1] * w[2])) % w[0], ay = (jmin[1] + (lane / w[2]) % w[1]) % w[1],
                  az = (jmin[2] + lane % w[2]) % w[2];
        const int cx = ((ic[0] - c.range[0] + ax) % c.cc[0] + c.cc[0]) % c.cc[0];
        const int cy = ((ic[1] - c.range[1] + ay) % c.cc[1] + c.cc[1]) % c.cc[1];
        const int cz = ((ic[2] - c.range[2] + az) % c.cc[2] + c.cc[2]) % c.cc[2];
        const int cell = cx * c.cc[1] * c.cc[2] + cy * c.cc[2] + cz;
        st_code = (ax - c.range[0] + 1) * 9 + (ay - c.range[1] + 1) * 3 + (az - c.range[2] + 1);
        st_b[0] = cellstart[cell];
        st_e[0] = cellstart[cell + 1];
        st_b[1] = cellstart[cell + c.tot];
        st_e[1] = cellstart[cell + c.tot + 1];
    }
    if (is_wall && __ballot_sync(0xffffffffu, st_b[0] < st_e[0]) == 0u) {
        for (int h0 = first; h0 < nh; h0 += key_warps * kMixListParts)
            if (lane < min(kMixListParts, nh - h0)) cnt_short[hb + h0 + lane] = cnt_all[hb + h0 + lane] = 0;
        return;
    }
    const int nf = cellstart[c.tot];
    const size_t n = (size_t)c.n;
    const int cap_s = m.cap_s;
    unsigned* const list_l = list + (size_t)cap_s * n;
    float4* const queue = queue_[wib];
    float4* const homes = home_[wib];
    unsigned char* const order = order_[wib];
    const bool sorted = nh > kMixListParts && nh <= kMixListSorted;
    if (sorted) {  // a counting sort by octant of the home cell, along a Gray code (neighbouring octants in a row)
        const float mx = 0.5f * (float)c.cell_width[0], my = 0.5f * (float)c.cell_width[1],
                    mz = 0.5f * (float)c.cell_width[2];
        int base[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (int pass = 0; pass < 2; ++pass) {
            for (int h = 0; h < nh; h += 32) {
                int o = 8;
                if (h + lane < nh) {
                    const float4 f = p32[hb + h + lane];
                    o = (f.x >= mx ? 4 : 0) | (f.y >= my ? 2 : 0) | (f.z >= mz ? 1 : 0);
                    o = (0x54672310u >> (4 * o)) & 7;
                }
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const unsigned mask = __ballot_sync(0xffffffffu, o == q);
                    if (pass == 1 && o == q)
                        order[base[q] + __popc(mask & ((1u << lane) - 1u))] = (unsigned char)(h + lane);
                    base[q] += __popc(mask);
                }
            }
            if (pass == 0) {
                int run = 0;
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const int v = base[q];
                    base[q] = run;
                    run += v;
                }
            }
        }
        __syncwarp();
    }
    const float kInf = __int_as_float(0x7f800000);
    int most = 0, most_s = 0, most_l = 0;
    for (int h0 = first; h0 < nh; h0 += key_warps * kMixListParts) {
        const int np = min(kMixListParts, nh - h0);
        // the group, a particle per lane (0..7), and the box of its hi positions: the
        // hi values, the cell offsets and their sums and differences are exact on the
        // hi grid, so a candidate whose distance to the box is beyond the cut-off is
        // no particle's neighbour
        float b0x = kInf, b0y = kInf, b0z = kInf, b1x = -kInf, b1y = -kInf, b1z = -kInf;
        __syncwarp();
        if (lane < np) {
            const int i = hb + (sorted ? (int)order[h0 + lane] : h0 + lane);
            float4 f = p32[i];
            b0x = b1x = f.x;
            b0y = b1y = f.y;
            b0z = b1z = f.z;
            f.w = __int_as_float(i);
            homes[lane] = f;
        }
#pragma unroll
        for (int o = kMixListParts / 2; o > 0; o >>= 1) {
            b0x = fminf(b0x, __shfl_xor_sync(0xffffffffu, b0x, o));
            b0y = fminf(b0y, __shfl_xor_sync(0xffffffffu, b0y, o));
            b0z = fminf(b0z, __shfl_xor_sync(0xffffffffu, b0z, o));
            b1x = fmaxf(b1x, __shfl_xor_sync(0xffffffffu, b1x, o));
            b1y = fmaxf(b1y, __shfl_xor_sync(0xffffffffu, b1y, o));
            b1z = fmaxf(b1z, __shfl_xor_sync(0xffffffffu, b1z, o));
        }
        b0x = __shfl_sync(0xffffffffu, b0x, 0);
        b0y = __shfl_sync(0xffffffffu, b0y, 0);
        b0z = __shfl_sync(0xffffffffu, b0z, 0);
        b1x = __shfl_sync(0xffffffffu, b1x, 0);
        b1y = __shfl_sync(0xffffffffu, b1y, 0);
        b1z = __shfl_sync(0xffffffffu, b1z, 0);
        __syncwarp();
        int cnt_s = 0, cnt_l = 0;                 // lane p: particle p's
        unsigned wet = is_wall ? 0u : 0xffu;      // by particle: a fluid one, or with a fluid neighbour
        int head = 0, queued = 0;
        auto test = [&](int mm) {  // the first mm (<= 32) of the queue
            const float4 q = queue[(head + lane) & 63];
            const unsigned entry = __float_as_uint(q.w);
            const int j = (int)(entry >> kCodeBits);
            const unsigned below = (1u << lane) - 1u;
#pragma unroll 1
            for (int p = 0; p < np; ++p) {
                const float4 f = homes[p];
                const int i = __float_as_int(f.w);
                const float dx = q.x - f.x, dy = q.y - f.y, dz = q.z - f.z;
                const float r2 = dx * dx + dy * dy + dz * dz;
                const bool in = lane < mm && r2 < m.list_r2 && j != i;
                const bool in_s = in && r2 < m.short_r2;
                const unsigned hits_s = __ballot_sync(0xffffffffu, in_s);
                const unsigned hits_l = __ballot_sync(0xffffffffu, in && !in_s);
                if (is_wall && __ballot_sync(0xffffffffu, in && j < nf)) wet |= 1u << p;
                const int base_l = __shfl_sync(0xffffffffu, cnt_l, p);
                if (in && !in_s) {
                    const int at = base_l + __popc(hits_l & below);
                    if (at < cap_l) list_l[((size_t)(at >> 2) * n + i) * 4 + (at & 3)] = entry;
                }
                if (hits_s != 0u) {
                    const int base = __shfl_sync(0xffffffffu, cnt_s, p);
                    if (in_s) {
                        const int at = base + __popc(hits_s & below);
                        if (at < cap_s) list[((size_t)(at >> 2) * n + i) * 4 + (at & 3)] = entry;
                    }
                }
                if (lane == p) {
                    cnt_l += __popc(hits_l);
                    cnt_s += __popc(hits_s);
                }
            }
        };
        // the candidate chunks one after the other (a slot's fluid, then its walls),
        // the next one's records loaded while this one is worked on
        int sl = -1, cb = 0, e = 0, code = 0;
        auto next = [&]() {  // the next chunk: [cb, min(cb + 32, e)) of half-slot sl
            cb += 32;
            while (cb >= e) {
                if (++sl >= 2 * nsl) return false;
                cb = __shfl_sync(0xffffffffu, sl & 1 ? st_b[1] : st_b[0], sl >> 1);
                e = __shfl_sync(0xffffffffu, sl & 1 ? st_e[1] : st_e[0], sl >> 1);
                code = __shfl_sync(0xffffffffu, st_code, sl >> 1);
            }
            return true;
        };
        bool more = next();
        float4 qn = make_float4(0.f, 0.f, 0.f, 0.f);
        if (more && cb + lane < e) qn = p32[cb + lane];
        while (more || queued > 0) {
            if (more) {
                float4 q = qn;
                const int j = cb + lane;
                const bool in_range = j < e;
                q.x += m.dhi[code][0];
                q.y += m.dhi[code][1];
                q.z += m.dhi[code][2];
                q.w = __uint_as_float(((unsigned)j << kCodeBits) | (unsigned)code);
                more = next();
                if (more && cb + lane < e) qn = p32[cb + lane];
                const float ex = fmaxf(0.f, fmaxf(b0x - q.x, q.x - b1x));
                const float ey = fmaxf(0.f, fmaxf(b0y - q.y, q.y - b1y));
                const float ez = fmaxf(0.f, fmaxf(b0z - q.z, q.z - b1z));
                const bool near = in_range && ex * ex + ey * ey + ez * ez < m.list_r2;
                const unsigned kept = __ballot_sync(0xffffffffu, near);
                if (near) queue[(head + queued + __popc(kept & ((1u << lane) - 1u))) & 63] = q;
                queued += __popc(kept);
                __syncwarp();
            }
            if (queued >= 32 || (!more && queued > 0)) {
                const int mm = min(queued, 32);
                test(mm);
                head += mm;
                queued -= mm;
                __syncwarp();
            }
        }
        if (lane < np) {
            const int i = __float_as_int(homes[lane].w);
            if (!(wet >> lane & 1u)) cnt_s = cnt_l = 0;
            cnt_short[i] = cnt_s;
            cnt_all[i] = cnt_s + cnt_l;
            most = max(most, cnt_s + cnt_l);
            most_s = max(most_s, cnt_s);
            most_l = max(most_l, cnt_l);
        }
    }
    most = __reduce_max_sync(0xffffffffu, most);
    most_s = __reduce_max_sync(0xffffffffu, most_s);
    most_l = __reduce_max_sync(0xffffffffu, most_l);
    if (lane == 0) {
        atomicMax(&scal->max_neighbors, most);
        atomicMax(&scal->max_short, most_s);
        atomicMax(&scal->max_long, most_l);
        if (most_s > cap_s || most_l > cap_l) atomicOr(&scal->flags, DEVFLAG_NEIGHBOR_OVERFLOW);
    }
}

// ---- per step -----------------------------------------------------------------

// Convection, wall motion, periodic wrap and the displacement maximum (the
// same FP64 expressions as the FP64 form's move), plus the FP32 copies of
// position (home-relative, hi/lo) and velocity for the pair sweeps.  AHEAD: a step
// launched ahead of the host, with the counters and the rebuild test of k_move.
template <bool AHEAD>
__global__ void __launch_bounds__(256)
k_mix_move(SimConst c, MixConst m, const int* __restrict__ cellstart, double4* __restrict__ pos,
           double4* __restrict__ vel, const double4* __restrict__ snap, const double* __restrict__ wall_center,
           const int* __restrict__ home, float4* __restrict__ phl, float4* __restrict__ p32,
           float4* __restrict__ v32, StepScalars* __restrict__ scal) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (AHEAD && scal->stop) return;  // set by an earlier launch only, or by this one's last block
    double s2 = 0.0;
    if (i < c.n) {
        const int nf = cellstart[c.tot], we = cellstart[2 * c.tot];
        double4 p = pos[i];
        double4 v = vel[i];
        if (i < nf) {
            p.x += v.x * c.dt;
            p.y += v.y * c.dt;
            p.z += v.z * c.dt;
        } else if (i < we) {
            const int t = (int)p.w;
            const double* C = wall_center + 3 * t;
            const double(*R)[3] = c.wall_rot[t];
            const double* W = c.wall_omega[t];
            const double* U = c.wall_velocity[t];
            double r0 = p.x - C[0], r1 = p.y - C[1], r2 = p.z - C[2];
            r0 = R[0][0] * r0 + R[0][1] * r1 + R[0][2] * r2;
            r1 = R[1][0] * r0 + R[1][1] * r1 + R[1][2] * r2;
            r2 = R[2][0] * r0 + R[2][1] * r1 + R[2][2] * r2;
            v.x = W[1] * r2 - W[2] * r1 + U[0];
            v.y = W[2] * r0 - W[0] * r2 + U[1];
            v.z = W[0] * r1 - W[1] * r0 + U[2];
            vel[i] = v;
            p.x = r0 + C[0] + U[0] * c.dt;
            p.y = r1 + C[1] + U[1] * c.dt;
            p.z = r2 + C[2] + U[2] * c.dt;
        }
        p.x = omod_fast(p.x - c.dmin[0], c.width[0]) + c.dmin[0];
        p.y = omod_fast(p.y - c.dmin[1], c.width[1]) + c.dmin[1];
        p.z = omod_fast(p.z - c.dmin[2], c.width[2]) + c.dmin[2];
        pos[i] = p;
        float4 hi, lo;
        rel32(c, m, p, home[i], hi, lo);
        phl[2 * (size_t)i] = hi;
        phl[2 * (size_t)i + 1] = lo;
        p32[i] = hi;
        v32[i] = make_float4((float)v.x, (float)v.y, (float)v.z, 0.0f);
        const double4 q = snap[i];
        const double d0 = omod_fast(p.x - q.x + c.half_width[0], c.width[0]) - c.half_width[0];
        const double d1 = omod_fast(p.y - q.y + c.half_width[1], c.width[1]) - c.half_width[1];
        const double d2 = omod_fast(p.z - q.z + c.half_width[2], c.width[2]) - c.half_width[2];
        s2 = d0 * d0 + d1 * d1 + d2 * d2;
        if (!(s2 > 0.0)) s2 = 0.0;
    }
    for (int o = 16; o > 0; o >>= 1) {
        const double t = __shfl_xor_sync(0xffffffffu, s2, o);
        s2 = t > s2 ? t : s2;
    }
    __shared__ double red[8];
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s2;
    __syncthreads();
    if (threadIdx.x == 0) {
        double mx = red[0];
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) mx = red[w] > mx ? red[w] : mx;
        if (mx > 0.0) atomicMax(&scal->max_shift2_bits, (unsigned long long)__double_as_longlong(mx));
        if (AHEAD) {
            __threadfence();
            if (atomicAdd(&scal->blocks_done, 1u) == gridDim.x - 1) {  // the last block
                __threadfence();
                const unsigned long long bits = atomicAdd(&scal->max_shift2_bits, 0ull);
                scal->last_shift2_bits = bits;
                scal->max_shift2_bits = 0ull;
                scal->blocks_done = 0u;
                scal->steps_done += 1;
                if (__longlong_as_double((long long)bits) > c.shift_thr) scal->stop = 1;
            }
        }
    }
}

// The hi offset of a code from one 32-bit word instead of four: per axis two bits
// that read, as the top bits of a float, 0.0, +2.0 or -2.0 for an offset of 0, 1 or
// -1 cells, so pj + offset is one FMA with half a cell's (rounded) width.  The
// offsets are these multiples of the grid exactly, so the sum is the same.  A
// shared-memory word at 27 addresses takes one wavefront of the L1 data pipe, the
// four words of dhi took 4.7 of the 30 that a long pair cost.
__device__ __forceinline__ unsigned cell_steps(int code) {
    const unsigned x = (unsigned)(code / 9 + 3) & 3u, y = (unsigned)(code / 3 % 3 + 3) & 3u,
                   z = (unsigned)(code % 3 + 3) & 3u;  // 0, 1, 2 -> 3, 0, 1
    return x << 30 | y << 28 | z << 26;
}

__device__ __forceinline__ float add_step(float a, unsigned steps, float half_width) {
    return fmaf(__uint_as_float(steps & 0xc0000000u), half_width, a);
}

// Offset tables in shared memory: per-lane codes differ, and shared memory
// serves divergent addresses in one access where the constant bank serialises.
struct SharedTables {
    float4 dhi[27];
    float4 dlo[27];
    unsigned steps[27];  // cell_steps
    float mu[MPH_TYPE_COUNT * MPH_TYPE_COUNT];
};

__device__ __forceinline__ void load_tables(const MixConst& m, SharedTables& t) {
    for (int k = threadIdx.x; k < 27; k += blockDim.x) {
        t.dhi[k] = make_float4(m.dhi[k][0], m.dhi[k][1], m.dhi[k][2], 0.f);
        t.dlo[k] = make_float4(m.dlo[k][0], m.dlo[k][1], m.dlo[k][2], 0.f);
        t.steps[k] = cell_steps(k);
    }
    for (int k = threadIdx.x; k < 16; k += blockDim.x) t.mu[k] = m.visc_mu[k / 4][k % 4];
    __syncthreads();
}

// One DensityP term wp = Cp (1 - r/RP)^2 as an unevaluated sum of two FP32
// numbers, added to the pair sum (sh, sl), with FP32 operations only.  The
// displacement arrives as its exact hi part (grid multiples) and its small lo
// part; error-free transformations (Knuth's TwoSum, Dekker's Fast2Sum, the
// FMA product error a*b - RN(a*b); Muller et al., Handbook of Floating-Point
// Arithmetic, chs. 4-5) carry r^2, r, 1 - r/RP and the square to about 2^-44
// relative.  The strain is a small difference of a sum near N0p, so the
// per-term rounding of plain FP32 (~1e-7 relative) would dominate the error.
// wp_square: the square, p2 + p2e; wp_add: times Cp, to the sum.
__device__ __forceinline__ void wp_square(const MixConst& m, float hx, float hy, float hz, float lx, float ly,
                                          float lz, float& p2, float& p2e) {
    // renormalise each axis so that hi is the FP32 rounding of hi + lo
    { const float t = hx + lx; lx -= t - hx; hx = t; }
    { const float t = hy + ly; ly -= t - hy; hy = t; }
    { const float t = hz + lz; lz -= t - hz; hz = t; }
    const float px = hx * hx, py = hy * hy, pz = hz * hz;
    const float ex = fmaf(hx, hx, -px), ey = fmaf(hy, hy, -py), ez = fmaf(hz, hz, -pz);
    const float s1 = px + py;
    float bb = s1 - px;
    const float e1 = (px - (s1 - bb)) + (py - bb);
    const float s2 = s1 + pz;
    bb = s2 - s1;
    const float e2 = (s1 - (s2 - bb)) + (pz - bb);
    float lo = e1 + e2 + ex + ey + ez + 2.0f * (hx * lx + hy * ly + hz * lz);
    const float hi = s2 + lo;
    lo -= hi - s2;
    // r = sqrt(hi + lo): r0 + rl
    const float y = rsqrt_nr(hi);
    const float r0 = hi * y;
    const float rl = (fmaf(-r0, r0, hi) + lo) * (0.5f * y);
    // q = 1 - r / RP: qh + ql
    const float t = r0 * m.inv_rp;
    const float te = fmaf(r0, m.inv_rp, -t) + r0 * m.inv_rp_lo + rl * m.inv_rp;
    const float qh = 1.0f - t;
    const float ql = ((1.0f - qh) - t) - te;
    p2 = qh * qh;
    p2e = fmaf(qh, qh, -p2) + 2.0f * qh * ql;
}
__device__ __forceinline__ void wp_add(const MixConst& m, float p2, float p2e, float& sh, float& sl) {
    // w = Cp q^2: wh + wl
    const float wh = m.cp * p2;
    const float wl = fmaf(m.cp, p2, -wh) + m.cp * p2e + m.cp_lo * p2;
    // (sh, sl) += (wh, wl)
    const float sn = sh + wh;
    const float bb = sn - sh;
    const float se = (sh - (sn - bb)) + (wh - bb);
    sh = sn;
    sl += se + wl;
}

// A pair's terms of sweep A as the factors of their last product, which the sums take
// in with that product's rounding (the compiler's or the sums' own fused
// multiply-add), whoever adds them: this thread, or another lane.
struct DensityTerms {   // DensityP, DivergenceP, within RadiusP
    float p2, p2e;      // wp_square
    float ue, dw;       // u.e, dwp/dr
};
struct DensityTerms64 {
    double wa, wb;      // DensityP: wa wb
    double da, db;      // DivergenceP: - da db
};
template <bool S64>
using DensityTermsOf = std::conditional_t<S64, DensityTerms64, DensityTerms>;

struct DensitySums {
    float sph = 0.f, spl = 0.f, sd = 0.f, cdk = 0.f;
    double spd = 0.0, sdd = 0.0;
    __device__ __forceinline__ void add_p(const MixConst& m, float p2, float p2e) { wp_add(m, p2, p2e, sph, spl); }
    __device__ __forceinline__ void add_p64(double wa, double wb) { spd += wa * wb; }
    __device__ __forceinline__ void add_d(float ue, float dw) { kahan_add(sd, cdk, -ue * dw); }
    __device__ __forceinline__ void add_d64(double da, double db) { sdd -= da * db; }
    // the pair sum is exact to ~2^-44: N0p is subtracted in FP64 (the strain is a
    // small difference of two numbers near N0p)
    template <bool S64>
    __device__ __forceinline__ double strain(const MixConst& m) const {
        return S64 ? spd - m.n0p_d : ((double)sph + (double)spl) - m.n0p_d;
    }
    template <bool S64>
    __device__ __forceinline__ double div() const {
        return S64 ? sdd : (double)sd - (double)cdk;
    }
};

// A pair of the short part: its displacement d (FP32) and squared distance r2, and, where it is within
// RadiusP, its terms to put(terms).  FP32: the exact displacement from the hi and lo parts.
// S64: pair arithmetic in FP64.  velocity(): the neighbour's.
template <bool S64, class Velocity, class Put>
__device__ __forceinline__ void density_pair(const MixConst& m, const SimConst& c, const float4& pi, const float4& li,
                                             const float4& vi, const float4& pj, const float4& lj,
                                             Velocity&& velocity, const float4& dh, const float4& dl, float* d,
                                             float& r2, Put&& put) {
    DensityTermsOf<S64> t;
    if constexpr (S64) {
        // FP64 displacement: the hi difference plus the cell offset is exact in
        // FP32 (grid multiples), the lo parts carry the rest to ~1e-14 l0
        const double dxd = (double)((pj.x - pi.x) + dh.x) + (((double)lj.x - (double)li.x) + (double)dl.x);
        const double dyd = (double)((pj.y - pi.y) + dh.y) + (((double)lj.y - (double)li.y) + (double)dl.y);
        const double dzd = (double)((pj.z - pi.z) + dh.z) + (((double)lj.z - (double)li.z) + (double)dl.z);
        const double r2d = dxd * dxd + dyd * dyd + dzd * dzd;
        if (r2d <= c.rp2) {
            const double y = rsqrt_dnr(r2d);
            const double q = 1.0 - r2d * y * m.inv_rp_d;
            t.wa = m.cp_d * q;
            t.wb = q;
            const double dw = m.cp_m2_d * q;
            const float4 vj = velocity();
            t.da = (((double)vj.x - (double)vi.x) * dxd + ((double)vj.y - (double)vi.y) * dyd +
                    ((double)vj.z - (double)vi.z) * dzd) * y;
            t.db = dw;
            put(t);
        }
        d[0] = (float)dxd;
        d[1] = (float)dyd;
        d[2] = (float)dzd;
        r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
    } else {
        d[0] = ((pj.x - pi.x) + dh.x) + ((lj.x - li.x) + dl.x);
        d[1] = ((pj.y - pi.y) + dh.y) + ((lj.y - li.y) + dl.y);
        d[2] = ((pj.z - pi.z) + dh.z) + ((lj.z - li.z) + dl.z);
        r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
        if (r2 <= m.rp2) {
            wp_square(m, (pj.x - pi.x) + dh.x, (pj.y - pi.y) + dh.y, (pj.z - pi.z) + dh.z, (lj.x - li.x) + dl.x,
                      (lj.y - li.y) + dl.y, (lj.z - li.z) + dl.z, t.p2, t.p2e);  // wp
            const float rinv = rsqrt_nr(r2);
            const float r = r2 * rinv;
            const float q = 1.0f - r * m.inv_rp;
            t.dw = m.cp_m2 * q;  // dwpdr
            const float4 vj = velocity();
            t.ue = ((vj.x - vi.x) * d[0] + (vj.y - vi.y) * d[1] + (vj.z - vi.z) * d[2]) * rinv;
            put(t);
        }
    }
}

// Epilogue of sweep A: coefficients, PressureP, PressureA (main.cpp:1631-1662, 1735-1740, 1904-1906).
template <bool ST, bool S64>
__device__ __forceinline__ void density_finish(const MixConst& m, const SimConst& c, int i, const float4& pi,
                                               const float4& vi, double strain, double div, float dens, float g0,
                                               float g1, float g2, float4* __restrict__ pv, float4* __restrict__ gca,
                                               double* __restrict__ strain_out, double* __restrict__ div_out,
                                               double* __restrict__ dens_a_out, const double4* __restrict__ vel64,
                                               double4* __restrict__ press64) {
    const int ti = __float_as_int(pi.w);
    double kappa = c.bulk_modulus[ti];
    if (strain < 0.0) kappa = 0.0;
    const double pp = -c.bulk_viscosity[ti] * div + kappa * strain;
    float pa = 0.0f;
    if (ST) {
        pa = m.cof_a[ti] * (dens - m.n0a) / m.l0;
        if (m.n0a <= dens) pa = 0.0f;
        dens_a_out[i] = dens;
        gca[i] = make_float4(g0, g1, g2, pa);
    }
    pv[2 * (size_t)i] = pi;
    pv[2 * (size_t)i + 1] = make_float4(vi.x, vi.y, vi.z, (float)pp);
    if (S64) {
        const double4 vid = vel64[i];
        press64[i] = make_double4(vid.x, vid.y, vid.z, pp);
    }
    strain_out[i] = strain;
    div_out[i] = div;
}

__device__ __forceinline__ void advance_wall_centers(const SimConst& c, double* __restrict__ wall_center) {
    if (wall_center != nullptr && blockIdx.x == 0 && threadIdx.x < 12) {
        const int t = threadIdx.x / 3, d = threadIdx.x % 3;
        if (t >= 2) wall_center[3 * t + d] += c.wall_velocity[t][d] * c.dt;
    }
}

// Sweep A: DensityP and DivergenceP over the short part of the list
// (density_pair), plus, with surface tension, DensityA and GravityCenter over all
// of it (main.cpp:1665-1727, 1831-1896), a thread per particle.
template <bool ST, bool RATIO, bool S64>
__global__ void __launch_bounds__(128)
k_mix_a(MixConst m, const float4* __restrict__ phl, const float4* __restrict__ p32, const float4* __restrict__ v32,
        const unsigned* __restrict__ list, const int* __restrict__ cnt_short, const int* __restrict__ cnt_all,
        float4* __restrict__ pv, float4* __restrict__ gca, double* __restrict__ strain_out,
        double* __restrict__ div_out, double* __restrict__ dens_a_out, double* __restrict__ wall_center,
        const SimConst c, const double4* __restrict__ vel64,
        double4* __restrict__ press64, const StepScalars* __restrict__ skip) {
    __shared__ SharedTables tb;
    if (skip != nullptr && skip->stop) return;  // launched ahead of a step that has to rebuild
    load_tables(m, tb);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    advance_wall_centers(c, wall_center);
    if (i >= m.n) return;
    const float4 pi = phl[2 * (size_t)i];
    const float4 li = phl[2 * (size_t)i + 1];
    const float4 vi = v32[i];
    const int ti = __float_as_int(pi.w);
    const int ns = cnt_short[i];
    const int na = ST ? cnt_all[i] : ns;
    const size_t n = (size_t)m.n;
    DensitySums q;
    float sa = 0.f, cak = 0.f, g0 = 0.f, g1 = 0.f, g2 = 0.f;
    const uint4* tab = reinterpret_cast<const uint4*>(list) + i;
    for_entries(tab, n, ns, [&](unsigned e) {
        const int j = (int)(e >> kCodeBits), code = (int)(e & 31u);
        float4 pj, lj;
        ldg_pv(phl, j, pj, lj);  // {hi, lo} in one 256-bit load
        float d[3], r2;
        density_pair<S64>(m, c, pi, li, vi, pj, lj, [&] { return v32[j]; }, tb.dhi[code], tb.dlo[code], d, r2,
                          [&](const DensityTermsOf<S64>& t) {
            if constexpr (S64) {
                q.add_p64(t.wa, t.wb);
                q.add_d64(t.da, t.db);
            } else {
                q.add_p(m, t.p2, t.p2e);
                q.add_d(t.ue, t.dw);
            }
        });
        if (ST) {
            const float rinv = rsqrt_nr(r2);
            st_density<RATIO>(m, ti, __float_as_int(pj.w), r2, r2 * rinv, d[0], d[1], d[2], sa, cak, g0, g1, g2);
        }
    });
    if (ST) {  // surface tension only: the long part, on the 16-byte hi records
        const uint4* tl = tab + (size_t)(m.cap_s >> 2) * n;
        const int nl = na - ns;
        for (int k = 0; k < nl; k += 4, tl += n) {
            const uint4 q4 = __ldg(tl);
            const unsigned e[4] = {q4.x, q4.y, q4.z, q4.w};
            float4 pj[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (k + u < nl) pj[u] = __ldg(p32 + (e[u] >> kCodeBits));
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (k + u < nl) {
                    const unsigned st = tb.steps[e[u] & 31u];
                    const float dx = add_step(pj[u].x - pi.x, st, m.half_cell[0]),
                                dy = add_step(pj[u].y - pi.y, st << 2, m.half_cell[1]),
                                dz = add_step(pj[u].z - pi.z, st << 4, m.half_cell[2]);
                    const float r2 = dx * dx + dy * dy + dz * dz;
                    st_density<RATIO>(m, ti, __float_as_int(pj[u].w), r2, r2 * rsqrtf(r2), dx, dy, dz, sa, cak, g0, g1,
                                      g2);
                }
        }
    }
    density_finish<ST, S64>(m, c, i, pi, vi, q.strain<S64>(m), q.div<S64>(), sa - cak, g0, g1, g2, pv, gca, strain_out,
                            div_out, dens_a_out, vel64, press64);
}

// A pair's terms of DensityA (sa x y) and GravityCenter (g += d w), as st_density has
// them; bit 0 of the return value: the first is in range, bit 1: the second.
template <bool RATIO>
__device__ __forceinline__ int st_density_terms(const MixConst& m, int ti, int tj, float r2, float r, float& x,
                                                float& y, float& w) {
    const float ratio = RATIO ? m.ratio[ti][tj] : 1.0f;
    int in = 0;
    if (r2 <= m.ra2) {
        const float q = r * m.inv_ra;
        x = ratio * m.ca * q * (1.0f - q);
        y = 1.0f - q;
        in = 1;
    }
    if (r2 <= m.rg2) {
        const float q = 1.0f - r * m.inv_rg;
        w = ratio * m.cg * q * q * m.inv_r2g_rg;
        in |= 2;
    }
    return in;
}

// Sweep A with G lanes per particle (small scenes, lanes_a): the lanes compute the
// terms of G consecutive entries, stage them in shared memory, and one lane per sum adds
// them in list order: the additions of k_mix_a in its order, so the same bits.
template <bool ST, bool RATIO, bool S64, int G>
__global__ void __launch_bounds__(128)
k_mix_a_g(MixConst m, const float4* __restrict__ phl, const float4* __restrict__ p32, const float4* __restrict__ v32,
          const unsigned* __restrict__ list, const int* __restrict__ cnt_short, const int* __restrict__ cnt_all,
          float4* __restrict__ pv, float4* __restrict__ gca, double* __restrict__ strain_out,
          double* __restrict__ div_out, double* __restrict__ dens_a_out, double* __restrict__ wall_center,
          const SimConst c, const double4* __restrict__ vel64,
          double4* __restrict__ press64, const StepScalars* __restrict__ skip) {
    __shared__ SharedTables tb;
    __shared__ LaneStage<G> stage_[4][S64 ? 2 : 1];            // DensityP's and DivergenceP's factors
    __shared__ LaneStage<G> stage_st_[ST ? 4 : 1][ST ? 2 : 1];  // {d, w}; {x, y} of DensityA
    if (skip != nullptr && skip->stop) return;  // launched ahead of a step that has to rebuild
    load_tables(m, tb);
    advance_wall_centers(c, wall_center);
    const int lane = threadIdx.x & 31, sub = lane & (G - 1), wib = threadIdx.x >> 5;
    const int iw = (blockIdx.x * 4 + wib) * (32 / G);
    if (iw >= m.n) return;  // whole warp
    const bool on = iw + lane / G < m.n;
    const int i = on ? iw + lane / G : m.n - 1;
    LaneStage<G>* const st = stage_[wib];
    LaneStage<G>* const ss = stage_st_[ST ? wib : 0];
    const int mine = LaneStage<G>::slot(lane), col = LaneStage<G>::slot(lane - sub);
    const float4 pi = phl[2 * (size_t)i];
    const float4 li = phl[2 * (size_t)i + 1];
    const float4 vi = v32[i];
    const int ti = __float_as_int(pi.w);
    const int ns = on ? cnt_short[i] : 0;
    const int nl = ST && on ? cnt_all[i] - ns : 0;
    const size_t n = (size_t)m.n;
    const unsigned self = (unsigned)i << kCodeBits | 13u;  // code 13: the home cell
    DensitySums q;              // lane 0: DensityP; lane 1: DivergenceP
    float sa = 0.f, cak = 0.f;  // lane 2: DensityA
    float gs = 0.f;             // GravityCenter: component gcomp
    const int gcomp = G >= 8 ? sub - 3 : (sub + 1) & 3;
    unsigned in_p = 0u, in_a = 0u, in_g = 0u;
    // DensityA and GravityCenter of one entry into the stage
    auto stage_st = [&](bool have, int tj, float r2, float r, float dx, float dy, float dz) {
        float x = 0.f, y = 0.f, w = 0.f;
        const int in = have ? st_density_terms<RATIO>(m, ti, tj, r2, r, x, y, w) : 0;
        ss[0].v[mine] = make_float4(dx, dy, dz, w);
        ss[ST ? 1 : 0].v[mine].x = x;
        ss[ST ? 1 : 0].v[mine].y = y;
        in_a = __ballot_sync(0xffffffffu, in & 1) >> (lane - sub);
        in_g = __ballot_sync(0xffffffffu, in & 2) >> (lane - sub);
    };
    auto add_st = [&]() {
        if (sub == 2) {
#pragma unroll
            for (int e = 0; e < G; ++e)
                if (in_a >> e & 1u) {
                    const float4 t = ss[ST ? 1 : 0].v[col + e];
                    kahan_add(sa, cak, t.x * t.y);
                }
        }
        if (gcomp >= 0 && gcomp < 3) {
#pragma unroll
            for (int e = 0; e < G; ++e)
                if (in_g >> e & 1u) {
                    const float* t = reinterpret_cast<const float*>(&ss[0].v[col + e]);
                    gs += t[gcomp] * t[3];
                }
        }
    };
    struct Rec {
        float4 p, l, v;
        unsigned code;
    };
    lane_walk<G>(
        list, n, i, ns, self,
        [&](unsigned e) {
            Rec r;
            ldg_pv(phl, (int)(e >> kCodeBits), r.p, r.l);
            r.v = __ldg(v32 + (e >> kCodeBits));
            r.code = e & 31u;
            return r;
        },
        [&](const Rec& rj, bool have) {
            float d[3] = {0.f, 0.f, 0.f}, r2 = 0.f;
            DensityTermsOf<S64> t{};
            bool in = false;
            if (have)
                density_pair<S64>(m, c, pi, li, vi, rj.p, rj.l, [&] { return rj.v; }, tb.dhi[rj.code],
                                  tb.dlo[rj.code], d, r2, [&](const DensityTermsOf<S64>& terms) {
                    t = terms;
                    in = true;
                });
            if constexpr (S64) {
                *reinterpret_cast<double2*>(&st[0].v[mine]) = make_double2(t.wa, t.wb);
                *reinterpret_cast<double2*>(&st[1].v[mine]) = make_double2(t.da, t.db);
            } else {
                st[0].v[mine] = make_float4(t.p2, t.p2e, t.ue, t.dw);
            }
            in_p = __ballot_sync(0xffffffffu, in) >> (lane - sub);
            if (ST) {
                const float rinv = rsqrt_nr(r2);
                stage_st(have, __float_as_int(rj.p.w), r2, r2 * rinv, d[0], d[1], d[2]);
            }
            __syncwarp();
        },
        [&](int) {
            if (sub < 2) {
#pragma unroll
                for (int e = 0; e < G; ++e)
                    if (in_p >> e & 1u) {
                        if constexpr (S64) {
                            const double2 t = *reinterpret_cast<const double2*>(&st[sub].v[col + e]);
                            if (sub == 0) q.add_p64(t.x, t.y);
                            else q.add_d64(t.x, t.y);
                        } else {
                            const float4 t = st[0].v[col + e];
                            if (sub == 0) q.add_p(m, t.x, t.y);
                            else q.add_d(t.z, t.w);
                        }
                    }
            }
            if (ST) add_st();
        });
    if (ST) {  // the long part, on the 16-byte hi records
        struct RecL {
            float4 p;
            unsigned steps;
        };
        lane_walk<G>(
            list + (size_t)m.cap_s * n, n, i, nl, self,
            [&](unsigned e) { return RecL{__ldg(p32 + (e >> kCodeBits)), tb.steps[e & 31u]}; },
            [&](const RecL& rj, bool have) {
                const float dx = add_step(rj.p.x - pi.x, rj.steps, m.half_cell[0]),
                            dy = add_step(rj.p.y - pi.y, rj.steps << 2, m.half_cell[1]),
                            dz = add_step(rj.p.z - pi.z, rj.steps << 4, m.half_cell[2]);
                const float r2 = dx * dx + dy * dy + dz * dz;
                stage_st(have, __float_as_int(rj.p.w), r2, r2 * rsqrtf(r2), dx, dy, dz);
                __syncwarp();
            },
            [&](int) { add_st(); });
    }
    const int l0 = lane - sub;
    const double strain = q.strain<S64>(m);
    const double div = __shfl_sync(0xffffffffu, q.div<S64>(), l0 + 1);
    float dens = 0.f, g[3] = {0.f, 0.f, 0.f};
    if (ST) {
        dens = __shfl_sync(0xffffffffu, sa - cak, l0 + 2);
#pragma unroll
        for (int k = 0; k < 3; ++k) g[k] = __shfl_sync(0xffffffffu, gs, l0 + (G >= 8 ? k + 3 : (k + 3) & 3));
    }
    if (sub != 0 || !on) return;
    density_finish<ST, S64>(m, c, i, pi, vi, strain, div, dens, g[0], g[1], g[2], pv, gca, strain_out, div_out,
                            dens_a_out, vel64, press64);
}

// A pair of the short part: exact displacement d, PressureP and ViscosityV (and the
// surface-tension terms); false when it is out of every range.  The force is s d + t.
template <bool ST, bool RATIO>
__device__ __forceinline__ bool force_pair_short(const MixConst& m, const SharedTables& tb, unsigned code,
                                                 const float4& pi, const float4& li, const float4& vi, int ti,
                                                 float mu_u, const float4& gi, float ai, const float4& pj,
                                                 const float4& lj, const float4& vj, const float4& gj, float* d,
                                                 float& s, float3& t) {
    const float4 dh = tb.dhi[code], dl = tb.dlo[code];
    const float dx = ((pj.x - pi.x) + dh.x) + ((lj.x - li.x) + dl.x);
    const float dy = ((pj.y - pi.y) + dh.y) + ((lj.y - li.y) + dl.y);
    const float dz = ((pj.z - pi.z) + dh.z) + ((lj.z - li.z) + dl.z);
    const float r2 = dx * dx + dy * dy + dz * dz;
    if (!(r2 < m.rv2 || r2 < m.rp2 || (ST && (r2 < m.ra2 || r2 < m.rg2)))) return false;
    const float rinv = rsqrt_nr(r2);
    const float r = r2 * rinv;
    const int tj = __float_as_int(pj.w);
    s = 0.0f;
    if (r2 < m.rp2) s += (vi.w + vj.w) * fmaf(m.p_b, r, m.p_a) * rinv;
    if (r2 < m.rv2) {
        const float mu = m.uniform_mu ? mu_u : tb.mu[ti * 4 + tj];
        const float ud = (vj.x - vi.x) * dx + (vj.y - vi.y) * dy + (vj.z - vi.z) * dz;
        s += mu * ud * fmaf(m.v_b, r, m.v_a) * (rinv * rinv * rinv);
    }
    t = make_float3(0.f, 0.f, 0.f);
    if (ST) s += st_terms<RATIO>(m, ti, tj, r2, r, rinv, dx, dy, dz, gi, gj, ai, t);
    d[0] = dx;
    d[1] = dy;
    d[2] = dz;
    return true;
}

// A pair of the long part: the hi displacement, ViscosityV (and surface tension); the
// force is t, where the return value says that there is one, then s d.
template <bool ST, bool RATIO>
__device__ __forceinline__ bool force_pair_long(const MixConst& m, const SharedTables& tb, unsigned code,
                                                const float4& pi, const float4& vi, int ti, float mu_u,
                                                const float4& gi, float ai, const float4& pj, const float4& vj,
                                                const float4& gj, float* d, float& s, float3& t) {
    float dx, dy, dz;
    if (ST) {  // short of registers: the table's three words cost less than the steps' one
        const float4 dh = tb.dhi[code];
        dx = (pj.x - pi.x) + dh.x;
        dy = (pj.y - pi.y) + dh.y;
        dz = (pj.z - pi.z) + dh.z;
    } else {
        const unsigned st = tb.steps[code];
        dx = add_step(pj.x - pi.x, st, m.half_cell[0]);
        dy = add_step(pj.y - pi.y, st << 2, m.half_cell[1]);
        dz = add_step(pj.z - pi.z, st << 4, m.half_cell[2]);
    }
    const float r2 = dx * dx + dy * dy + dz * dz;
    const float rinv = rsqrtf(r2);
    s = 0.0f;
    if (r2 < m.rv2) {
        const float r = r2 * rinv;
        const float mu = m.uniform_mu ? mu_u : tb.mu[ti * 4 + __float_as_int(pj.w)];
        const float ud = (vj.x - vi.x) * dx + (vj.y - vi.y) * dy + (vj.z - vi.z) * dz;
        s = mu * ud * fmaf(m.v_b, r, m.v_a) * (rinv * rinv * rinv);
    }
    d[0] = dx;
    d[1] = dy;
    d[2] = dz;
    if (ST && (r2 < m.ra2 || r2 < m.rg2)) {
        t = make_float3(0.f, 0.f, 0.f);
        s += st_terms<RATIO>(m, ti, __float_as_int(pj.w), r2, r2 * rinv, rinv, dx, dy, dz, gi, gj, ai, t);
        return true;
    }
    return false;
}

// Gravity and the FP64 velocity update of a fluid particle with pair force F.
__device__ __forceinline__ void force_finish(const SimConst& c, int i, int ti, double F0, double F1, double F2,
                                             const double4* __restrict__ vel, double4* __restrict__ vel_out,
                                             double4* __restrict__ force, StepScalars* __restrict__ scal) {
    double4 v = vel[i];
    const double mass = c.density[ti] * c.vol;
    F0 += mass * c.gravity[0];
    F1 += mass * c.gravity[1];
    F2 += mass * c.gravity[2];
    v.x += F0 / mass * c.dt;
    v.y += F1 / mass * c.dt;
    v.z += F2 / mass * c.dt;
    if (!(isfinite(v.x) && isfinite(v.y) && isfinite(v.z))) atomicOr(&scal->flags, DEVFLAG_NONFINITE);
    force[i] = make_double4(F0, F1, F2, 0.0);
    vel_out[i] = v;
}

// Sweep B for fluid particles (WALLS: for the wall particles, output only), a thread per particle,
// FP32 in both mixed forms (the FP64 density sweep of MPH_MODE_MIXED_P64 sets
// the pressures this sweep reads).  The short part of the list
// (force_pair_short): Kahan sums.  The long part (force_pair_long):
// plain FP32 sum.  Then gravity and the FP64 velocity update
// (main.cpp:1908-2010).
//
// What bounds it: the L1 data pipe (90 % of its cycles without surface tension), which
// spends 17.6 of them on a warp's gather, one for each 128-byte line that holds
// some of its 32 records.  With the offset's one word (cell_steps) a launch takes 656 us
// instead of 696 at 1,024,000 fluid particles.  A thread per two neighbouring particles
// with a common list gathered once took 884: the warp runs the longest of its lanes'
// lists, and the order within cells that keeps its records in few lines is lost.
template <bool ST, bool RATIO, bool WALLS>
__global__ void __launch_bounds__(128, ST ? MPH_MIXB_MINB_ST : MPH_MIXB_MINB_FUSED)
k_mix_b(MixConst m, SimConst c, const int* __restrict__ cellstart, const float4* __restrict__ phl,
        const float4* __restrict__ pv, const float4* __restrict__ gca,
        const unsigned* __restrict__ list, const int* __restrict__ cnt_short, const int* __restrict__ cnt_all,
        const double4* __restrict__ vel, double4* __restrict__ vel_out, double4* __restrict__ force,
        StepScalars* __restrict__ scal, bool ahead) {
    __shared__ SharedTables tb;
    if (ahead && scal->stop) return;
    load_tables(m, tb);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m.n) return;
    const int nf = cellstart[c.tot];
    if (WALLS ? i < nf : i >= nf) {
        if (!WALLS) vel_out[i] = vel[i];
        return;
    }
    const float4 pi = phl[2 * (size_t)i];
    const float4 li = phl[2 * (size_t)i + 1];
    const float4 vi = pv[2 * (size_t)i + 1];
    const int ti = __float_as_int(pi.w);
    float4 gi = make_float4(0.f, 0.f, 0.f, 0.f);
    if (ST) gi = gca[i];
    const float ai = m.a_k[ti];
    const int ns = cnt_short[i], na = cnt_all[i];
    const size_t n = (size_t)m.n;
    const float mu_u = tb.mu[ti * 4 + ti];
    float fx = 0.f, fy = 0.f, fz = 0.f, cx = 0.f, cy = 0.f, cz = 0.f;  // short part, Kahan
    float gx = 0.f, gy = 0.f, gz = 0.f;                                 // long part
    const uint4* tab = reinterpret_cast<const uint4*>(list) + i;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    for_entries(tab, n, ns, [&](unsigned e) {
        const int j = (int)(e >> kCodeBits);
        float4 pj, vj;
        ldg_pv(pv, j, pj, vj);
        float d[3], s;
        float3 t;
        if (!force_pair_short<ST, RATIO>(m, tb, e & 31u, pi, li, vi, ti, mu_u, gi, ai, pj, phl[2 * (size_t)j + 1], vj,
                                         ST ? gca[j] : zero, d, s, t))
            return;
        kahan_add(fx, cx, fmaf(s, d[0], t.x));
        kahan_add(fy, cy, fmaf(s, d[1], t.y));
        kahan_add(fz, cz, fmaf(s, d[2], t.z));
    });
    // long part: a row of four pairs per iteration, their gathers issued
    // together so a thread keeps four independent loads in flight
    const uint4* tl = tab + (size_t)(m.cap_s >> 2) * n;
    const int nl = na - ns;
    for (int k = 0; k < nl; k += 4) {
        const uint4 q = __ldg(tl + (size_t)(k >> 2) * n);
        const unsigned e[4] = {q.x, q.y, q.z, q.w};
        float4 pj[4], vj[4], gj[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (k + u < nl) {
                ldg_pv(pv, (int)(e[u] >> kCodeBits), pj[u], vj[u]);
                if (ST) gj[u] = __ldg(gca + (e[u] >> kCodeBits));
            }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (k + u < nl) {
                float d[3], s;
                float3 t;
                if (force_pair_long<ST, RATIO>(m, tb, e[u] & 31u, pi, vi, ti, mu_u, gi, ai, pj[u], vj[u], gj[u], d, s,
                                               t)) {
                    gx += t.x;
                    gy += t.y;
                    gz += t.z;
                }
                gx = fmaf(s, d[0], gx);
                gy = fmaf(s, d[1], gy);
                gz = fmaf(s, d[2], gz);
            }
    }
    const double F0 = ((double)fx - (double)cx) + (double)gx;
    const double F1 = ((double)fy - (double)cy) + (double)gy;
    const double F2 = ((double)fz - (double)cz) + (double)gz;
    if (WALLS) force[i] = make_double4(F0, F1, F2, 0.0);
    else force_finish(c, i, ti, F0, F1, F2, vel, vel_out, force, scal);
}

// Sweep B with G lanes per fluid particle (small scenes, lanes_b), as k_mix_a_g: lane k
// < 3 adds component k of the staged terms in list order, with the additions of k_mix_b, so
// the same bits.  The walls keep their velocity in the blocks behind.
template <bool ST, bool RATIO, int G>
__global__ void __launch_bounds__(128)
k_mix_b_g(MixConst m, SimConst c, int nf, int group_blocks, const float4* __restrict__ phl,
          const float4* __restrict__ pv, const float4* __restrict__ gca, const unsigned* __restrict__ list,
          const int* __restrict__ cnt_short, const int* __restrict__ cnt_all, const double4* __restrict__ vel,
          double4* __restrict__ vel_out, double4* __restrict__ force, StepScalars* __restrict__ scal, bool ahead) {
    __shared__ SharedTables tb;
    __shared__ LaneStage<G> stage_[4][ST ? 2 : 1];  // short: s d + t; long: {d, s}, t
    if (ahead && scal->stop) return;
    if ((int)blockIdx.x >= group_blocks) {  // walls
        const int i = nf + ((int)blockIdx.x - group_blocks) * 128 + (int)threadIdx.x;
        if (i < m.n) vel_out[i] = vel[i];
        return;
    }
    load_tables(m, tb);
    const int lane = threadIdx.x & 31, sub = lane & (G - 1), wib = threadIdx.x >> 5;
    const int iw = (blockIdx.x * 4 + wib) * (32 / G);
    if (iw >= nf) return;  // whole warp
    const bool on = iw + lane / G < nf;
    const int i = on ? iw + lane / G : nf - 1;
    LaneStage<G>* const st = stage_[wib];
    const int mine = LaneStage<G>::slot(lane), col = LaneStage<G>::slot(lane - sub);
    const float4 pi = phl[2 * (size_t)i];
    const float4 li = phl[2 * (size_t)i + 1];
    const float4 vi = pv[2 * (size_t)i + 1];
    const int ti = __float_as_int(pi.w);
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 gi = ST ? gca[i] : zero;
    const float ai = m.a_k[ti];
    const int ns = on ? cnt_short[i] : 0, nl = on ? cnt_all[i] - ns : 0;
    const size_t n = (size_t)m.n;
    const float mu_u = tb.mu[ti * 4 + ti];
    const unsigned self = (unsigned)i << kCodeBits | 13u;  // code 13: the home cell
    float f = 0.f, ck = 0.f;  // lane k < 3: component k of the short part, Kahan
    float g = 0.f;            // ... of the long part
    unsigned in = 0u;
    struct Rec {
        float4 p, v, l, g;
        unsigned code;
    };
    lane_walk<G>(
        list, n, i, ns, self,
        [&](unsigned e) {
            const int j = (int)(e >> kCodeBits);
            Rec r;
            ldg_pv(pv, j, r.p, r.v);
            r.l = __ldg(phl + 2 * (size_t)j + 1);
            r.g = ST ? __ldg(gca + j) : zero;
            r.code = e & 31u;
            return r;
        },
        [&](const Rec& rj, bool have) {
            float d[3], s;
            float3 t;
            const bool hit = have && force_pair_short<ST, RATIO>(m, tb, rj.code, pi, li, vi, ti, mu_u, gi, ai, rj.p,
                                                                 rj.l, rj.v, rj.g, d, s, t);
            if (hit) st[0].v[mine] = make_float4(fmaf(s, d[0], t.x), fmaf(s, d[1], t.y), fmaf(s, d[2], t.z), 0.f);
            in = __ballot_sync(0xffffffffu, hit) >> (lane - sub);
            __syncwarp();
        },
        [&](int) {
            if (sub < 3) {
#pragma unroll
                for (int e = 0; e < G; ++e)
                    if (in >> e & 1u) kahan_add(f, ck, reinterpret_cast<const float*>(&st[0].v[col + e])[sub]);
            }
        });
    struct RecL {
        float4 p, v, g;
        unsigned code;
    };
    lane_walk<G>(
        list + (size_t)m.cap_s * n, n, i, nl, self,
        [&](unsigned e) {
            const int j = (int)(e >> kCodeBits);
            RecL r;
            ldg_pv(pv, j, r.p, r.v);
            r.g = ST ? __ldg(gca + j) : zero;
            r.code = e & 31u;
            return r;
        },
        [&](const RecL& rj, bool have) {
            if (have) {
                float d[3], s;
                float3 t;
                const bool has_t =
                    force_pair_long<ST, RATIO>(m, tb, rj.code, pi, vi, ti, mu_u, gi, ai, rj.p, rj.v, rj.g, d, s, t);
                st[0].v[mine] = make_float4(d[0], d[1], d[2], s);
                if (ST)  // none: -0.0, which leaves a sum as it is
                    st[ST ? 1 : 0].v[mine] = has_t ? make_float4(t.x, t.y, t.z, 0.f) : make_float4(-0.f, -0.f, -0.f, 0.f);
            }
            __syncwarp();
        },
        [&](int mm) {
            if (sub < 3) {
#pragma unroll
                for (int e = 0; e < G; ++e)
                    if (e < mm) {
                        const float* q = reinterpret_cast<const float*>(&st[0].v[col + e]);
                        if (ST) g += reinterpret_cast<const float*>(&st[ST ? 1 : 0].v[col + e])[sub];
                        g = fmaf(q[3], q[sub], g);
                    }
            }
        });
    const double F = ((double)f - (double)ck) + (double)g;
    const int l0 = lane - sub;
    const double F0 = __shfl_sync(0xffffffffu, F, l0), F1 = __shfl_sync(0xffffffffu, F, l0 + 1),
                 F2 = __shfl_sync(0xffffffffu, F, l0 + 2);
    if (sub == 0 && on) force_finish(c, i, ti, F0, F1, F2, vel, vel_out, force, scal);
}

// The force sweep without the long table (MPH_MIXED_CELL_WALK).  One warp per
// home key walks the 3^D stencil in the table build's order (main.cpp:
// 1356-1392), reading each candidate range 32 records at a time (coalesced).
// A lane keeps its candidate when the candidate's hi position lies within
// the largest force radius of the bounding box of the warp's own particles;
// the kept records go to the warp's stage in shared memory (compacted by a
// ballot), and every lane evaluates every kept candidate against its own
// particle, reading the stage with broadcast loads.  Pair terms as in k_mix_b:
// where the hi-only distance is within RP (plus the hi/lo slack) the exact
// hi/lo displacement and Kahan sums, beyond it the hi displacement and plain
// sums.  Then gravity and the FP64 velocity update (main.cpp:1908-2010).  Wall
// keys carry their velocities over (walls never accelerate).
constexpr int kWalkWarps = 4;

struct WalkRec {
    float4 p;  // hi position + the cell offset's hi part (home-relative), type bits
    float4 v;  // velocity, PressureP
    float4 l;  // lo position + the cell offset's lo part, index bits
};

template <bool ST, bool RATIO>
__global__ void __launch_bounds__(32 * kWalkWarps, MPH_WALK_MINB)
k_mix_b_walk(MixConst m, SimConst c, const int* __restrict__ cellstart, const float4* __restrict__ phl,
             const float4* __restrict__ pv, const float4* __restrict__ gca, const double4* __restrict__ vel,
             double4* __restrict__ vel_out, double4* __restrict__ force, StepScalars* __restrict__ scal,
             bool ahead) {
    if (ahead && scal->stop) return;
    __shared__ WalkRec stage_all[kWalkWarps][32];
    __shared__ float4 gstage_all[kWalkWarps][ST ? 32 : 1];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int key = blockIdx.x * kWalkWarps + wib;
    if (key >= 2 * c.tot) return;  // whole warp
    const int hb = cellstart[key], he = cellstart[key + 1];
    if (hb == he) return;
    if (key >= c.tot) {  // wall key
        for (int i = hb + lane; i < he; i += 32) vel_out[i] = vel[i];
        return;
    }
    WalkRec* const stage = stage_all[wib];
    float4* const gstage = gstage_all[wib];
    const int ic[3] = {key / (c.cc[1] * c.cc[2]), (key / c.cc[2]) % c.cc[1], key % c.cc[2]};
    int jmin[3], w[3];
    for (int d = 0; d < 3; ++d) {
        const int r = c.range[d];
        w[d] = 2 * r + 1;
        const int b = (2 * r) - (ic[d] + r) % c.cc[d];
        jmin[d] = b > 0 ? b : 0;
    }
    const float kInf = __int_as_float(0x7f800000);
    for (int h0 = hb; h0 < he; h0 += 32) {
        const int i = h0 + lane;
        const bool act = i < he;
        const int ii = act ? i : hb;
        const float4 pi = phl[2 * (size_t)ii];
        const float4 li = phl[2 * (size_t)ii + 1];
        const float4 vi = pv[2 * (size_t)ii + 1];
        const int ti = __float_as_int(pi.w);
        float4 gi = make_float4(0.f, 0.f, 0.f, 0.f);
        if (ST) gi = gca[ii];
        const float ai = m.a_k[ti];
        const float mu_u = m.visc_mu[ti][ti];
        // bounding box of the chunk's hi positions
        float b0x = act ? pi.x : kInf, b0y = act ? pi.y : kInf, b0z = act ? pi.z : kInf;
        float b1x = act ? pi.x : -kInf, b1y = act ? pi.y : -kInf, b1z = act ? pi.z : -kInf;
        for (int o = 16; o > 0; o >>= 1) {
            b0x = fminf(b0x, __shfl_xor_sync(0xffffffffu, b0x, o));
            b0y = fminf(b0y, __shfl_xor_sync(0xffffffffu, b0y, o));
            b0z = fminf(b0z, __shfl_xor_sync(0xffffffffu, b0z, o));
            b1x = fmaxf(b1x, __shfl_xor_sync(0xffffffffu, b1x, o));
            b1y = fmaxf(b1y, __shfl_xor_sync(0xffffffffu, b1y, o));
            b1z = fmaxf(b1z, __shfl_xor_sync(0xffffffffu, b1z, o));
        }
        float fx = 0.f, fy = 0.f, fz = 0.f, cx = 0.f, cy = 0.f, cz = 0.f;  // within RP: Kahan
        float gx = 0.f, gy = 0.f, gz = 0.f;                                 // beyond
        for (int jx = jmin[0]; jx < jmin[0] + w[0]; ++jx)
            for (int jy = jmin[1]; jy < jmin[1] + w[1]; ++jy)
                for (int jz = jmin[2]; jz < jmin[2] + w[2]; ++jz) {
                    const int ax = jx % w[0], ay = jy % w[1], az = jz % w[2];
                    const int ncx = ((ic[0] - c.range[0] + ax) % c.cc[0] + c.cc[0]) % c.cc[0];
                    const int ncy = ((ic[1] - c.range[1] + ay) % c.cc[1] + c.cc[1]) % c.cc[1];
                    const int ncz = ((ic[2] - c.range[2] + az) % c.cc[2] + c.cc[2]) % c.cc[2];
                    const int cell = ncx * c.cc[1] * c.cc[2] + ncy * c.cc[2] + ncz;
                    const int code = (ax - c.range[0] + 1) * 9 + (ay - c.range[1] + 1) * 3 + (az - c.range[2] + 1);
                    const float dhx = m.dhi[code][0], dhy = m.dhi[code][1], dhz = m.dhi[code][2];
                    const float dlx = m.dlo[code][0], dly = m.dlo[code][1], dlz = m.dlo[code][2];
                    for (int kind = 0; kind < 2; ++kind) {
                        const int off = kind ? c.tot : 0;
                        const int b = cellstart[cell + off], e = cellstart[cell + off + 1];
                        for (int cb = b; cb < e; cb += 32) {
                            const int t = cb + lane;
                            bool keep = false;
                            float4 pj, vj, lj;
                            if (t < e) {
                                ldg_pv(pv, t, pj, vj);
                                lj = phl[2 * (size_t)t + 1];
                                pj.x += dhx;  // exact: both on the hi grid
                                pj.y += dhy;
                                pj.z += dhz;
                                const float ex = fmaxf(0.0f, fmaxf(b0x - pj.x, pj.x - b1x));
                                const float ey = fmaxf(0.0f, fmaxf(b0y - pj.y, pj.y - b1y));
                                const float ez = fmaxf(0.0f, fmaxf(b0z - pj.z, pj.z - b1z));
                                keep = ex * ex + ey * ey + ez * ez < m.walk_r2;
                            }
                            const unsigned kept = __ballot_sync(0xffffffffu, keep);
                            if (keep) {
                                const int slot = __popc(kept & ((1u << lane) - 1u));
                                stage[slot].p = pj;
                                stage[slot].v = vj;
                                stage[slot].l = make_float4(lj.x + dlx, lj.y + dly, lj.z + dlz, __int_as_float(t));
                                if (ST) gstage[slot] = gca[t];
                            }
                            __syncwarp();
                            const int cnt = __popc(kept);
                            if (act) {
                                for (int q = 0; q < cnt; ++q) {
                                    const float4 A = stage[q].p;
                                    const float hx = A.x - pi.x, hy = A.y - pi.y, hz = A.z - pi.z;  // exact
                                    const float r2h = hx * hx + hy * hy + hz * hz;
                                    if (!(r2h < m.walk_r2)) continue;
                                    const float4 L = stage[q].l;
                                    const int j = __float_as_int(L.w);
                                    if (j == i) continue;
                                    const float4 V = stage[q].v;
                                    const int tj = __float_as_int(A.w);
                                    if (r2h < m.walk_short2) {
                                        const float dx = hx + (L.x - li.x);
                                        const float dy = hy + (L.y - li.y);
                                        const float dz = hz + (L.z - li.z);
                                        const float r2 = dx * dx + dy * dy + dz * dz;
                                        if (!(r2 < m.rv2 || r2 < m.rp2 || (ST && (r2 < m.ra2 || r2 < m.rg2)))) continue;
                                        const float rinv = rsqrt_nr(r2);
                                        const float r = r2 * rinv;
                                        float sc = 0.0f;
                                        if (r2 < m.rp2) sc += (vi.w + V.w) * fmaf(m.p_b, r, m.p_a) * rinv;
                                        if (r2 < m.rv2) {
                                            const float mu = m.uniform_mu ? mu_u : m.visc_mu[ti][tj];
                                            const float ud = (V.x - vi.x) * dx + (V.y - vi.y) * dy + (V.z - vi.z) * dz;
                                            sc += mu * ud * fmaf(m.v_b, r, m.v_a) * (rinv * rinv * rinv);
                                        }
                                        float3 tt = make_float3(0.f, 0.f, 0.f);
                                        if (ST) sc += st_terms<RATIO>(m, ti, tj, r2, r, rinv, dx, dy, dz, gi, gstage[q], ai, tt);
                                        kahan_add(fx, cx, fmaf(sc, dx, tt.x));
                                        kahan_add(fy, cy, fmaf(sc, dy, tt.y));
                                        kahan_add(fz, cz, fmaf(sc, dz, tt.z));
                                    } else {
                                        const float rinv = rsqrtf(r2h);
                                        float sc = 0.0f;
                                        if (r2h < m.rv2) {
                                            const float r = r2h * rinv;
                                            const float mu = m.uniform_mu ? mu_u : m.visc_mu[ti][tj];
                                            const float ud = (V.x - vi.x) * hx + (V.y - vi.y) * hy + (V.z - vi.z) * hz;
                                            sc = mu * ud * fmaf(m.v_b, r, m.v_a) * (rinv * rinv * rinv);
                                        }
                                        if (ST) {
                                            if (r2h < m.ra2 || r2h < m.rg2) {
                                                float3 tt = make_float3(0.f, 0.f, 0.f);
                                                sc += st_terms<RATIO>(m, ti, tj, r2h, r2h * rinv, rinv, hx, hy, hz, gi,
                                                                      gstage[q], ai, tt);
                                                gx += tt.x;
                                                gy += tt.y;
                                                gz += tt.z;
                                            }
                                        }
                                        gx = fmaf(sc, hx, gx);
                                        gy = fmaf(sc, hy, gy);
                                        gz = fmaf(sc, hz, gz);
                                    }
                                }
                            }
                            __syncwarp();
                        }
                    }
                }
        if (!act) continue;
        double F0 = ((double)fx - (double)cx) + (double)gx;
        double F1 = ((double)fy - (double)cy) + (double)gy;
        double F2 = ((double)fz - (double)cz) + (double)gz;
        double4 v = vel[i];
        const double mass = c.density[ti] * c.vol;
        F0 += mass * c.gravity[0];
        F1 += mass * c.gravity[1];
        F2 += mass * c.gravity[2];
        v.x += F0 / mass * c.dt;
        v.y += F1 / mass * c.dt;
        v.z += F2 / mass * c.dt;
        if (!(isfinite(v.x) && isfinite(v.y) && isfinite(v.z))) atomicOr(&scal->flags, DEVFLAG_NONFINITE);
        force[i] = make_double4(F0, F1, F2, 0.0);
        vel_out[i] = v;
    }
}

// DensityA over the whole list (output only, without surface tension).
__global__ void k_mix_density_a(MixConst m, const float4* __restrict__ p32, const unsigned* __restrict__ list,
                                const int* __restrict__ cnt_short, const int* __restrict__ cnt_all,
                                double* __restrict__ dens_a_out) {
    __shared__ SharedTables tb;
    load_tables(m, tb);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m.n) return;
    const float4 pi = p32[i];
    const int ti = __float_as_int(pi.w);
    const size_t n = (size_t)m.n;
    float sa = 0.f, ck = 0.f;
    const int ns = cnt_short[i], na = cnt_all[i];
    const uint4* tab = reinterpret_cast<const uint4*>(list) + i;
    auto visit = [&](unsigned e) {
        const int j = (int)(e >> kCodeBits), code = (int)(e & 31u);
        const float4 pj = p32[j];
        const float4 dh = tb.dhi[code];
        const float dx = (pj.x - pi.x) + dh.x, dy = (pj.y - pi.y) + dh.y, dz = (pj.z - pi.z) + dh.z;
        const float r2 = dx * dx + dy * dy + dz * dz;
        if (r2 <= m.ra2) {
            const float r = sqrtf(r2);
            const float q = r * m.inv_ra;
            const float ratio = m.ratio_all_one ? 1.0f : m.ratio[ti][__float_as_int(pj.w)];
            kahan_add(sa, ck, ratio * m.ca * q * (1.0f - q) * (1.0f - q));
        }
    };
    for_entries(tab, n, ns, visit);
    for_entries(tab + (size_t)(m.cap_s >> 2) * n, n, na - ns, visit);
    dens_a_out[i] = sa - ck;
}

// Virial pressure at particles for the mixed forms (output only; the FP64
// form's k_virial restates main.cpp:2057-2302).  Only the trace of the pair
// stress enters VirialPressureAtParticle = -trace / D, so each term reduces to
// a scalar per pair (x = x_j - x_i, r = |x|, e = x / r):
//   PressureP  (r < RP): P_i dwpdr(r) r
//   PressureA  (r < RA): PA_i ratio_ij dwadr(r) r
//   ViscosityV (r < RV): 0.5 C mu_ij (u_ij . e) (-dwvdr(r))
//   DiffuseInterface (r < RG): a_i (GC_i . x) ratio_ij (wg + dwgdr r) Rg / R2g / l0
// in FP32 on the exact cell-relative displacement, Kahan-compensated, with
// the velocities after the step (the reference calls it after
// calculateAcceleration, main.cpp:432-435).
template <bool ST, bool RATIO>
__global__ void __launch_bounds__(128)
k_mix_virial(MixConst m, const float4* __restrict__ phl, const float4* __restrict__ pv,
             const float4* __restrict__ gca, const double4* __restrict__ vel, const unsigned* __restrict__ list,
             const int* __restrict__ cnt_short, const int* __restrict__ cnt_all, double* __restrict__ virial) {
    __shared__ SharedTables tb;
    load_tables(m, tb);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m.n) return;
    const float4 pi = phl[2 * (size_t)i];
    const float4 li = phl[2 * (size_t)i + 1];
    const int ti = __float_as_int(pi.w);
    const float ppi = pv[2 * (size_t)i + 1].w;
    const float4 gi = ST ? gca[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    const double4 vd = vel[i];
    const float vix = (float)vd.x, viy = (float)vd.y, viz = (float)vd.z;
    const float ai = m.a_k[ti];
    const float inv_l0 = 1.0f / m.l0;
    const size_t n = (size_t)m.n;
    float tr = 0.f, ck = 0.f;
    auto visit = [&](unsigned e) {
        const int j = (int)(e >> kCodeBits), code = (int)(e & 31u);
        const float4 pj = phl[2 * (size_t)j];
        const float4 lj = phl[2 * (size_t)j + 1];
        const float4 dh = tb.dhi[code], dl = tb.dlo[code];
        const float dx = ((pj.x - pi.x) + dh.x) + ((lj.x - li.x) + dl.x);
        const float dy = ((pj.y - pi.y) + dh.y) + ((lj.y - li.y) + dl.y);
        const float dz = ((pj.z - pi.z) + dh.z) + ((lj.z - li.z) + dl.z);
        const float r2 = dx * dx + dy * dy + dz * dz;
        if (!(r2 < m.rv2 || r2 < m.rp2 || (ST && (r2 < m.ra2 || r2 < m.rg2)))) return;
        const float r = sqrtf(r2);
        const int tj = __float_as_int(pj.w);
        const float ratio = RATIO ? m.ratio[ti][tj] : 1.0f;
        float t = 0.f;
        if (r2 < m.rp2) t += ppi * (m.cp_m2 * (1.0f - r * m.inv_rp)) * r;
        if (ST && r2 < m.ra2) {
            const float q = r * m.inv_ra;
            t += gi.w * ratio * (m.ca_inv * (1.0f - q) * (1.0f - 3.0f * q)) * r;
        }
        if (r2 < m.rv2) {
            const double4 vj = vel[j];
            const float ue = (((float)vj.x - vix) * dx + ((float)vj.y - viy) * dy + ((float)vj.z - viz) * dz) / r;
            t += 0.5f * tb.mu[ti * 4 + tj] * ue * (-(m.cv_m2 * (1.0f - r * m.inv_rv)));
        }
        if (ST && r2 < m.rg2) {
            const float q = 1.0f - r * m.inv_rg;
            const float gx = gi.x * dx + gi.y * dy + gi.z * dz;
            t += ai * gx * ratio * (m.cg * q * q + m.cg_m2 * q * r) * m.inv_r2g_rg * inv_l0;
        }
        kahan_add(tr, ck, t);
    };
    const uint4* tab = reinterpret_cast<const uint4*>(list) + i;
    const int ns = cnt_short[i], na = cnt_all[i];
    for_entries(tab, n, ns, visit);
    for_entries(tab + (size_t)(m.cap_s >> 2) * n, n, na - ns, visit);
    virial[i] = -((double)tr - (double)ck) / (double)m.dim;
}

// NeighborCount for output: the list counts plus self (the reference lists
// self), except walls without a fluid neighbour, whose list is empty there
// (main.cpp:1416).
__global__ void k_mix_counts(int n, const int* __restrict__ cnt_all, const int* __restrict__ cellstart, int tot,
                             int* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int c = cnt_all[i];
    out[i] = c > 0 ? c + 1 : (i < cellstart[tot] ? 1 : 0);
}

inline int blocks(long long n, int t) { return (int)((n + t - 1) / t); }

}  // namespace

struct MixedState {
    MixConst mc;
    int* keys_unsorted = nullptr;
    int* slot = nullptr;
    int* counts = nullptr;
    int* sums = nullptr;  // of the scan's blocks, behind counts
    int* tmp = nullptr;
    int* home = nullptr;
    float4* phl = nullptr;  // [2n]: {hi position + type, lo position} per particle (home-cell relative)
    float4* p32 = nullptr;  // [n]: the hi parts alone, for the table build
    float4* v32 = nullptr;
    float4* pv = nullptr;  // [2n]: {hi position + type, (v, PressureP)} per particle, written by sweep A
    float4* gca = nullptr;
    unsigned* list = nullptr;
    int cap = 0;          // cap_s + cap_l rows
    int cap_l = 0;        // rows of the long part (mc.cap_s: the short part)
    int max_short = 0, max_long = 0;
    int* cnt_short = nullptr;
    int* cnt_all = nullptr;
    StepScalars* h_scal = nullptr;
    int max_neighbors = 0;
    int n_fluid = 0;
    bool exported = false;
    bool s64 = false;  // FP64 pressure core (MPH_MODE_MIXED_P64)
    bool walk = false; // force sweep by cell walk (MPH_MIXED_CELL_WALK)
};

static void mfree(MixedState* m) {
    void* ptrs[] = {m->keys_unsorted, m->slot, m->counts, m->tmp, m->home, m->phl, m->p32, m->v32, m->pv,
                    m->gca, m->list, m->cnt_short, m->cnt_all};
    for (void* p : ptrs)
        if (p) cudaFree(p);
    if (m->h_scal) cudaFreeHost(m->h_scal);
}

#define MTRY(expr)                                                                     \
    do {                                                                               \
        cudaError_t e_ = (expr);                                                       \
        if (e_ != cudaSuccess) {                                                       \
            if (err) *err = std::string(#expr ": ") + cudaGetErrorString(e_);          \
            return MPH_ERR_CUDA;                                                       \
        }                                                                              \
    } while (0)

template <class T>
static cudaError_t malloc_n(T** p, size_t n) {
    return cudaMalloc((void**)p, (n ? n : 1) * sizeof(T));
}

static int grow_list(MixedState* m, int need_s, int need_l, int n, std::string* err) {
    const int cs = ((int)(need_s * 1.15) + 8 + 7) / 8 * 8, cl = ((int)(need_l * 1.15) + 8 + 7) / 8 * 8;
    if (m->list) cudaFree(m->list);
    m->list = nullptr;
    m->cap = m->cap_l = m->mc.cap_s = 0;
    MTRY(malloc_n(&m->list, (size_t)(cs + cl) * (size_t)n));
    m->mc.cap_s = cs;
    m->cap_l = cl;
    m->cap = cs + cl;
    return MPH_OK;
}

// Counting sort by cell, reorder the FP64 state, home cells, list build.
int mixed_rebuild(MixedState* m, const SimConst& c, DevFP64& d, cudaStream_t s, std::string* err, int* launches) {
    const int n = c.n, nb = 2 * c.tot;
    const int a = d.cur, b = 1 - d.cur, va = d.vcur, vb = 1 - d.vcur;
    int nl = 0;
    MTRY(cudaMemsetAsync(m->counts, 0, sizeof(int) * (size_t)(nb + 1), s));
    k_mix_cellkey<<<blocks(n, 256), 256, 0, s>>>(c, d.pos[a], m->keys_unsorted, m->slot, m->counts);
    k_mix_scan_sums<<<blocks(nb + 1, kScanKeys), kScanThreads, 0, s>>>(m->counts, nb, m->sums);
    k_mix_scan<<<blocks(nb + 1, kScanKeys), kScanThreads, 0, s>>>(m->counts, nb, m->sums, d.cellstart);
    k_mix_place<<<blocks(n, 256), 256, 0, s>>>(n, m->keys_unsorted, m->slot, d.cellstart, m->tmp);
    k_mix_rank<<<blocks(n, 256), 256, 0, s>>>(n, m->keys_unsorted, d.cellstart, m->tmp, d.vals, d.keys);
    launch_reorder(c, d.vals, d.pidx[a], d.type[a], d.pos[a], d.vel[va], d.pidx[b], d.type[b], d.pos[b], d.vel[vb],
                   nullptr, d.snap, s);
    d.cur = b;
    d.vcur = vb;
    k_mix_home<<<blocks(n, 256), 256, 0, s>>>(c, m->mc, d.pos[d.cur], d.keys, d.vel[d.vcur], m->home, m->phl,
                                              m->p32, m->v32);
    nl += 7;
    for (int attempt = 0; attempt < 3; ++attempt) {
        MTRY(cudaMemsetAsync(&d.scal->max_neighbors, 0, sizeof(int), s));
        MTRY(cudaMemsetAsync(&d.scal->max_short, 0, 2 * sizeof(int), s));
        const int key_warps = list_key_warps(c.dim, n, c.tot);
        k_mix_list<<<blocks(2LL * c.tot * key_warps, kListWarps), 32 * kListWarps, 0, s>>>(
            c, m->mc, m->p32, d.cellstart, m->list, m->cap_l, m->cnt_short, m->cnt_all, d.scal, key_warps);
        ++nl;
        MTRY(cudaGetLastError());
        MTRY(cudaMemcpyAsync(m->h_scal, d.scal, sizeof(StepScalars), cudaMemcpyDeviceToHost, s));
        MTRY(cudaStreamSynchronize(s));
        m->max_neighbors = m->h_scal->max_neighbors;
        m->max_short = m->h_scal->max_short;
        m->max_long = m->h_scal->max_long;
        if (m->max_short <= m->mc.cap_s && m->max_long <= m->cap_l) break;
        const int st = grow_list(m, std::max(m->max_short, m->mc.cap_s), std::max(m->max_long, m->cap_l), n, err);
        if (st != MPH_OK) return st;
    }
    if (launches) *launches = nl;
    if (m->max_short > m->mc.cap_s || m->max_long > m->cap_l) {
        if (err) *err = "mixed neighbour table could not grow";
        return MPH_ERR_CAPACITY;
    }
    MTRY(cudaMemsetAsync(&d.scal->flags, 0, sizeof(int), s));
    m->exported = false;
    return MPH_OK;
}

// Lanes per particle of a sweep: enough threads to fill the GPU, and no more (the
// ordered sums cost more than one thread's walk then).  us at 1, 4, 8 lanes (a particle's
// list: 40 entries in 2-D and in sweep A without surface tension, else 200):
//   2-D, sweep A / B         1,600   23 / 17 / 15   28 / 13 / 11
//                           12,100   23 / 17 / 15   27 / 15 / 15
//                           16,900   23 / 19 / 21   29 / 16 / 19
//                           32,400   25 / 22 / 27   31 / 24 / 25
//                           46,225   23 / 26 / 30   31 / 27 / 33
//                           57,600   25 / 30 / 37   33 / 33 / 37
//   3-D, sweep A, no surface tension, 13,320 particles  23 / 17 / 17; 27,936  22 / 16 / 17;
//                           45,561   24 / 19 / 23; 58,848  23 / 24 / 26
//   3-D, sweep A, surface tension, 8,000   59 / 32 / 26; 13,824  62 / 34 / 30;
//                           32,768   66 / 48 / 61; 64,000  66 / 82 / 104
//   3-D, sweep B, 2,304 fluid  55 / 21 / 17; 9,600  56 / 26 / 23; 14,283  58 / 27 / 28;
//                           36,864   60 / 54 / 51; 60,648  70 / 69 / 79; 75,645  80 / 91 / 95
//   same with surface tension, 8,000  99 / 29 / 25; 21,952  103 / 50 / 48;
//                           85,184   - / 134 / 152; 125,000  237 / 195 / 217; 262,144  372 / 385 / 438
// Sixteen lanes win 1 or 2 us below 5,000 particles alone.
static int lanes_for(const SimConst& c, int n, int eight, int four) {
    if (c.sweep_layout) return c.sweep_layout == 1 ? 1 : 8;  // mph_set_sweep_layout
    return n <= eight ? 8 : n <= four ? 4 : 1;
}
static int lanes_a(const MixedState* m, const SimConst& c) {
    if (m->mc.dim == 2) return lanes_for(c, m->mc.n, 14000, 35000);
    return m->mc.has_st ? lanes_for(c, m->mc.n, 20000, 48000) : lanes_for(c, m->mc.n, 14000, 50000);
}
static int lanes_b(const MixedState* m, const SimConst& c) {
    if (m->mc.dim == 2) return lanes_for(c, m->n_fluid, 12000, 50000);
    return m->mc.has_st ? lanes_for(c, m->n_fluid, 25000, 150000) : lanes_for(c, m->n_fluid, 12000, 62000);
}

void mixed_sweep_a(MixedState* m, const SimConst& c, DevFP64& d, bool advance_wall, cudaStream_t s, bool ahead) {
    const int g = lanes_a(m, c), nb = blocks((long long)c.n * g, 128);
    double* wc = advance_wall ? d.wall_center : nullptr;
#define MIX_A(KERNEL)                                                                                               \
    KERNEL<<<nb, 128, 0, s>>>(m->mc, m->phl, m->p32, m->v32, m->list, m->cnt_short, m->cnt_all, m->pv, m->gca,      \
                              d.strain_p, d.div_p, d.dens_a, wc, c, d.vel[d.vcur], d.press, ahead ? d.scal : nullptr)
#define MIX_A3(ST, RATIO, S64)                                  \
    if (g == 1) MIX_A((k_mix_a<ST, RATIO, S64>));               \
    else if (g == 4) MIX_A((k_mix_a_g<ST, RATIO, S64, 4>));     \
    else MIX_A((k_mix_a_g<ST, RATIO, S64, 8>))
#define MIX_A2(ST, RATIO) \
    if (m->s64) { MIX_A3(ST, RATIO, true); } else { MIX_A3(ST, RATIO, false); }
    if (!m->mc.has_st) { MIX_A2(false, false); }  // the ratios weigh surface-tension sums alone
    else if (m->mc.ratio_all_one) { MIX_A2(true, false); }
    else { MIX_A2(true, true); }
#undef MIX_A2
#undef MIX_A3
#undef MIX_A
    m->exported = false;
}

template <bool WALLS>
static void launch_b(MixedState* m, const SimConst& c, DevFP64& d, cudaStream_t s, bool ahead) {
    const int g = WALLS ? 1 : lanes_b(m, c);
    if (g > 1) {
        const int gb = blocks((long long)m->n_fluid * g, 128), nw = gb + blocks(c.n - m->n_fluid, 128);
#define MIX_BG(ST, RATIO, G)                                                                                        \
    k_mix_b_g<ST, RATIO, G><<<nw, 128, 0, s>>>(m->mc, c, m->n_fluid, gb, m->phl, m->pv, m->gca, m->list,          \
                                               m->cnt_short, m->cnt_all, d.vel[d.vcur], d.vel[1 - d.vcur], d.force, \
                                               d.scal, ahead)
#define MIX_BG2(ST, RATIO)               \
    if (g == 4) MIX_BG(ST, RATIO, 4);    \
    else MIX_BG(ST, RATIO, 8)
        if (!m->mc.has_st) { MIX_BG2(false, false); }
        else if (m->mc.ratio_all_one) { MIX_BG2(true, false); }
        else { MIX_BG2(true, true); }
#undef MIX_BG2
#undef MIX_BG
        return;
    }
    const int nb = blocks(c.n, 128);
    double4* vout = WALLS ? nullptr : d.vel[1 - d.vcur];
#define MIX_B(ST, RATIO)                                                                                            \
    k_mix_b<ST, RATIO, WALLS><<<nb, 128, 0, s>>>(m->mc, c, d.cellstart, m->phl, m->pv, m->gca, m->list,           \
                                                 m->cnt_short, m->cnt_all, d.vel[d.vcur], vout, d.force, d.scal, ahead)
    if (!m->mc.has_st) MIX_B(false, false);
    else if (m->mc.ratio_all_one) MIX_B(true, false);
    else MIX_B(true, true);
#undef MIX_B
}

static void launch_b_walk(MixedState* m, const SimConst& c, DevFP64& d, cudaStream_t s, bool ahead) {
    const int nb = (2 * c.tot + kWalkWarps - 1) / kWalkWarps;
#define MIX_W(ST, RATIO)                                                                                      \
    k_mix_b_walk<ST, RATIO><<<nb, 32 * kWalkWarps, 0, s>>>(m->mc, c, d.cellstart, m->phl, m->pv, m->gca,    \
                                                          d.vel[d.vcur], d.vel[1 - d.vcur], d.force, d.scal, ahead)
    if (m->mc.has_st) {
        if (m->mc.ratio_all_one) { MIX_W(true, false); } else { MIX_W(true, true); }
    } else {
        if (m->mc.ratio_all_one) { MIX_W(false, false); } else { MIX_W(false, true); }
    }
#undef MIX_W
}

int mixed_sweep_b(MixedState* m, const SimConst& c, DevFP64& d, cudaStream_t s, bool ahead) {
    if (m->walk) launch_b_walk(m, c, d, s, ahead);
    else launch_b<false>(m, c, d, s, ahead);
    m->exported = false;
    return 1;
}

void mixed_set_cell_walk(MixedState* m, bool on) { m->walk = on; }

void mixed_move(MixedState* m, const SimConst& c, DevFP64& d, cudaStream_t s, bool ahead) {
    const int nb = blocks(c.n, 256);
    if (ahead)
        k_mix_move<true><<<nb, 256, 0, s>>>(c, m->mc, d.cellstart, d.pos[d.cur], d.vel[d.vcur], d.snap, d.wall_center,
                                            m->home, m->phl, m->p32, m->v32, d.scal);
    else
        k_mix_move<false><<<nb, 256, 0, s>>>(c, m->mc, d.cellstart, d.pos[d.cur], d.vel[d.vcur], d.snap, d.wall_center,
                                             m->home, m->phl, m->p32, m->v32, d.scal);
    m->exported = false;
}

int mixed_create(MixedState** out, const SimConst& c, const mph_constants& k, DevFP64& d, int n_fluid,
                 bool fp64_pressure, cudaStream_t s, std::string* err) {
    *out = nullptr;
    if (c.cc[0] > 1024 || c.cc[1] > 1024 || c.cc[2] > 1024) {
        if (err) *err = "mixed form: at most 1024 cells per axis";
        return MPH_ERR_GEOMETRY;
    }
    if ((long long)c.n >= (1LL << (32 - kCodeBits))) {
        if (err) *err = "mixed form: too many particles for the packed list";
        return MPH_ERR_ARG;
    }
    MixedState* m = new MixedState();
    m->s64 = fp64_pressure;
    m->n_fluid = n_fluid;
    MixConst& mc = m->mc;
    std::memset(&mc, 0, sizeof(mc));
    mc.n = c.n;
    mc.tot = c.tot;
    mc.dim = c.dim;
    mc.has_st = c.has_st;
    mc.ratio_all_one = c.ratio_all_one;
    for (int dd = 0; dd < 3; ++dd) {
        mc.cc[dd] = c.cc[dd];
        mc.range[dd] = c.range[dd];
    }
    // hi-part grid: a power of two g with 2.2 cell widths below 2^24 g
    const double cwmax = std::max(c.cell_width[0], std::max(c.cell_width[1], c.cell_width[2]));
    mc.grid = std::ldexp(1.0, (int)std::ceil(std::log2(2.2 * cwmax)) - 24);
    mc.inv_grid = 1.0 / mc.grid;
    for (int code = 0; code < 27; ++code) {
        const int dc[3] = {code / 9 - 1, (code / 3) % 3 - 1, code % 3 - 1};
        for (int dd = 0; dd < 3; ++dd) {
            const double off = dc[dd] * c.cell_width[dd];
            const double q = std::rint(off * mc.inv_grid) * mc.grid;
            mc.dhi[code][dd] = (float)q;
            mc.dlo[code][dd] = (float)(off - q);
        }
        mc.dhi[code][3] = mc.dlo[code][3] = 0.0f;
    }
    const int one[3] = {22, 16, 14};  // the codes of one cell up along x, y, z
    for (int dd = 0; dd < 3; ++dd) mc.half_cell[dd] = 0.5f * mc.dhi[one[dd]][dd];
    mc.uniform_mu = 1;
    for (int t = 0; t < MPH_TYPE_COUNT; ++t)
        for (int u = 0; u < MPH_TYPE_COUNT; ++u)
            if (c.visc_mu[t][u] != c.visc_mu[0][0]) mc.uniform_mu = 0;
    const double margin = 0.1 * c.l0;
    const double rl = k.max_radius + margin, rs = k.radius_p + margin;
    mc.list_r2 = (float)(rl * rl);
    mc.short_r2 = (float)(rs * rs);
    {
        // the hi-only distance is within 3 * 1.5 grid steps of the exact one
        // (the lo parts of both particles and of the cell offset): 8 steps of slack
        double rf = std::max(c.rv, c.rp);
        if (c.has_st) rf = std::max(rf, std::max(c.ra, c.rg));
        const double sl = 8.0 * mc.grid;
        mc.walk_r2 = (float)((rf + sl) * (rf + sl));
        mc.walk_short2 = (float)((c.rp + sl) * (c.rp + sl));
    }
    mc.ra2 = (float)c.ra2;
    mc.rp2 = (float)c.rp2;
    mc.rv2 = (float)c.rv2;
    mc.rg2 = (float)c.rg2;
    mc.inv_ra = (float)(1.0 / c.ra);
    mc.inv_rp = (float)(1.0 / c.rp);
    mc.inv_rv = (float)(1.0 / c.rv);
    mc.inv_rg = (float)(1.0 / c.rg);
    mc.ca = (float)c.ca;
    mc.cp = (float)c.cp;
    mc.cg = (float)c.cg;
    mc.cv = (float)c.cv;
    mc.cp_m2 = (float)(c.cp * c.m2_rp);
    mc.cg_m2 = (float)(c.cg * c.m2_rg);
    mc.cv_m2 = (float)(c.cv * c.m2_rv);
    mc.ca_inv = (float)(c.ca * c.inv_ra);
    mc.p_a = (float)(c.cp * c.m2_rp * c.vol);
    mc.p_b = (float)(-c.cp * c.m2_rp * c.vol / c.rp);
    mc.v_a = (float)(-c.cv * c.m2_rv * c.vol);
    mc.v_b = (float)(c.cv * c.m2_rv * c.vol / c.rv);
    mc.p_a_d = c.cp * c.m2_rp * c.vol;
    mc.p_b_d = -c.cp * c.m2_rp * c.vol / c.rp;
    mc.v_a_d = -c.cv * c.m2_rv * c.vol;
    mc.v_b_d = c.cv * c.m2_rv * c.vol / c.rv;
    mc.cp_d = c.cp;
    mc.cp_m2_d = c.cp * c.m2_rp;
    mc.inv_rp_d = 1.0 / c.rp;
    mc.n0p_d = c.n0p;
    mc.inv_rp_lo = (float)(1.0 / c.rp - (double)mc.inv_rp);
    mc.cp_lo = (float)(c.cp - (double)mc.cp);
    mc.vol = (float)c.vol;
    mc.vol_over_l0 = (float)c.vol_over_l0;
    mc.n0a = (float)c.n0a;
    mc.n0p = (float)c.n0p;
    mc.inv_r2g_rg = (float)(c.rg / c.r2g);
    mc.l0 = (float)c.l0;
    for (int t = 0; t < MPH_TYPE_COUNT; ++t) {
        mc.a_k[t] = (float)c.a_k[t];
        mc.cof_a[t] = (float)c.cof_a[t];
        mc.bulk_modulus[t] = (float)c.bulk_modulus[t];
        mc.bulk_viscosity[t] = (float)c.bulk_viscosity[t];
        for (int u = 0; u < MPH_TYPE_COUNT; ++u) {
            mc.visc_mu[t][u] = (float)c.visc_mu[t][u];
            mc.ratio[t][u] = (float)c.ratio[t][u];
        }
    }
    const size_t n = (size_t)c.n;
    cudaError_t e = cudaSuccess;
    if (e == cudaSuccess) e = malloc_n(&m->keys_unsorted, n);
    if (e == cudaSuccess) e = malloc_n(&m->slot, n);
    if (e == cudaSuccess) e = malloc_n(&m->counts, 2 * (size_t)c.tot + 1 + blocks(2LL * c.tot + 1, kScanKeys));
    if (e == cudaSuccess) m->sums = m->counts + 2 * (size_t)c.tot + 1;
    if (e == cudaSuccess) e = malloc_n(&m->tmp, n);
    if (e == cudaSuccess) e = malloc_n(&m->home, n);
    if (e == cudaSuccess) e = malloc_n(&m->phl, 2 * n);
    if (e == cudaSuccess) e = malloc_n(&m->p32, n);
    if (e == cudaSuccess) e = malloc_n(&m->v32, n);
    if (e == cudaSuccess) e = malloc_n(&m->pv, 2 * n);
    if (e == cudaSuccess) e = malloc_n(&m->gca, n);
    if (e == cudaSuccess) e = malloc_n(&m->cnt_short, n);
    if (e == cudaSuccess) e = malloc_n(&m->cnt_all, n);
    if (e == cudaSuccess) e = cudaMallocHost((void**)&m->h_scal, sizeof(StepScalars));
    if (e == cudaSuccess) e = cudaMemsetAsync(m->gca, 0, n * sizeof(float4), s);
    if (e != cudaSuccess) {
        if (err) *err = std::string("mixed form allocation: ") + cudaGetErrorString(e);
        mfree(m);
        delete m;
        return MPH_ERR_NOMEM;
    }
    // initial table: lattice points within the short and the long cut-off, with head room
    const double ratio = rl / c.l0, rs_l0 = rs / c.l0;
    const int r = (int)ratio + 1, zr = c.dim == 2 ? 0 : r;
    int lat_s = 0, lat_l = 0;
    for (int x = -r; x <= r; ++x)
        for (int y = -r; y <= r; ++y)
            for (int z = -zr; z <= zr; ++z) {
                const double q2 = x * x + y * y + z * z;
                if (q2 <= rs_l0 * rs_l0) ++lat_s;
                else if (q2 <= ratio * ratio) ++lat_l;
            }
    int st = grow_list(m, (int)(lat_s * 1.1) + 4, (int)(lat_l * 1.1) + 8, c.n, err);
    if (st == MPH_OK) st = mixed_rebuild(m, c, d, s, err, nullptr);
    if (st == MPH_OK) {
        mixed_sweep_a(m, c, d, false, s, false);
        e = cudaGetLastError();
        if (e != cudaSuccess) {
            if (err) *err = cudaGetErrorString(e);
            st = MPH_ERR_CUDA;
        }
    }
    if (st != MPH_OK) {
        mfree(m);
        delete m;
        return st;
    }
    *out = m;
    return MPH_OK;
}

int mixed_export(MixedState* m, const SimConst& c, DevFP64& d, cudaStream_t s, std::string* err, int* launches) {
    int nl = 0;
    if (!m->exported) {
        if (!m->mc.has_st) {
            k_mix_density_a<<<blocks(c.n, 128), 128, 0, s>>>(m->mc, m->p32, m->list, m->cnt_short, m->cnt_all,
                                                               d.dens_a);
            ++nl;
        }
        launch_b<true>(m, c, d, s, false);  // wall forces
        k_mix_counts<<<blocks(c.n, 256), 256, 0, s>>>(c.n, m->cnt_all, d.cellstart, c.tot, d.ncount);
        nl += 2;
        MTRY(cudaGetLastError());
        m->exported = true;
    }
    if (launches) *launches = nl;
    return MPH_OK;
}

int mixed_virial(MixedState* m, const SimConst& c, DevFP64& d, cudaStream_t s, std::string* err) {
    const int nb = blocks(c.n, 128);
#define MIX_V(ST, RATIO)                                                                                    \
    k_mix_virial<ST, RATIO><<<nb, 128, 0, s>>>(m->mc, m->phl, m->pv, m->gca, d.vel[d.vcur], m->list,        \
                                               m->cnt_short, m->cnt_all, d.virial_p)
    if (m->mc.has_st) {
        if (m->mc.ratio_all_one) { MIX_V(true, false); } else { MIX_V(true, true); }
    } else {
        if (m->mc.ratio_all_one) { MIX_V(false, false); } else { MIX_V(false, true); }
    }
#undef MIX_V
    MTRY(cudaGetLastError());
    return MPH_OK;
}

int mixed_import(MixedState* m, const SimConst& c, DevFP64& d, cudaStream_t s, std::string* err) {
    // positions/velocities changed from the host: refresh the FP32 copies
    k_mix_home<<<blocks(c.n, 256), 256, 0, s>>>(c, m->mc, d.pos[d.cur], d.keys, d.vel[d.vcur], m->home, m->phl,
                                                m->p32, m->v32);
    MTRY(cudaGetLastError());
    m->exported = false;
    return MPH_OK;
}

void mixed_mark_stale(MixedState* m) { m->exported = false; }
int mixed_max_neighbors(const MixedState* m) { return m ? m->max_neighbors : 0; }
int mixed_capacity(const MixedState* m) { return m ? m->cap : 0; }

void mixed_destroy(MixedState* m) {
    if (!m) return;
    mfree(m);
    delete m;
}

}  // namespace mph
