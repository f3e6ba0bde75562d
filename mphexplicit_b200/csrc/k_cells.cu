// k_cells.cu — cell assignment, bitonic cell sort, per-cell ranges, reorder and
// the Verlet neighbour list of the FP64 form (sm_100a).
//
// This is integer/index work plus the FP64 distance test of the list build.
// The results are bit-exact against the reference:
//   * cell index:      main.cpp:1115-1133 (same floor/modulo expressions);
//   * sort:            the reference's bitonic compare-exchange network
//                      (main.cpp:1137-1158), pass for pass, so ties inside a
//                      cell end in the same order and the permutation matches;
//   * per-cell ranges: main.cpp:1160-1247 (begin/end equal the number of sorted
//                      keys below each key value, found here by binary search);
//   * neighbour list:  main.cpp:1329-1596, same stencil order, self included,
//                      wall particles without a fluid neighbour get no list.
// Compiled with -fmad=false so the distance test is not FMA-contracted.
#include <cmath>
#include "mph_internal.h"

namespace mph {

namespace {

constexpr int kLogLocal = 12;               // 4096 keys per shared-memory block
constexpr int kLocal = 1 << kLogLocal;
constexpr int kSortThreads = 1024;

__device__ __forceinline__ double omod(double x, double w) { return x - w * floor(x / w); }

// Mod(x,w) of main.cpp:70.  When 0 <= x < 0.75 w the quotient rounds below 1,
// floor gives +0 and the expression returns x exactly; skip the division then.
__device__ __forceinline__ double omod_fast(double x, double w) {
    return (x >= 0.0 && x < 0.75 * w) ? x : omod(x, w);
}

__device__ __forceinline__ int cell_id(const SimConst& c, int ix, int iy, int iz) {  // main.cpp:96-100
    return ((ix % c.cc[0] + c.cc[0]) % c.cc[0]) * c.cc[1] * c.cc[2] +
           ((iy % c.cc[1] + c.cc[1]) % c.cc[1]) * c.cc[2] + ((iz % c.cc[2] + c.cc[2]) % c.cc[2]);
}

__global__ void k_cell_index(SimConst c, const double4* __restrict__ pos, const int* __restrict__ type,
                             int* __restrict__ keys, int* __restrict__ vals) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.pow2) return;
    if (i < c.n) {
        const double4 p = pos[i];
        const int cx = ((int)floor((p.x - c.dmin[0]) / c.cell_width[0])) % c.cc[0];
        const int cy = ((int)floor((p.y - c.dmin[1]) / c.cell_width[1])) % c.cc[1];
        const int cz = ((int)floor((p.z - c.dmin[2]) / c.cell_width[2])) % c.cc[2];
        int id = cell_id(c, cx, cy, cz);
        const int t = type[i];
        if (t >= 2 && t < 4) id += c.tot;
        keys[i] = id;
        vals[i] = i;
    } else {
        keys[i] = 2 * c.tot;
        vals[i] = c.n;
    }
}

// One compare-exchange of pass (m, dist): element i (bit log2(dist) clear) and
// i|dist; ascending when bit m+1 of i is clear (main.cpp:1146-1148).
__device__ __forceinline__ void cmpx(int* k, int* v, int a, int b, bool up) {
    const int ka = k[a], kb = k[b];
    if ((ka > kb) == up) {
        const int va = v[a], vb = v[b];
        k[a] = kb; k[b] = ka;
        v[a] = vb; v[b] = va;
    }
}

// All passes whose distance is below the block size, for main-stage m in
// [m_begin, m_end); for each m the sub-stages with dist < block run here.
// Block b owns keys [b*L, (b+1)*L).
__global__ void __launch_bounds__(kSortThreads)
k_bitonic_local(int* __restrict__ keys, int* __restrict__ vals, int L, int logL, int m_begin, int m_end) {
    __shared__ int sk[kLocal];
    __shared__ int sv[kLocal];
    const int base = blockIdx.x * L;
    for (int t = threadIdx.x; t < L; t += blockDim.x) {
        sk[t] = keys[base + t];
        sv[t] = vals[base + t];
    }
    __syncthreads();
    const int half = L >> 1;
    for (int m = m_begin; m < m_end; ++m) {
        // sub-stages with dist = 2^(m-k) < L, i.e. log2(dist) <= min(m, logL-1)
        const int top = m < logL - 1 ? m : logL - 1;
        for (int ld = top; ld >= 0; --ld) {
            const int dist = 1 << ld;
            for (int t = threadIdx.x; t < half; t += blockDim.x) {
                const int i = ((t >> ld) << (ld + 1)) | (t & (dist - 1));
                const bool up = (((base + i) >> m) & 2) == 0;
                cmpx(sk, sv, i, i | dist, up);
            }
            __syncthreads();
        }
    }
    for (int t = threadIdx.x; t < L; t += blockDim.x) {
        keys[base + t] = sk[t];
        vals[base + t] = sv[t];
    }
}

// One pass with dist >= block size, one pair per thread.
__global__ void k_bitonic_global(int* __restrict__ keys, int* __restrict__ vals, int npairs, int m, int ld) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= npairs) return;
    const int dist = 1 << ld;
    const int i = ((t >> ld) << (ld + 1)) | (t & (dist - 1));
    const bool up = ((i >> m) & 2) == 0;
    cmpx(keys, vals, i, i | dist, up);
}

// cellstart[b] = number of sorted keys below b, b in [0, 2*tot].  These are
// the reference's CellFluidParticleBegin/End (b < tot) and
// CellWallParticleBegin/End (b >= tot) after its prefix sum (main.cpp:1191-1247).
__global__ void k_cell_ranges(const int* __restrict__ keys, int n, int nb, int* __restrict__ cellstart) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nb) return;
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (keys[mid] < b) lo = mid + 1; else hi = mid;
    }
    cellstart[b] = lo;
}

// Gather by the sorted CellParticle (main.cpp:1262-1325); the snapshot of the
// positions for the rebuild test is taken here (main.cpp:1587-1595: the
// positions do not change between the reorder and the end of the build).
__global__ void k_reorder(int n, const int* __restrict__ vals, const int* __restrict__ pidx_in,
                          const int* __restrict__ type_in, const double4* __restrict__ pos_in,
                          const double4* __restrict__ vel_in, int* __restrict__ pidx_out,
                          int* __restrict__ type_out, double4* __restrict__ pos_out,
                          double4* __restrict__ vel_out, double2* __restrict__ xv, double4* __restrict__ snap) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int s = vals[i];
    pidx_out[i] = pidx_in[s];
    type_out[i] = type_in[s];
    const double4 p = pos_in[s];
    pos_out[i] = p;
    snap[i] = p;
    const double4 v = vel_in[s];
    vel_out[i] = v;
    if (xv) {
        double2* q = xv + 3 * (size_t)i;
        q[0] = make_double2(p.x, p.y);
        q[1] = make_double2(p.z, v.x);
        q[2] = make_double2(v.y, v.z);
    }
}

// Neighbour list (main.cpp:1329-1585).  The particles of one home key (a cell's
// fluid, or its walls) share their 3^D stencil and its visiting order; a warp walks
// it with eight of them at a time, taken octant by octant of the cell so that the
// box around them is small.  Each candidate range is read 32 candidates at a time
// (one coalesced FP32 record per lane); those near the box are queued in order in
// shared memory, and every full queue is tested with a candidate per lane against
// one of the eight particles after the other: the FP32 prefilter, the exact FP64
// test of the reference where that leaves a doubt, and a ballot that numbers the
// hits in candidate order.  A particle's entries are therefore the reference's, in
// the reference's order: fluid candidates of the 27 cells, then wall candidates (a
// wall with no fluid neighbour skips the walls, main.cpp:1416), self included, each
// range ascending.  The order in which the particles are taken changes no list.
//
// What bounds it: the instruction count.  A particle's list costs about 1150
// warp instructions (its share of queueing 600 candidates for eight particles, then
// 20 to test 32 candidates against one), issued at 80 % of the peak (2,779,256 particles;
// 78 % at 258,392).  With a lane per particle, 32 candidates tested one after
// the other into a bit mask and the hits pushed one by one, half of the lanes idled
// in the pushes and in part-filled warps, and a small scene's few warps ran one long
// serial chain: 8.03 -> 4.37 ms a build at 2,779,256 particles (3-D dam), 436 -> 311 us
// at 213,868, 290 -> 106 at 20,116, 894 -> 710 at 314,432 (3-D column), 47 -> 36 at
// 22,500 in 2-D.
//
// The count and the fill of the reference are one pass: entries go to a
// table in rows of four, [cap / 4][n][4] (list_at): with single entries in rows
// every store filled an eighth of a sector that was evicted before its neighbours
// came (eight times the lists' bytes in DRAM traffic).  A list longer than cap is still counted,
// raises DEVFLAG_NEIGHBOR_OVERFLOW and the host rebuilds with a larger table.
// The entries within rs2 also go, in the same order, to the
// short sublist: a particle moves at most MARGIN/2 between builds (the
// rebuild test of main.cpp:1086-1108), so every pair within RadiusP until the
// next build is in it, and a sum over the pairs within RadiusP visits them in
// list order.
//
// Prefilter: FP32 positions relative to the domain origin (k_pos32) give a
// displacement within the bound of make_prefilter of the one the exact FP64
// test computes, so a candidate whose FP32 distance squared exceeds pf.r2_hi
// cannot pass that test and is skipped.  An axis with fewer than 4 cells
// contributes nothing to the FP32 distance (its minimum image need not be the
// neighbouring cell's), which only keeps more candidates.
constexpr int kListParts = 8;     // particles per group
constexpr int kListSorted = 128;  // home particles that are taken octant by octant (more: in slot order)

template <bool ALL3>  // every axis in the FP32 prefilter (pf.use all set)
__global__ void __launch_bounds__(32 * kListWarps, 8)
k_neighbor_list(SimConst c, const double4* __restrict__ pos, const float4* __restrict__ pos32, Prefilter pf,
                const int* __restrict__ cellstart, int* __restrict__ ncount, int* __restrict__ nlist, int cap,
                int* __restrict__ ncount_s, int* __restrict__ nlist_s, int cap_s, StepScalars* __restrict__ scal,
                int key_warps) {
    __shared__ float4 queue_[kListWarps][64];           // candidates near the box, in order (a ring)
    __shared__ float4 home_[kListWarps][kListParts];    // the group's FP32 positions and slots
    __shared__ unsigned char order_[kListWarps][kListSorted];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int gw = blockIdx.x * kListWarps + wib;
    const int key = gw / key_warps;   // home key in [0, 2*tot), key_warps warps share it
    if (key >= 2 * c.tot) return;     // whole warp
    const int hb = cellstart[key], he = cellstart[key + 1], first = (gw % key_warps) * kListParts;
    if (hb + first >= he) return;
    // the stencil of the home cell as main.cpp:1356-1392 computes it from the
    // key (a wall's key carries +TotalCellCount: its icx is cx + cc[0])
    const int icx = (key / (c.cc[1] * c.cc[2])) % c.tot;
    const int ic[3] = {icx, (key / c.cc[2]) % c.cc[1], key % c.cc[2]};
    int jmin[3], w[3], home[3];
    for (int d = 0; d < 3; ++d) {
        const int r = c.range[d];
        w[d] = 2 * r + 1;
        home[d] = ic[d] % c.cc[d];
        const int b = (2 * r) - (ic[d] + r) % c.cc[d];  // main.cpp:1376-1381
        jmin[d] = b > 0 ? b : 0;
    }
    // stencil slot s of axis d: the cell coordinate (main.cpp:1360-1372) and
    // the FP32 image offset (0, or -+ the domain width where the slot wraps)
    auto slot = [&](int d, int s_, float& off) {
        const int raw = home[d] - c.range[d] + s_;
        off = raw < 0 ? -pf.width[d] : (raw >= c.cc[d] ? pf.width[d] : 0.0f);
        return ((ic[d] - c.range[d] + s_) % c.cc[d] + c.cc[d]) % c.cc[d];
    };
    // lane s < w0*w1*w2 holds stencil slot s of the loop order of
    // main.cpp:1356-1392 (x outer, z inner): its ranges and image offsets
    const int nsl = w[0] * w[1] * w[2];  // at most 27: range <= 1 on every axis
    int st_b[2] = {0, 0}, st_e[2] = {0, 0};
    float st_x = 0.f, st_y = 0.f, st_z = 0.f;
    if (lane < nsl) {
        const int a0 = lane / (w[1] * w[2]), a1 = (lane / w[2]) % w[1], a2 = lane % w[2];
        const int cx = slot(0, (jmin[0] + a0) % w[0], st_x), cy = slot(1, (jmin[1] + a1) % w[1], st_y),
                  cz = slot(2, (jmin[2] + a2) % w[2], st_z);
        const int cell = cell_id(c, cx, cy, cz);
        st_b[0] = cellstart[cell];
        st_e[0] = cellstart[cell + 1];
        st_b[1] = cellstart[cell + c.tot];
        st_e[1] = cellstart[cell + c.tot + 1];
    }
    const int wall_begin = cellstart[c.tot], wall_end = cellstart[2 * c.tot];
    const bool is_wall = wall_begin <= hb && hb < wall_end;  // one key holds walls or fluid
    const size_t n = (size_t)c.n;
    float4* const queue = queue_[wib];
    float4* const homes = home_[wib];
    unsigned char* const order = order_[wib];
    const int nh = he - hb;
    const bool sorted = nh > kListParts && nh <= kListSorted;
    if (sorted) {  // a counting sort by octant of the home cell, along a Gray code (neighbouring octants in a row)
        const float mx = ((float)home[0] + 0.5f) * pf.cell_width[0], my = ((float)home[1] + 0.5f) * pf.cell_width[1],
                    mz = ((float)home[2] + 0.5f) * pf.cell_width[2];
        int base[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (int pass = 0; pass < 2; ++pass) {
            for (int h = 0; h < nh; h += 32) {
                int o = 8;
                if (h + lane < nh) {
                    const float4 f = pos32[hb + h + lane];
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
    int most = 0, most_s = 0;
    for (int h0 = first; h0 < nh; h0 += key_warps * kListParts) {
        const int np = min(kListParts, nh - h0);
        // the group, a particle per lane (0..7), and the box of its FP32 positions: a
        // candidate farther than the cut-off from it is no particle's neighbour
        // (Prefilter::r2_box)
        float b0x = kInf, b0y = kInf, b0z = kInf, b1x = -kInf, b1y = -kInf, b1z = -kInf;
        __syncwarp();
        if (lane < np) {
            const int i = hb + (sorted ? (int)order[h0 + lane] : h0 + lane);
            float4 f = pos32[i];
            b0x = b1x = f.x;
            b0y = b1y = f.y;
            b0z = b1z = f.z;
            f.w = __int_as_float(i);
            homes[lane] = f;
        }
#pragma unroll
        for (int o = kListParts / 2; o > 0; o >>= 1) {
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
        int cnt = 0, cnt_s = 0;  // lane p: particle p's
        unsigned takes = (1u << np) - 1u;
        int head = 0, queued = 0;
        auto test = [&](int m) {  // the first m (<= 32) of the queue
            const float4 q = queue[(head + lane) & 63];
            const int j = __float_as_int(q.w);
            const unsigned below = (1u << lane) - 1u;
#pragma unroll 1
            for (unsigned left = takes; left != 0u; left &= left - 1u) {
                const int p = __ffs(left) - 1;
                const float4 f = homes[p];
                const float fx = (ALL3 || pf.use[0]) ? q.x - f.x : 0.f;
                const float fy = (ALL3 || pf.use[1]) ? q.y - f.y : 0.f;
                const float fz = (ALL3 || pf.use[2]) ? q.z - f.z : 0.f;
                // FMA: fewer roundings than the bound allows for
                const float r2f = __fmaf_rn(fx, fx, __fmaf_rn(fy, fy, __fmul_rn(fz, fz)));
                bool in = lane < m && r2f <= pf.r2_hi;  // within rm unless in its shell
                bool in_short = in && r2f <= pf.rs2_lo;  // within rs for certain
                const int i = __float_as_int(f.w);
                if (in && (r2f > pf.r2_lo || (r2f > pf.rs2_lo && r2f <= pf.rs2_hi))) {
                    const double4 pi = pos[i], pj = pos[j];
                    const double q0 = omod_fast(pj.x - pi.x + c.half_width[0], c.width[0]) - c.half_width[0];
                    const double q1 = omod_fast(pj.y - pi.y + c.half_width[1], c.width[1]) - c.half_width[1];
                    const double q2 = omod_fast(pj.z - pi.z + c.half_width[2], c.width[2]) - c.half_width[2];
                    const double r2 = q0 * q0 + q1 * q1 + q2 * q2;
                    in = r2 <= c.rm2;
                    in_short = in && r2 <= c.rs2;
                }
                const unsigned hits = __ballot_sync(0xffffffffu, in);
                const unsigned hits_s = __ballot_sync(0xffffffffu, in_short);
                const int base_l = __shfl_sync(0xffffffffu, cnt, p);
                if (in) {
                    const int at = base_l + __popc(hits & below);
                    if (at < cap) nlist[list_at(at, n, i)] = j;
                }
                if (hits_s != 0u) {
                    const int base = __shfl_sync(0xffffffffu, cnt_s, p);
                    if (in_short) {
                        const int at = base + __popc(hits_s & below);
                        if (at < cap_s) nlist_s[list_at(at, n, i)] = j;
                    }
                }
                if (lane == p) {
                    cnt += __popc(hits);
                    cnt_s += __popc(hits_s);
                }
            }
        };
        for (int kind = 0; kind < 2; ++kind) {
            if (kind == 1 && is_wall) {  // main.cpp:1416: a wall with no fluid neighbour gets no wall entries
                takes &= __ballot_sync(0xffffffffu, cnt != 0);
                if (takes == 0u) break;
            }
            // the candidate chunks one after the other, the next one's records loaded
            // while this one is worked on
            int sl = -1, cb = 0, e = 0;
            float gx = 0.f, gy = 0.f, gz = 0.f;
            auto next = [&]() {  // the next chunk: [cb, min(cb + 32, e)) of stencil slot sl
                cb += 32;
                while (cb >= e) {
                    if (++sl >= nsl) return false;
                    cb = __shfl_sync(0xffffffffu, st_b[kind], sl);
                    e = __shfl_sync(0xffffffffu, st_e[kind], sl);
                    if (cb < e) {
                        gx = __shfl_sync(0xffffffffu, st_x, sl);
                        gy = __shfl_sync(0xffffffffu, st_y, sl);
                        gz = __shfl_sync(0xffffffffu, st_z, sl);
                    }
                }
                return true;
            };
            bool more = next();
            float4 qn = make_float4(0.f, 0.f, 0.f, 0.f);
            if (more && cb + lane < e) qn = pos32[cb + lane];
            while (more || queued > 0) {
                if (more) {
                    float4 q = qn;
                    const int j = cb + lane;
                    const bool in_range = j < e;
                    q.x += gx;
                    q.y += gy;
                    q.z += gz;
                    more = next();
                    if (more && cb + lane < e) qn = pos32[cb + lane];
                    const float ex = (ALL3 || pf.use[0]) ? fmaxf(0.f, fmaxf(b0x - q.x, q.x - b1x)) : 0.f;
                    const float ey = (ALL3 || pf.use[1]) ? fmaxf(0.f, fmaxf(b0y - q.y, q.y - b1y)) : 0.f;
                    const float ez = (ALL3 || pf.use[2]) ? fmaxf(0.f, fmaxf(b0z - q.z, q.z - b1z)) : 0.f;
                    const bool near =
                        in_range && __fmaf_rn(ex, ex, __fmaf_rn(ey, ey, __fmul_rn(ez, ez))) <= pf.r2_box;
                    const unsigned kept = __ballot_sync(0xffffffffu, near);
                    if (near) {
                        q.w = __int_as_float(j);
                        queue[(head + queued + __popc(kept & ((1u << lane) - 1u))) & 63] = q;
                    }
                    queued += __popc(kept);
                    __syncwarp();
                }
                if (queued >= 32 || (!more && queued > 0)) {
                    const int m = min(queued, 32);
                    test(m);
                    head += m;
                    queued -= m;
                    __syncwarp();
                }
            }
        }
        if (lane < np) {
            const int i = __float_as_int(homes[lane].w);
            ncount[i] = cnt;
            ncount_s[i] = cnt_s;
            most = max(most, cnt);
            most_s = max(most_s, cnt_s);
        }
    }
    most = __reduce_max_sync(0xffffffffu, most);
    most_s = __reduce_max_sync(0xffffffffu, most_s);
    if (lane == 0) {
        atomicMax(&scal->max_neighbors, most);
        atomicMax(&scal->max_short, most_s);
        if (most > cap || most_s > cap_s) atomicOr(&scal->flags, DEVFLAG_NEIGHBOR_OVERFLOW);
    }
}

// FP32 copies of the positions relative to the domain origin, for the list
// build's prefilter: Mod(x - dmin, W) in [0, W), the coordinate of the
// particle's image in the cell its CellId names (main.cpp:96-100).
__global__ void k_pos32(SimConst c, const double4* __restrict__ pos, float4* __restrict__ pos32) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    const double4 p = pos[i];
    pos32[i] = make_float4((float)omod(p.x - c.dmin[0], c.width[0]), (float)omod(p.y - c.dmin[1], c.width[1]),
                           (float)omod(p.z - c.dmin[2], c.width[2]), 0.f);
}

__global__ void k_pack3(int n, const double4* __restrict__ src, double* __restrict__ dst) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double4 p = src[i];
    dst[3 * (size_t)i + 0] = p.x;
    dst[3 * (size_t)i + 1] = p.y;
    dst[3 * (size_t)i + 2] = p.z;
}

__global__ void k_unpack3(int n, const double* __restrict__ src, double4* __restrict__ dst,
                          const int* __restrict__ type) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double w = type ? (double)type[i] : 0.0;
    dst[i] = make_double4(src[3 * (size_t)i], src[3 * (size_t)i + 1], src[3 * (size_t)i + 2], w);
}

inline int blocks(long long n, int t) { return (int)((n + t - 1) / t); }

}  // namespace

void launch_cell_index(const SimConst& c, const double4* pos, const int* type, int* keys, int* vals,
                       cudaStream_t s) {
    k_cell_index<<<blocks(c.pow2, 256), 256, 0, s>>>(c, pos, type, keys, vals);
}

// The reference's network (main.cpp:1137-1158): for m in [0, log2 P), k in [0, m],
// dist = 2^(m-k).  Passes with dist below the shared-memory block run inside
// k_bitonic_local; the others one launch each.  Same passes, same order.
int launch_bitonic_sort(const SimConst& c, int* keys, int* vals, cudaStream_t s) {
    const int P = c.pow2;
    int logP = 0;
    while ((1 << logP) < P) ++logP;
    if (logP == 0) return 0;
    const int logL = logP < kLogLocal ? logP : kLogLocal;
    const int L = 1 << logL;
    const int nblk = P / L;
    const int thr = (L / 2) < kSortThreads ? (L / 2) : kSortThreads;
    int launches = 0;
    // every main stage m < logL is entirely local
    k_bitonic_local<<<nblk, thr, 0, s>>>(keys, vals, L, logL, 0, logL);
    ++launches;
    for (int m = logL; m < logP; ++m) {
        for (int ld = m; ld >= logL; --ld) {
            k_bitonic_global<<<blocks(P / 2, 256), 256, 0, s>>>(keys, vals, P / 2, m, ld);
            ++launches;
        }
        k_bitonic_local<<<nblk, thr, 0, s>>>(keys, vals, L, logL, m, m + 1);
        ++launches;
    }
    return launches;
}

void launch_cell_ranges(const SimConst& c, const int* keys, int* cellstart, cudaStream_t s) {
    const int nb = 2 * c.tot + 1;
    k_cell_ranges<<<blocks(nb, 256), 256, 0, s>>>(keys, c.n, nb, cellstart);
}

void launch_reorder(const SimConst& c, const int* vals, const int* pidx_in, const int* type_in,
                    const double4* pos_in, const double4* vel_in, int* pidx_out, int* type_out,
                    double4* pos_out, double4* vel_out, double2* xv, double4* snap, cudaStream_t s) {
    k_reorder<<<blocks(c.n, 256), 256, 0, s>>>(c.n, vals, pidx_in, type_in, pos_in, vel_in, pidx_out,
                                               type_out, pos_out, vel_out, xv, snap);
}

// Bound of the prefilter (see k_neighbor_list).  An FP32 coordinate in
// [0, W) is within 2^-24 W of its FP64 value (two coordinates: 2 * 2^-24 W);
// a component is formed as (q + offset) - p_i with |q + offset| < 2W
// (2 * 2^-24 W more) and a small result (less than 2^-24 W more), so each
// component is within e = 5 * 2^-24 * W of the FP64 minimum-image
// displacement (W rounded to FP32 for the offset adds 2^-24 W), which is
// itself within 2^-50 W of the true one.  The FP32 distance is then within
// sqrt(3) e < 2e of the FP64 one, and the FP32 sum of squares (three
// roundings: a product and two FMAs) within a factor 1 + 2^-21 of its exact
// value: a candidate the FP64 test accepts (r <= rm)
// has an FP32 distance squared below (rm + 2e)^2 (1 + 2^-20), rounded up to
// the next float.  e is taken as 8 * 2^-24 * W for room.
// The box test of a candidate (its image q + offset against the box of the
// FP32 positions of the warp's particles) bounds each axis' gap by the
// component for every particle in the box, within the same e (the image sum
// q + offset rounds once, within 2^-24 2W): a candidate within rm of any of
// them has a box distance squared below (rm + 2e)^2 (1 + 2^-20); r2_box takes
// 4e for room.
Prefilter make_prefilter(const SimConst& c) {
    Prefilter pf{};
    double wmax = 0.0;
    for (int d = 0; d < 3; ++d) {
        pf.use[d] = c.cc[d] >= 4 && c.range[d] == 1;
        pf.width[d] = (float)c.width[d];
        pf.cell_width[d] = (float)c.cell_width[d];
        if (pf.use[d]) wmax = std::fmax(wmax, c.width[d]);
    }
    const double e = 8.0 * std::ldexp(wmax, -24);
    const double rm = std::sqrt(c.rm2);
    const double t = (rm + 2.0 * e) * (rm + 2.0 * e) * (1.0 + std::ldexp(1.0, -20));
    pf.r2_hi = std::nextafter((float)t, 3.0e38f);
    const double tb = (rm + 4.0 * e) * (rm + 4.0 * e) * (1.0 + std::ldexp(1.0, -20));
    pf.r2_box = std::nextafter((float)tb, 3.0e38f);
    // The other side of the same bounds: an FP32 distance squared at or below
    // (R - 2e)^2 (1 - 2^-20), rounded down to the previous float, puts the FP64
    // distance below R - 2e + 2e = R, so the FP64 test r2 <= R^2 holds for
    // certain and is skipped; only the candidates in the shell between the two
    // bounds take it.  Valid when every axis is compared in FP32 (an axis left
    // out of the prefilter contributes 0 in FP32 but not in FP64), or the axis
    // left out is the flat one of a 2-D run.
    bool all_axes = true;
    for (int d = 0; d < 3; ++d)
        if (!pf.use[d] && !(c.dim == 2 && d == 2)) all_axes = false;
    auto lo_bound = [&](double r) {
        if (!all_axes || r <= 2.0 * e) return -1.0f;
        const double t2 = (r - 2.0 * e) * (r - 2.0 * e) * (1.0 - std::ldexp(1.0, -20));
        return std::nextafter((float)t2, -1.0f);
    };
    const double rs = std::sqrt(c.rs2);
    pf.r2_lo = lo_bound(rm);
    pf.rs2_lo = lo_bound(rs);
    pf.rs2_hi = all_axes ? std::nextafter((float)((rs + 2.0 * e) * (rs + 2.0 * e) * (1.0 + std::ldexp(1.0, -20))),
                                          3.0e38f)
                         : 3.0e38f;
    return pf;
}

void launch_pos32(const SimConst& c, const double4* pos, float4* pos32, cudaStream_t s) {
    k_pos32<<<blocks(c.n, 256), 256, 0, s>>>(c, pos, pos32);
}

void launch_neighbor_list(const SimConst& c, const double4* pos, const float4* pos32, const int* cellstart,
                          int* ncount, int* nlist, int cap, int* ncount_s, int* nlist_s, int cap_s,
                          StepScalars* scal, cudaStream_t s) {
    const int key_warps = list_key_warps(c.dim, c.n, c.tot);
    const long long warps = 2LL * c.tot * key_warps;
    const Prefilter pf = make_prefilter(c);
    const int nb = (int)((warps + kListWarps - 1) / kListWarps);
    if (pf.use[0] && pf.use[1] && pf.use[2])
        k_neighbor_list<true><<<nb, 32 * kListWarps, 0, s>>>(c, pos, pos32, pf, cellstart, ncount, nlist, cap,
                                                              ncount_s, nlist_s, cap_s, scal, key_warps);
    else
        k_neighbor_list<false><<<nb, 32 * kListWarps, 0, s>>>(c, pos, pos32, pf, cellstart, ncount, nlist, cap,
                                                               ncount_s, nlist_s, cap_s, scal, key_warps);
}

void launch_pack3(int n, const double4* src, double* dst, cudaStream_t s) {
    k_pack3<<<blocks(n, 256), 256, 0, s>>>(n, src, dst);
}

void launch_unpack3(int n, const double* src, double4* dst, const int* type, cudaStream_t s) {
    k_unpack3<<<blocks(n, 256), 256, 0, s>>>(n, src, dst, type);
}

}  // namespace mph
