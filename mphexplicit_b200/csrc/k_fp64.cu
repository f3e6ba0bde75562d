// k_fp64.cu — the plain FP64 MPH-WC step on sm_100a, bit-exact against the
// reference's x86-64 build.
//
// The reference runs eight neighbour sweeps per step (main.cpp:1665-1985).
// Here they are two, a thread per particle or, in small scenes, several lanes,
// list order kept:
//   sweep A = DensityA + GravityCenter + DensityP + DivergenceP
//             (four independent sums over the same list) and, in the epilogue,
//             PhysicalCoefficients + PressureP value + PressureA value;
//   sweep B = PressureP + PressureA + DiffuseInterface + ViscosityV forces,
//             each in its own accumulator, added to Force in the reference's
//             order, then Gravity + Acceleration (velocity double-buffered).
// plus one per-particle kernel for Convection + Wall + PeriodicBoundary +
// the rebuild test.  Every FP expression keeps the reference's association
// order; the file is compiled with -fmad=false and uses IEEE division and
// square root, so each operation rounds exactly as on the CPU.
#include "mph_internal.h"
#include "mph_exact.cuh"

// Resident 128-thread blocks per SM the sweeps are compiled for (register cap
// 65536 / (128 * blocks)); latency hiding vs. spills, set by measurement.  The
// FP64 pipe and the L1 data pipe bound the sweeps (76 and 77 % active in the force sweep of
// the 2,779,256-particle dam break, 64 and 56 at 258,392): about 84 FP64 operations and
// one 48-byte gather per list entry.  On the 2,779,256-particle
// dam break the force sweep takes 2.34 ms at 6 blocks (80 registers, two spilled
// values), 2.42 at 5; sweep A 0.314 ms at 7, 0.332 at 6, 0.366 at 8.  Blocks of 64 or
// 256 threads give the same times, of 32 up to 13 % more.
#ifndef MPH_SWEEP_MINB
#define MPH_SWEEP_MINB 7
#endif
#ifndef MPH_SWEEPB_MINB
#define MPH_SWEEPB_MINB 6
#endif
// The surface-tension variants hold more live values per pair.  On the
// 314,432-particle two-fluid column: the force sweep 0.75 ms at 4 blocks (no
// spills), 0.85 at 5, 0.94 at 3; sweep A 0.323 ms at 7, 0.339 at 6, 0.376 at 5.
#ifndef MPH_SWEEP_MINB_ST
#define MPH_SWEEP_MINB_ST 7
#endif
#ifndef MPH_SWEEPB_MINB_ST
#define MPH_SWEEPB_MINB_ST 4
#endif

namespace mph {

namespace {

__device__ __forceinline__ double omod(double x, double w) { return x - w * floor(x / w); }

// Mod(x,w), main.cpp:70.  When 0 <= x < 0.75 w the rounded quotient is below 1,
// floor gives +0 and x - w*0 == x exactly: the division is skipped then.
__device__ __forceinline__ double omod_fast(double x, double w) {
    return (x >= 0.0 && x < 0.75 * w) ? x : omod(x, w);
}

// The record the pair sweeps gather per neighbour: position and velocity, 48
// bytes as three 16-byte words {x, y}, {z, vx}, {vy, vz}, written by the move
// (k_move) and by the reorder.  The gathers are the L1 data pipe's work, which bounded
// the sweeps before: a warp's gather of one neighbour per lane costs it 50-57 cycles as
// two 32-byte double4 (four 16-byte loads), 37 as two 32-byte loads and 27-32 as this
// record (measured with 40 to 1000 records in reach of a warp).  Force sweep 299 -> 255
// us on the 258,392-particle dam break and 3.08 -> 2.90 ms on the 2,779,256 one,
// sweep A 49 -> 43 us and 0.39 -> 0.36 ms, the move, which writes the records,
// 13 -> 16 us and 0.058 -> 0.082 ms.
struct XV {
    double2 a, b, c;
};
struct XVT {  // with the type
    XV p;
    int t;
};
struct XVP {  // with PressureP
    XV p;
    double pressure;
};
__device__ __forceinline__ XV ld_xv(const double2* __restrict__ xv, int j) {
    const double2* p = xv + 3 * (size_t)j;
    XV r;
    r.a = __ldg(p);
    r.b = __ldg(p + 1);
    r.c = __ldg(p + 2);
    return r;
}
// One 32-byte record of a 32-byte aligned array in one load (18-19 cycles of
// the L1 data pipe per warp-wide gather; two 16-byte loads take about 27).
__device__ __forceinline__ double4 ld_d4(const double4* __restrict__ a, int j) {
    double4 r;
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
        : "=d"(r.x), "=d"(r.y), "=d"(r.z), "=d"(r.w)
        : "l"(a + j));
    return r;
}
__device__ __forceinline__ void st_xv(double2* __restrict__ xv, int i, const double4& p, const double4& v) {
    double2* q = xv + 3 * (size_t)i;
    q[0] = make_double2(p.x, p.y);
    q[1] = make_double2(p.z, v.x);
    q[2] = make_double2(v.y, v.z);
}

// Minimum-image displacement x_j - x_i (main.cpp:1680 and every sweep):
// Mod(x_j - x_i + W/2, W) - W/2.  The division-free range 0 <= t < 0.75 W of Mod
// is tested for the three axes at once on the high words of t against that of
// 0.75 W (SimConst::q75_hi; a negative t, -0.0 and NaN have the sign bit set and
// compare above it): one branch instead of three.  A t with the bound's own high
// word takes Mod's general expression, which gives t itself where t < 0.75 W, and
// so does -0.0, which becomes +0.0 and the same displacement.
__device__ __forceinline__ void disp(const SimConst& c, double xi, double yi, double zi, double xj, double yj,
                                     double zj, double* x) {
    double t0 = xj - xi + c.half_width[0], t1 = yj - yi + c.half_width[1], t2 = zj - zi + c.half_width[2];
    if (!((unsigned)__double2hiint(t0) < c.q75_hi[0] && (unsigned)__double2hiint(t1) < c.q75_hi[1] &&
          (unsigned)__double2hiint(t2) < c.q75_hi[2])) {
        t0 = omod(t0, c.width[0]);
        t1 = omod(t1, c.width[1]);
        t2 = omod(t2, c.width[2]);
    }
    x[0] = t0 - c.half_width[0];
    x[1] = t1 - c.half_width[1];
    x[2] = t2 - c.half_width[2];
}
__device__ __forceinline__ void disp(const SimConst& c, const XV& pi, const XV& pj, double* x) {
    disp(c, pi.a.x, pi.a.y, pi.b.x, pj.a.x, pj.a.y, pj.b.x, x);
}
__device__ __forceinline__ void disp(const SimConst& c, const double4& pi, const double4& pj, double* x) {
    disp(c, pi.x, pi.y, pi.z, pj.x, pj.y, pj.z, x);
}

// Visits the cnt entries of particle i's list in order: visit(j, load(j)).  Two
// indices are loaded at a time, two to three entries ahead, and records one entry
// ahead, so the gathers overlap the previous pair's FP64 arithmetic; two entries
// per trip, so the records alternate between two sets of registers instead of
// being moved.  With disp's single branch and pair_root's, 158 -> 123 instructions
// per entry of the force sweep (2.60 -> 2.34 ms on the 2,779,256-particle dam break, 0.81
// -> 0.75 ms on the 314,432-particle column).  Whole rows of four indices and four entries
// per trip take more registers: 2.38 ms.
template <class Load, class Visit>
__device__ __forceinline__ void walk_list(const int* __restrict__ list, size_t n, int i, int cnt, Load&& load,
                                          Visit&& visit) {
    if (cnt <= 0) return;
    const int* lp = list + list_at(0, n, i);
    const size_t row = 4 * n - 2;  // from the second half of a row to the next row
    int2 q = __ldg(reinterpret_cast<const int2*>(lp));
    int ja = q.x, jb = cnt > 1 ? q.y : q.x;
    auto a = load(ja);
    for (int k = 0;; k += 2) {
        lp += (k & 2) ? row : (size_t)2;
        if (k + 2 < cnt) q = __ldg(reinterpret_cast<const int2*>(lp));
        auto b = load(jb);
        visit(ja, a);
        if (k + 1 >= cnt) break;
        a = load(q.x);  // past the end: a record again, not visited
        visit(jb, b);
        if (k + 2 >= cnt) break;
        ja = q.x;
        jb = k + 3 < cnt ? q.y : q.x;
    }
}

__device__ __forceinline__ int type_of(const double4& p) { return (int)p.w; }

// The distance r = sqrt(r2) of a pair that is in range (near) and its
// reciprocal; false for one that is not, and for a particle paired with itself
// (r2 = 0, which the list holds).  One branch on the way of every other pair.
__device__ __forceinline__ bool pair_root(double r2, bool near, bool self, double& r, Recip& ri) {
    if (near && plain_root(r2)) {
        sqrt_recip(r2, r, ri);
        return true;
    }
    if (!near || self) return false;
    sqrt_recip_any(r2, r, ri);
    return true;
}

// Convection (main.cpp:1605-1615), Wall (2013-2043), PeriodicBoundary
// (2306-2317) and the displacement maximum of neighborCalculation (1086-1100).
// AHEAD (a step launched ahead of the host): nothing to do once a step has asked
// for a rebuild; the last block to finish makes that test on the maximum
// (main.cpp:1102), counts the step and clears the maximum for the next move.
template <bool AHEAD>
__global__ void __launch_bounds__(256)
k_move(SimConst c, const int* __restrict__ cellstart, double4* __restrict__ pos, double4* __restrict__ vel,
       double2* __restrict__ xv, const double4* __restrict__ snap, const double* __restrict__ wall_center, StepScalars* __restrict__ scal) {
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
            const int t = type_of(p);
            const double* C = wall_center + 3 * t;
            const double (*R)[3] = c.wall_rot[t];
            const double* W = c.wall_omega[t];
            const double* U = c.wall_velocity[t];
            double r0 = p.x - C[0], r1 = p.y - C[1], r2 = p.z - C[2];
            r0 = R[0][0] * r0 + R[0][1] * r1 + R[0][2] * r2;   // in place, as main.cpp:2033-2035
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
        st_xv(xv, i, p, v);
        const double4 q = snap[i];
        double d[3];
        d[0] = omod_fast(p.x - q.x + c.half_width[0], c.width[0]) - c.half_width[0];
        d[1] = omod_fast(p.y - q.y + c.half_width[1], c.width[1]) - c.half_width[1];
        d[2] = omod_fast(p.z - q.z + c.half_width[2], c.width[2]) - c.half_width[2];
        s2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
        if (!(s2 > 0.0)) s2 = 0.0;  // a NaN never wins the reference's `>` test
    }
    // block maximum, then one atomic on the ordered bit pattern (s2 >= 0)
    for (int o = 16; o > 0; o >>= 1) {
        const double t = __shfl_xor_sync(0xffffffffu, s2, o);
        s2 = t > s2 ? t : s2;
    }
    __shared__ double red[8];
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s2;
    __syncthreads();
    if (threadIdx.x == 0) {
        double m = red[0];
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) m = red[w] > m ? red[w] : m;
        if (m > 0.0) atomicMax(&scal->max_shift2_bits, (unsigned long long)__double_as_longlong(m));
        if (AHEAD) {
            __threadfence();
            if (atomicAdd(&scal->blocks_done, 1u) == gridDim.x - 1) {  // the last block
                __threadfence();
                const unsigned long long bits = atomicAdd(&scal->max_shift2_bits, 0ull);
                scal->last_shift2_bits = bits;
                scal->max_shift2_bits = 0ull;
                scal->blocks_done = 0u;
                scal->steps_done += 1;
                scal->move_flags = scal->flags;
                if (__longlong_as_double((long long)bits) > c.shift_thr) scal->stop = 1;
            }
        }
    }
}

// Kernel shapes as functions of q = r/h (main.cpp:214-284; the reference's
// (1.0/h) factor is the rounded reciprocal inv_h, as there).
__device__ __forceinline__ double s_wa(const SimConst& c, double q) { return ((c.ca * q) * (1.0 - q)) * (1.0 - q); }
__device__ __forceinline__ double s_dwa(const SimConst& c, double q) {
    return ((c.ca * (1.0 - q)) * (1.0 - 3.0 * q)) * c.inv_ra;
}
__device__ __forceinline__ double s_wg(const SimConst& c, double q) { return c.cg * ((1.0 - q) * (1.0 - q)); }
__device__ __forceinline__ double s_dwg(const SimConst& c, double q) { return c.cg * (c.m2_rg * (1.0 - q)); }
__device__ __forceinline__ double s_wp(const SimConst& c, double q) { return c.cp * ((1.0 - q) * (1.0 - q)); }
__device__ __forceinline__ double s_dwp(const SimConst& c, double q) { return c.cp * (c.m2_rp * (1.0 - q)); }
__device__ __forceinline__ double s_dwv(const SimConst& c, double q) { return c.cv * (c.m2_rv * (1.0 - q)); }

// Sweep A: DensityA (main.cpp:1665-1692), GravityCenter (1695-1727),
// DensityP (1831-1858), DivergenceP (1860-1896), then
// calculatePhysicalCoefficients (1631-1662) and the PressureP / PressureA
// values (1904-1906, 1735-1740).  Every division of the reference is an
// exactly rounded div_rn (mph_exact.cuh) against one reciprocal per pair.
// DensityP and DivergenceP visit the short sublist (ncount_p, nlist_p: the
// list's entries within RadiusP+MARGIN, in list order, so every pair within
// RadiusP in the reference's order).  With surface tension DensityA and
// GravityCenter visit the list in a loop of their own; without, the step does
// not use DensityA (PressureA is zero and its force terms are not evaluated),
// and k_density_a computes it when it is read.
template <bool ST, bool RATIO>
__global__ void __launch_bounds__(128, ST ? MPH_SWEEP_MINB_ST : MPH_SWEEP_MINB)
k_sweep_a(SimConst c, const double2* __restrict__ xv, const int* __restrict__ type,
          const int* __restrict__ ncount, const int* __restrict__ nlist, const int* __restrict__ ncount_p,
          const int* __restrict__ nlist_p, double* __restrict__ dens_a,
          double* __restrict__ strain_p, double* __restrict__ div_p, double4* __restrict__ velp,
          double4* __restrict__ gcpa, double* __restrict__ wall_center, const StepScalars* __restrict__ skip) {
    if (skip && skip->stop) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (wall_center != nullptr && blockIdx.x == 0 && threadIdx.x < 12) {
        // WallCenter += WallVelocity*Dt (main.cpp:2048-2052); the move kernel of
        // this step has already used the old value.
        const int t = threadIdx.x / 3, d = threadIdx.x % 3;
        if (t >= 2) wall_center[3 * t + d] += c.wall_velocity[t][d] * c.dt;
    }
    if (i >= c.n) return;
    const XV pi = ld_xv(xv, i);
    const int ti = type[i];
    const size_t n = (size_t)c.n;
    double sum_a = 0.0, sum_p = 0.0, sum_d = 0.0;
    double g0 = 0.0, g1 = 0.0, g2 = 0.0;
    walk_list(nlist_p, n, i, ncount_p[i], [&](int j) { return ld_xv(xv, j); }, [&](int j, const XV& pj) {
        // DensityP, DivergenceP
        double x[3];
        disp(c, pi, pj, x);
        const double r2 = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
        // R*R - r2 >= 0 (main.cpp:1683 and the other density sums) is r2 <= R*R:
        // with gradual underflow a - b is zero only when a == b, and its sign exact
        double r;
        Recip ri;
        if (!pair_root(r2, r2 <= c.rp2, j == i, r, ri)) return;
        const double qp = div_q(r, c.rp, recip_const(c.inv_rp, c.inv_rp_lo));
        sum_p += s_wp(c, qp);
        const double dw = s_dwp(c, qp);
        const double e0 = div_q(x[0], r, ri), e1 = div_q(x[1], r, ri), e2 = div_q(x[2], r, ri);
        const double u0 = pj.b.y - pi.b.y, u1 = pj.c.x - pi.c.x, u2 = pj.c.y - pi.c.y;
        sum_d -= u0 * e0 * dw;
        sum_d -= u1 * e1 * dw;
        sum_d -= u2 * e2 * dw;
    });
    if (ST) {  // DensityA, GravityCenter
        walk_list(nlist, n, i, ncount[i],
                  [&](int j) { return XVT{ld_xv(xv, j), RATIO ? __ldg(type + j) : 0}; },  // unused words: no loads
                  [&](int j, const XVT& rj) {
            double x[3];
            disp(c, pi, rj.p, x);
            const double r2 = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
            const bool in_a = r2 <= c.ra2;
            const bool in_g = r2 <= c.rg2;
            double r;
            Recip ri;  // not used: its operations are not compiled
            if (!pair_root(r2, in_a || in_g, j == i, r, ri)) return;
            double ratio = 1.0;
            if (RATIO) ratio = c.ratio[ti][rj.t];
            const double qa = div_q(r, c.ra, recip_const(c.inv_ra, c.inv_ra_lo));
            if (in_a) {
                const double w = RATIO ? ratio * s_wa(c, qa) : s_wa(c, qa);
                sum_a += w;
            }
            if (in_g) {
                const double qg = c.rg_eq_ra ? qa : div_q(r, c.rg, recip_const(c.inv_rg, c.inv_rg_lo));
                const double w = RATIO ? ratio * s_wg(c, qg) : s_wg(c, qg);
                g0 += div_q(x[0] * w, c.r2g, recip_const(c.inv_r2g, c.inv_r2g_lo)) * c.rg;
                g1 += div_q(x[1] * w, c.r2g, recip_const(c.inv_r2g, c.inv_r2g_lo)) * c.rg;
                g2 += div_q(x[2] * w, c.r2g, recip_const(c.inv_r2g, c.inv_r2g_lo)) * c.rg;
            }
        });
        dens_a[i] = sum_a;
    }
    const double strain = sum_p - c.n0p;
    strain_p[i] = strain;
    div_p[i] = sum_d;
    double kappa = c.bulk_modulus[ti];
    if (strain < 0.0) kappa = 0.0;
    const double lambda = c.bulk_viscosity[ti];
    const double pp = -lambda * sum_d + kappa * strain;
    // sweep B gathers PressureP and {GravityCenter, PressureA} per neighbour;
    // without surface tension the latter stay zero (PressureA: k_density_a)
    velp[i] = make_double4(pi.b.y, pi.c.x, pi.c.y, pp);
    if (ST) {
        double pa = c.cof_a[ti] * (sum_a - c.n0a) / c.l0;
        if (c.n0a <= sum_a) pa = 0.0;
        gcpa[i] = make_double4(g0, g1, g2, pa);
    }
}

// DensityA (main.cpp:1665-1692) and PressureA (1735-1740) alone, for the
// readers of a form without surface tension: the pairs of k_sweep_a's DensityA
// sum in the same list order with the same arithmetic, from the positions
// that sweep used (the step changes only velocities after it), so the values
// are those the reference holds after the step.
template <bool RATIO>
__global__ void __launch_bounds__(128) k_density_a(SimConst c, const double4* __restrict__ pos,
                                                   const int* __restrict__ ncount, const int* __restrict__ nlist,
                                                   double* __restrict__ dens_a, double4* __restrict__ gcpa) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    const double4 pi = pos[i];
    const int ti = type_of(pi);
    const int cnt = ncount[i];
    const size_t n = (size_t)c.n;
    double sum_a = 0.0;
    walk_list(nlist, n, i, cnt, [&](int j) { return ld_d4(pos, j); }, [&](int j, const double4& pj) {
        double x[3];
        disp(c, pi, pj, x);
        const double r2 = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
        double r;
        Recip ri;
        if (!pair_root(r2, r2 <= c.ra2, j == i, r, ri)) return;
        const double qa = div_q(r, c.ra, recip_const(c.inv_ra, c.inv_ra_lo));
        sum_a += RATIO ? c.ratio[ti][type_of(pj)] * s_wa(c, qa) : s_wa(c, qa);
    });
    dens_a[i] = sum_a;
    double pa = c.cof_a[ti] * (sum_a - c.n0a) / c.l0;
    if (c.n0a <= sum_a) pa = 0.0;
    reinterpret_cast<double*>(gcpa + i)[3] = pa;
}

// Sweep B: PressureP force (main.cpp:1908-1938), PressureA force
// (1742-1775), DiffuseInterface (1782-1828, aj uses the type of i as in the
// reference), ViscosityV (1943-1984); Force = 0 + fP + fA + fDI + fV, then
// Gravity (1988-1998) and Acceleration (2000-2010) for fluid particles.
// The PressureP force visits only pairs within RadiusP, all of which are in
// the short sublist, in list order (the argument of k_neighbor_list), so that
// sum runs as its own loop over the short sublist and the main loop carries
// the other terms.  The terms and their order in each sum are the reference's;
// the main loop does not run the pressure block under a branch that some lane
// takes on nearly every entry while most lanes wait.
// LRN: the learned form.  The PressureA, DiffuseInterface and ViscosityV pair
// terms are not evaluated; fluid particle i adds instead the sum of its
// edge-MLP pair forces eforce[eoff[i] .. eoff[i+1]) (FP32, in edge order),
// which is also stored in lsum[i].
// MU1: visc_c * muij is one number for every pair of types, so the type of j
// is not gathered.
template <bool ST, bool RATIO, bool LRN, bool MU1>
__global__ void __launch_bounds__(128, ST ? MPH_SWEEPB_MINB_ST : MPH_SWEEPB_MINB)
k_sweep_b(SimConst c, const int* __restrict__ cellstart, const double2* __restrict__ xv,
          const int* __restrict__ type, const double4* __restrict__ velp, double4* __restrict__ vel_out,
          const double4* __restrict__ gcpa, const int* __restrict__ ncount, const int* __restrict__ nlist,
          const int* __restrict__ ncount_s, const int* __restrict__ nlist_s, double4* __restrict__ force,
          StepScalars* __restrict__ scal, const int* __restrict__ eoff, const float4* __restrict__ eforce,
          float4* __restrict__ lsum, int part, double* __restrict__ vel_host,
          const StepScalars* __restrict__ skip) {
    if (skip && skip->stop) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    const int nf = cellstart[c.tot];
    const XV pi = ld_xv(xv, i);
    // part 1: fluid only; a wall keeps its velocity (what the full sweep
    // writes for it) and its force is left for part 2 (output only)
    if (part == 1 && i >= nf) {
        vel_out[i] = make_double4(pi.b.y, pi.c.x, pi.c.y, 0.0);
        if (vel_host) {
            vel_host[3 * (size_t)i] = pi.b.y;
            vel_host[3 * (size_t)i + 1] = pi.c.x;
            vel_host[3 * (size_t)i + 2] = pi.c.y;
        }
        return;
    }
    if (part == 2 && i < nf) return;
    const int ti = type[i];
    const size_t n = (size_t)c.n;
    double fp0 = 0.0, fp1 = 0.0, fp2 = 0.0;
    double fa0 = 0.0, fa1 = 0.0, fa2 = 0.0;
    double fd0 = 0.0, fd1 = 0.0, fd2 = 0.0;
    double fv0 = 0.0, fv1 = 0.0, fv2 = 0.0;
    {  // PressureP force (main.cpp:1908-1938) over the short sublist
        const double ppi = velp[i].w;
        walk_list(nlist_s, n, i, ncount_s[i],
                  [&](int j) { return XVP{ld_xv(xv, j), __ldg(&velp[j].w)}; },
                  [&](int j, const XVP& rj) {
            double x[3];
            disp(c, pi, rj.p, x);
            const double r2 = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
            // R*R - r2 > 0 (main.cpp:1926 and the other force sums) is r2 < R*R
            double r;
            Recip ri;
            if (!pair_root(r2, r2 < c.rp2, j == i, r, ri)) return;
            const double qp = div_q(r, c.rp, recip_const(c.inv_rp, c.inv_rp_lo));
            const double dw = s_dwp(c, qp);
            const double gw0 = div_q(dw * x[0], r, ri), gw1 = div_q(dw * x[1], r, ri),
                         gw2 = div_q(dw * x[2], r, ri);
            const double ps = ppi + rj.pressure;
            fp0 += ps * gw0 * c.vol;
            fp1 += ps * gw1 * c.vol;
            fp2 += ps * gw2 * c.vol;
        });
    }
    if (!LRN) {
        const double ai = ST ? c.a_k[ti] : 0.0;
        double4 gci = make_double4(0, 0, 0, 0);
        if (ST) gci = gcpa[i];        // .w = PressureA
        constexpr bool TYPES = RATIO || !MU1;
        walk_list(nlist, n, i, ncount[i],
                  [&](int j) { return XVT{ld_xv(xv, j), TYPES ? __ldg(type + j) : 0}; },
                  [&](int j, const XVT& rj) {
            const XV& pj = rj.p;
            const int tj = rj.t;
            double x[3];
            disp(c, pi, pj, x);
            const double r2 = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
            // Without surface tension every CofA is 0, PressureA is +-0 and each
            // PressureA term adds a signed zero to a sum that starts at +0: the sum
            // stays +0 exactly, so the term is skipped (ST == false).
            const bool in_a = ST && (r2 < c.ra2);
            const bool in_g = ST && (r2 < c.rg2);
            const bool in_v = r2 < c.rv2;
            double r;
            Recip ri;
            if (!pair_root(r2, in_a || in_g || in_v, j == i, r, ri)) return;
            const double e0 = div_q(x[0], r, ri), e1 = div_q(x[1], r, ri), e2 = div_q(x[2], r, ri);
            const double qa = div_q(r, c.ra, recip_const(c.inv_ra, c.inv_ra_lo));
            double rij = 1.0, rji = 1.0;
            if (RATIO) { rij = c.ratio[ti][tj]; rji = c.ratio[tj][ti]; }
            if (ST) {
                const double4 gcj = ld_d4(gcpa, j);  // .w = PressureA
                if (in_a) {
                    const double dwa = s_dwa(c, qa);
                    const double dwij = RATIO ? rij * dwa : dwa;
                    const double dwji = RATIO ? rji * dwa : dwa;
                    const double s = gci.w * dwij + gcj.w * dwji;
                    fa0 += s * e0 * c.vol;
                    fa1 += s * e1 * c.vol;
                    fa2 += s * e2 * c.vol;
                }
                if (in_g) {
                    const double aj = ai;
                    const double qg = c.rg_eq_ra ? qa : div_q(r, c.rg, recip_const(c.inv_rg, c.inv_rg_lo));
                    const double wg = s_wg(c, qg);
                    const double wij = RATIO ? rij * wg : wg;
                    const double wji = RATIO ? rji * wg : wg;
                    fd0 -= div_q(aj * gcj.x * wji - ai * gci.x * wij, c.r2g, recip_const(c.inv_r2g, c.inv_r2g_lo)) * c.rg * c.vol_over_l0;
                    fd1 -= div_q(aj * gcj.y * wji - ai * gci.y * wij, c.r2g, recip_const(c.inv_r2g, c.inv_r2g_lo)) * c.rg * c.vol_over_l0;
                    fd2 -= div_q(aj * gcj.z * wji - ai * gci.z * wij, c.r2g, recip_const(c.inv_r2g, c.inv_r2g_lo)) * c.rg * c.vol_over_l0;
                    const double dg = s_dwg(c, qg);
                    const double dwij = RATIO ? rij * dg : dg;
                    const double dwji = RATIO ? rji * dg : dg;
                    double gr = 0.0;
                    gr += (aj * gcj.x * dwji - ai * gci.x * dwij) * x[0];
                    gr += (aj * gcj.y * dwji - ai * gci.y * dwij) * x[1];
                    gr += (aj * gcj.z * dwji - ai * gci.z * dwij) * x[2];
                    fd0 -= div_q((gr) * e0, c.r2g, recip_const(c.inv_r2g, c.inv_r2g_lo)) * c.rg * c.vol_over_l0;
                    fd1 -= div_q((gr) * e1, c.r2g, recip_const(c.inv_r2g, c.inv_r2g_lo)) * c.rg * c.vol_over_l0;
                    fd2 -= div_q((gr) * e2, c.r2g, recip_const(c.inv_r2g, c.inv_r2g_lo)) * c.rg * c.vol_over_l0;
                }
            }
            if (in_v) {
                const double qv = c.rv_eq_ra ? qa : div_q(r, c.rv, recip_const(c.inv_rv, c.inv_rv_lo));
                const double dw = -s_dwv(c, qv);
                const double u0 = pj.b.y - pi.b.y, u1 = pj.c.x - pi.c.x, u2 = pj.c.y - pi.c.y;
                const double cm = MU1 ? c.visc_mu[0][0] : c.visc_mu[ti][tj];
                const double dot = u0 * e0 + u1 * e1 + u2 * e2;
                fv0 += div_q(cm * dot * e0 * dw, r, ri) * c.vol;
                fv1 += div_q(cm * dot * e1 * dw, r, ri) * c.vol;
                fv2 += div_q(cm * dot * e2 * dw, r, ri) * c.vol;
            }
        });
    }
    if (LRN) {
        float l0 = 0.f, l1 = 0.f, l2 = 0.f;
        if (i < nf) {
            for (int g = eoff[i], ge = eoff[i + 1]; g < ge; ++g) {
                const float4 q = eforce[g];
                l0 += q.x;
                l1 += q.y;
                l2 += q.z;
            }
        }
        lsum[i] = make_float4(l0, l1, l2, 0.f);
        fv0 = l0;
        fv1 = l1;
        fv2 = l2;
    }
    double F0 = 0.0, F1 = 0.0, F2 = 0.0;   // resetForce (main.cpp:1617-1628)
    F0 += fp0; F1 += fp1; F2 += fp2;
    F0 += fa0; F1 += fa1; F2 += fa2;
    F0 += fd0; F1 += fd1; F2 += fd2;
    F0 += fv0; F1 += fv1; F2 += fv2;
    double4 vn = make_double4(pi.b.y, pi.c.x, pi.c.y, 0.0);
    if (i < nf) {
        const double m = c.density[ti] * c.vol;
        F0 += m * c.gravity[0];
        F1 += m * c.gravity[1];
        F2 += m * c.gravity[2];
        vn.x += F0 / m * c.dt;
        vn.y += F1 / m * c.dt;
        vn.z += F2 / m * c.dt;
        if (!(isfinite(vn.x) && isfinite(vn.y) && isfinite(vn.z))) atomicOr(&scal->flags, DEVFLAG_NONFINITE);
    }
    force[i] = make_double4(F0, F1, F2, 0.0);
    if (part != 2) {
        vel_out[i] = vn;
        if (vel_host) {  // mapped pinned host memory: the read-back travels while the sweep runs
            vel_host[3 * (size_t)i] = vn.x;
            vel_host[3 * (size_t)i + 1] = vn.y;
            vel_host[3 * (size_t)i + 2] = vn.z;
        }
    }
}

// ---- G lanes per particle (small scenes) ---------------------------------------
// With few particles the thread-per-particle sweeps leave most of the GPU idle
// and each thread's chain of dependent FP64 work over its ~200 list entries
// sets the time.  Here G lanes (4 to 32) take one particle: they compute the pair
// terms of G consecutive list entries at once (the expressions of k_sweep_a /
// k_sweep_b), stage them in shared memory, and one lane per sum adds them in list
// order: the same additions in the same order, so the same bits.  An entry without
// a term stages -0.0, which leaves any sum as it is (sums start at +0.0 and never
// hold -0.0), and a subtracted term is staged negated (a - t is a + (-t)).
constexpr int kGroupWarps = 4;

// The warp's stage: NV terms of its 32 lanes' entries (rows one double apart from
// a multiple of the banks, so the lanes that sum different terms do not collide).
template <int NV>
struct GroupStage {
    double v[NV][33];
};

// Walks the lists of the warp's particles, G entries of each per trip: lane sub of
// a particle evaluates entry k0 + sub (eval(j, record, v), on -0.0 terms), then
// add(stage, column of the particle's first entry) sums the G staged entries.
// Indices are loaded two trips ahead and records one.
template <int G, int NV, class Load, class Eval, class Add>
__device__ __forceinline__ void group_walk(GroupStage<NV>& st, const int* __restrict__ list, size_t n, int cnt, int self,
                                           Load&& load, Eval&& eval, Add&& add) {
    const int lane = threadIdx.x & 31, sub = lane & (G - 1);
    const int most = __reduce_max_sync(0xffffffffu, cnt);
    int ja = sub < cnt ? __ldg(list + list_at(sub, n, self)) : self;
    int jb = sub + G < cnt ? __ldg(list + list_at(sub + G, n, self)) : self;
    auto a = load(ja);
    for (int k0 = 0; k0 < most; k0 += G) {
        int jc = self;
        if (k0 + 2 * G + sub < cnt) jc = __ldg(list + list_at(k0 + 2 * G + sub, n, self));
        const auto b = load(jb);
        double v[NV];
#pragma unroll
        for (int q = 0; q < NV; ++q) v[q] = -0.0;
        if (k0 + sub < cnt) eval(ja, a, v);
#pragma unroll
        for (int q = 0; q < NV; ++q) st.v[q][lane] = v[q];
        __syncwarp();
        add(lane - sub);
        __syncwarp();
        ja = jb;
        jb = jc;
        a = b;
    }
}

// Sweep A (see k_sweep_a), all particles.
template <int G, bool ST, bool RATIO>
__global__ void __launch_bounds__(32 * kGroupWarps)
k_sweep_a_g(SimConst c, const double2* __restrict__ xv, const int* __restrict__ type,
            const int* __restrict__ ncount, const int* __restrict__ nlist, const int* __restrict__ ncount_p,
            const int* __restrict__ nlist_p, double* __restrict__ dens_a,
            double* __restrict__ strain_p, double* __restrict__ div_p, double4* __restrict__ velp,
            double4* __restrict__ gcpa, double* __restrict__ wall_center, const StepScalars* __restrict__ skip) {
    if (skip && skip->stop) return;
    __shared__ GroupStage<4> stage[kGroupWarps];
    if (wall_center != nullptr && blockIdx.x == 0 && threadIdx.x < 12) {
        // WallCenter += WallVelocity*Dt (main.cpp:2048-2052), as k_sweep_a
        const int t = threadIdx.x / 3, d = threadIdx.x % 3;
        if (t >= 2) wall_center[3 * t + d] += c.wall_velocity[t][d] * c.dt;
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, sub = lane & (G - 1);
    const int iw = (blockIdx.x * kGroupWarps + w) * (32 / G);
    if (iw >= c.n) return;  // whole warp
    const bool on = iw + lane / G < c.n;
    const int i = on ? iw + lane / G : c.n - 1;
    GroupStage<4>& st = stage[w];
    const XV pi = ld_xv(xv, i);
    const int ti = type[i];
    const size_t n = (size_t)c.n;
    double acc = 0.0;  // lane 0: DensityP; lane 1: DivergenceP (three terms per entry)
    group_walk<G, 4>(st, nlist_p, n, on ? ncount_p[i] : 0, i, [&](int j) { return ld_xv(xv, j); },
                     [&](int j, const XV& pj, double* v) {
        double x[3];
        disp(c, pi, pj, x);
        const double r2 = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
        double r;
        Recip ri;
        if (!pair_root(r2, r2 <= c.rp2, j == i, r, ri)) return;
        const double qp = div_q(r, c.rp, recip_const(c.inv_rp, c.inv_rp_lo));
        v[0] = s_wp(c, qp);
        const double dw = s_dwp(c, qp);
        const double e0 = div_q(x[0], r, ri), e1 = div_q(x[1], r, ri), e2 = div_q(x[2], r, ri);
        const double u0 = pj.b.y - pi.b.y, u1 = pj.c.x - pi.c.x, u2 = pj.c.y - pi.c.y;
        v[1] = -(u0 * e0 * dw);
        v[2] = -(u1 * e1 * dw);
        v[3] = -(u2 * e2 * dw);
    }, [&](int col) {
        if (sub < 2) {
#pragma unroll
            for (int e = 0; e < G; ++e) {
                acc += st.v[sub][col + e];
                if (sub == 1) {
                    acc += st.v[2][col + e];
                    acc += st.v[3][col + e];
                }
            }
        }
    });
    const double sum_p = __shfl_sync(0xffffffffu, acc, lane - sub);
    const double sum_d = __shfl_sync(0xffffffffu, acc, lane - sub + 1);
    double sum_a = 0.0, g0 = 0.0, g1 = 0.0, g2 = 0.0;
    if (ST) {  // DensityA, GravityCenter: sum s on lane s
        double as = 0.0;
        group_walk<G, 4>(st, nlist, n, on ? ncount[i] : 0, i,
                         [&](int j) { return XVT{ld_xv(xv, j), RATIO ? __ldg(type + j) : 0}; },
                         [&](int j, const XVT& rj, double* v) {
            double x[3];
            disp(c, pi, rj.p, x);
            const double r2 = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
            const bool in_a = r2 <= c.ra2;
            const bool in_g = r2 <= c.rg2;
            double r;
            Recip ri;  // not used: its operations are not compiled
            if (!pair_root(r2, in_a || in_g, j == i, r, ri)) return;
            double ratio = 1.0;
            if (RATIO) ratio = c.ratio[ti][rj.t];
            const double qa = div_q(r, c.ra, recip_const(c.inv_ra, c.inv_ra_lo));
            if (in_a) v[0] = RATIO ? ratio * s_wa(c, qa) : s_wa(c, qa);
            if (in_g) {
                const double qg = c.rg_eq_ra ? qa : div_q(r, c.rg, recip_const(c.inv_rg, c.inv_rg_lo));
                const double wgt = RATIO ? ratio * s_wg(c, qg) : s_wg(c, qg);
                v[1] = div_q(x[0] * wgt, c.r2g, recip_const(c.inv_r2g, c.inv_r2g_lo)) * c.rg;
                v[2] = div_q(x[1] * wgt, c.r2g, recip_const(c.inv_r2g, c.inv_r2g_lo)) * c.rg;
                v[3] = div_q(x[2] * wgt, c.r2g, recip_const(c.inv_r2g, c.inv_r2g_lo)) * c.rg;
            }
        }, [&](int col) {
            if (sub < 4) {
#pragma unroll
                for (int e = 0; e < G; ++e) as += st.v[sub][col + e];
            }
        });
        const int l0 = lane - sub;
        sum_a = __shfl_sync(0xffffffffu, as, l0);
        g0 = __shfl_sync(0xffffffffu, as, l0 + 1);
        g1 = __shfl_sync(0xffffffffu, as, l0 + 2);
        g2 = __shfl_sync(0xffffffffu, as, l0 + 3);
    }
    if (sub != 0 || !on) return;
    if (ST) dens_a[i] = sum_a;
    const double strain = sum_p - c.n0p;
    strain_p[i] = strain;
    div_p[i] = sum_d;
    double kappa = c.bulk_modulus[ti];
    if (strain < 0.0) kappa = 0.0;
    const double lambda = c.bulk_viscosity[ti];
    const double pp = -lambda * sum_d + kappa * strain;
    velp[i] = make_double4(pi.b.y, pi.c.x, pi.c.y, pp);
    if (ST) {
        double pa = c.cof_a[ti] * (sum_a - c.n0a) / c.l0;
        if (c.n0a <= sum_a) pa = 0.0;
        gcpa[i] = make_double4(g0, g1, g2, pa);
    }
}

// Force sweep (see k_sweep_b) of the particles [i0, i1); with walls, the walls
// [i1, n) keep their velocity in the blocks behind.
template <int G, bool ST, bool RATIO>
__global__ void __launch_bounds__(32 * kGroupWarps)
k_sweep_b_g(SimConst c, const double2* __restrict__ xv, const int* __restrict__ type,
            const double4* __restrict__ velp, double4* __restrict__ vel_out,
            const double4* __restrict__ gcpa, const int* __restrict__ ncount, const int* __restrict__ nlist,
            const int* __restrict__ ncount_s, const int* __restrict__ nlist_s, double4* __restrict__ force,
            StepScalars* __restrict__ scal, int i0, int i1, int group_blocks, double* __restrict__ vel_host,
            const StepScalars* __restrict__ skip) {
    if (skip && skip->stop) return;
    constexpr int NV = ST ? 12 : 3, NS = ST ? 9 : 3;  // terms; sums: fv, fa, fd (two terms each)
    constexpr int PER = (NS + G - 1) / G;             // sums per lane
    __shared__ GroupStage<NV> stage[kGroupWarps];
    auto put_velocity = [&](int i, double x, double y, double z) {
        vel_out[i] = make_double4(x, y, z, 0.0);
        if (vel_host) {  // mapped pinned host memory: the read-back travels while the sweep runs
            vel_host[3 * (size_t)i] = x;
            vel_host[3 * (size_t)i + 1] = y;
            vel_host[3 * (size_t)i + 2] = z;
        }
    };
    if ((int)blockIdx.x >= group_blocks) {  // walls
        const int i = i1 + ((int)blockIdx.x - group_blocks) * 32 * kGroupWarps + (int)threadIdx.x;
        if (i >= c.n) return;
        const XV p = ld_xv(xv, i);
        put_velocity(i, p.b.y, p.c.x, p.c.y);
        return;
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, sub = lane & (G - 1);
    const int iw = i0 + (blockIdx.x * kGroupWarps + w) * (32 / G);
    if (iw >= i1) return;  // whole warp
    const bool on = iw + lane / G < i1;
    const int i = on ? iw + lane / G : i1 - 1;
    GroupStage<NV>& st = stage[w];
    const XV pi = ld_xv(xv, i);
    const int ti = type[i];
    const size_t n = (size_t)c.n;
    double fp = 0.0;  // lane s: component s
    {  // PressureP over the short sublist
        const double ppi = velp[i].w;
        GroupStage<3>& sp = reinterpret_cast<GroupStage<3>&>(st);
        group_walk<G, 3>(sp, nlist_s, n, on ? ncount_s[i] : 0, i,
                         [&](int j) { return XVP{ld_xv(xv, j), __ldg(&velp[j].w)}; },
                         [&](int j, const XVP& rj, double* v) {
            double x[3];
            disp(c, pi, rj.p, x);
            const double r2 = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
            double r;
            Recip ri;
            if (!pair_root(r2, r2 < c.rp2, j == i, r, ri)) return;
            const double qp = div_q(r, c.rp, recip_const(c.inv_rp, c.inv_rp_lo));
            const double dw = s_dwp(c, qp);
            const double gw0 = div_q(dw * x[0], r, ri), gw1 = div_q(dw * x[1], r, ri),
                         gw2 = div_q(dw * x[2], r, ri);
            const double ps = ppi + rj.pressure;
            v[0] = ps * gw0 * c.vol;
            v[1] = ps * gw1 * c.vol;
            v[2] = ps * gw2 * c.vol;
        }, [&](int col) {
            if (sub < 3) {
#pragma unroll
                for (int e = 0; e < G; ++e) fp += sp.v[sub][col + e];
            }
        });
    }
    double fs[PER];
#pragma unroll
    for (int q = 0; q < PER; ++q) fs[q] = 0.0;
    {
        const double ai = ST ? c.a_k[ti] : 0.0;
        double4 gci = make_double4(0, 0, 0, 0);
        if (ST) gci = gcpa[i];        // .w = PressureA
        group_walk<G, NV>(st, nlist, n, on ? ncount[i] : 0, i,
                          [&](int j) { return XVT{ld_xv(xv, j), __ldg(type + j)}; },
                          [&](int j, const XVT& rj, double* v) {
            const XV& pj = rj.p;
            const int tj = rj.t;
            double x[3];
            disp(c, pi, pj, x);
            const double r2 = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
            const bool in_a = ST && (r2 < c.ra2);
            const bool in_g = ST && (r2 < c.rg2);
            const bool in_v = r2 < c.rv2;
            double r;
            Recip ri;
            if (!pair_root(r2, in_a || in_g || in_v, j == i, r, ri)) return;
            const double e0 = div_q(x[0], r, ri), e1 = div_q(x[1], r, ri), e2 = div_q(x[2], r, ri);
            const double qa = div_q(r, c.ra, recip_const(c.inv_ra, c.inv_ra_lo));
            double rij = 1.0, rji = 1.0;
            if (RATIO) { rij = c.ratio[ti][tj]; rji = c.ratio[tj][ti]; }
            if (in_v) {
                const double qv = c.rv_eq_ra ? qa : div_q(r, c.rv, recip_const(c.inv_rv, c.inv_rv_lo));
                const double dw = -s_dwv(c, qv);
                const double u0 = pj.b.y - pi.b.y, u1 = pj.c.x - pi.c.x, u2 = pj.c.y - pi.c.y;
                const double cm = c.visc_mu[ti][tj];
                const double dot = u0 * e0 + u1 * e1 + u2 * e2;
                v[0] = div_q(cm * dot * e0 * dw, r, ri) * c.vol;
                v[1] = div_q(cm * dot * e1 * dw, r, ri) * c.vol;
                v[2] = div_q(cm * dot * e2 * dw, r, ri) * c.vol;
            }
            if (ST) {
                const double4 gcj = ld_d4(gcpa, j);  // .w = PressureA
                if (in_a) {
                    const double dwa = s_dwa(c, qa);
                    const double dwij = RATIO ? rij * dwa : dwa;
                    const double dwji = RATIO ? rji * dwa : dwa;
                    const double sa = gci.w * dwij + gcj.w * dwji;
                    v[3 % NV] = sa * e0 * c.vol;
                    v[4 % NV] = sa * e1 * c.vol;
                    v[5 % NV] = sa * e2 * c.vol;
                }
                if (in_g) {
                    const Recip ir2g = recip_const(c.inv_r2g, c.inv_r2g_lo);
                    const double aj = ai;
                    const double qg = c.rg_eq_ra ? qa : div_q(r, c.rg, recip_const(c.inv_rg, c.inv_rg_lo));
                    const double wg = s_wg(c, qg);
                    const double wij = RATIO ? rij * wg : wg;
                    const double wji = RATIO ? rji * wg : wg;
                    v[6 % NV] = -(div_q(aj * gcj.x * wji - ai * gci.x * wij, c.r2g, ir2g) * c.rg * c.vol_over_l0);
                    v[7 % NV] = -(div_q(aj * gcj.y * wji - ai * gci.y * wij, c.r2g, ir2g) * c.rg * c.vol_over_l0);
                    v[8 % NV] = -(div_q(aj * gcj.z * wji - ai * gci.z * wij, c.r2g, ir2g) * c.rg * c.vol_over_l0);
                    const double dg = s_dwg(c, qg);
                    const double dwij = RATIO ? rij * dg : dg;
                    const double dwji = RATIO ? rji * dg : dg;
                    double gr = 0.0;
                    gr += (aj * gcj.x * dwji - ai * gci.x * dwij) * x[0];
                    gr += (aj * gcj.y * dwji - ai * gci.y * dwij) * x[1];
                    gr += (aj * gcj.z * dwji - ai * gci.z * dwij) * x[2];
                    v[9 % NV] = -(div_q((gr) * e0, c.r2g, ir2g) * c.rg * c.vol_over_l0);
                    v[10 % NV] = -(div_q((gr) * e1, c.r2g, ir2g) * c.rg * c.vol_over_l0);
                    v[11 % NV] = -(div_q((gr) * e2, c.r2g, ir2g) * c.rg * c.vol_over_l0);
                }
            }
        }, [&](int col) {
#pragma unroll
            for (int q = 0; q < PER; ++q) {
                const int s_ = sub + q * G;
                if (s_ < NS) {
#pragma unroll
                    for (int e = 0; e < G; ++e) {
                        fs[q] += st.v[s_][col + e];
                        if (ST && s_ >= 6) fs[q] += st.v[(s_ + 3) % NV][col + e];
                    }
                }
            }
        });
    }
    const int l0 = lane - sub;
    double S[9], P[3];
#pragma unroll
    for (int q = 0; q < 9; ++q) S[q] = q < NS ? __shfl_sync(0xffffffffu, fs[(q / G) % PER], l0 + q % G) : 0.0;
#pragma unroll
    for (int q = 0; q < 3; ++q) P[q] = __shfl_sync(0xffffffffu, fp, l0 + q);
    if (sub != 0 || !on) return;
    double F0 = 0.0, F1 = 0.0, F2 = 0.0;   // resetForce (main.cpp:1617-1628), as k_sweep_b
    F0 += P[0]; F1 += P[1]; F2 += P[2];
    F0 += S[3]; F1 += S[4]; F2 += S[5];
    F0 += S[6]; F1 += S[7]; F2 += S[8];
    F0 += S[0]; F1 += S[1]; F2 += S[2];
    double4 vn = make_double4(pi.b.y, pi.c.x, pi.c.y, 0.0);
    if (i < c.nf) {
        const double m = c.density[ti] * c.vol;
        F0 += m * c.gravity[0];
        F1 += m * c.gravity[1];
        F2 += m * c.gravity[2];
        vn.x += F0 / m * c.dt;
        vn.y += F1 / m * c.dt;
        vn.z += F2 / m * c.dt;
        if (!(isfinite(vn.x) && isfinite(vn.y) && isfinite(vn.z))) atomicOr(&scal->flags, DEVFLAG_NONFINITE);
    }
    force[i] = make_double4(F0, F1, F2, 0.0);
    if (vel_out) put_velocity(i, vn.x, vn.y, vn.z);
}

// Self-check of div_rn, div_q and sqrt_recip against the hardware IEEE
// operations: operands with random significands and exponents in [-40, 40],
// all-ones significands, and the operands nearest to a wrong rounding.

// Odd M in [2^53, 2^54) with M^2 = a 2^54 + k for a double a, k = 1 (mod 8): the
// square roots nearest to the middle of two doubles.  2-adic Newton iteration for
// 1/sqrt(k); each k has two such M.
__device__ double hard_root(int k, int which) {
    unsigned long long y = 1ull;
    for (int it = 0; it < 8; ++it) y *= (3ull - (unsigned long long)(long long)k * y * y) >> 1;
    unsigned long long m = (unsigned long long)(long long)k * y;  // sqrt(k)
    if (which) m = 0ull - m;
    m = (m & ((1ull << 53) - 1)) | (1ull << 53);
    // a root modulo 2^54, or (that + 2^53) is one
    if (((m * m - (unsigned long long)(long long)k) & ((1ull << 54) - 1)) != 0ull) m ^= 1ull << 53;
    const unsigned long long lo = m * m, hi = __umul64hi(m, m);
    const unsigned long long l2 = lo - (unsigned long long)(long long)k;
    const unsigned long long h2 = hi - (k > 0 && lo < (unsigned long long)k) + (k < 0 && l2 < lo);
    return (double)((h2 << 10) | (l2 >> 54));  // exact when the low bit allows, else a neighbour
}

// The x with |2^(j+1) x - T d| = 1 for an odd T in [2^53, 2^54): x/d nearest to the
// middle of two doubles (0: there is none).
__device__ double hard_numerator(unsigned long long d, int s, int j) {
    unsigned long long inv = d;
    for (int it = 0; it < 6; ++it) inv *= 2ull - d * inv;
    unsigned long long t = s > 0 ? 0ull - inv : inv;
    t &= (2ull << j) - 1;
    if (j == 52) t |= 1ull << 53;
    if (t < (1ull << 53)) return 0.0;
    const unsigned long long lo = t * d, hi = __umul64hi(t, d);
    const unsigned long long l2 = lo + (unsigned long long)(long long)s;
    const unsigned long long h2 = hi + (s > 0 && l2 < lo) - (s < 0 && lo == 0ull);
    const unsigned long long x = (h2 << (63 - j)) | (l2 >> (j + 1));
    return x >= (1ull << 52) && x < (1ull << 53) ? (double)x : 0.0;
}

__global__ void k_check_division(unsigned long long seed, long long n, unsigned long long* mismatches,
                                 double* first) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    auto same = [](double a, double b) { return __double_as_longlong(a) == __double_as_longlong(b); };
    auto bad = [&](double x, double y) {
        if (atomicAdd(mismatches, 1ull) == 0) { first[0] = x; first[1] = y; }
    };
    auto check = [&](double x, double y) {
        const double h = __drcp_rn(y), ref = x / y;
        if (!same(div_rn(x, y, h), ref)) bad(x, y);
        if (!same(div_q(x, y, recip_const(h, __fma_rn(-y, h, 1.0) * h)), ref)) bad(x, y);
    };
    auto check_root = [&](double a, double x) {
        double r;
        Recip c;
        if (plain_root(a)) sqrt_recip(a, r, c);
        else sqrt_recip_any(a, r, c);
        if (!same(r, sqrt(a))) bad(a, a);
        if (!same(div_q(x, r, c), x / r)) bad(x, r);
    };
    const long long t0 = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t0 < 40) {  // k = -79, -71, ..., 73, two roots each, and the doubles beside them
        const double a = hard_root(-79 + 8 * (int)(t0 >> 1), (int)(t0 & 1));
        for (int q = -4; q <= 4; ++q) check_root(a + q, 1.0 + q);
    } else if (t0 >= 64 && t0 < 192) {  // divisors 2^53 - 1, - 3, ..., - 63
        const int q = (int)t0 - 64;
        const unsigned long long d = (1ull << 53) - 1 - 2 * (q >> 2);
        const double x = hard_numerator(d, (q & 1) ? 1 : -1, (q & 2) ? 52 : 53);
        if (x != 0.0) {
            for (int e = -4; e <= 4; ++e) check(x + e, (double)d);
            const double y = (double)d;  // the same through a square root's reciprocal
            check_root(y * y, x);
        }
    }
    for (long long t = t0; t < n; t += stride) {
        unsigned long long z = seed + 0x9E3779B97F4A7C15ull * (unsigned long long)(t + 1);
        auto mix = [](unsigned long long v) {
            v ^= v >> 30; v *= 0xBF58476D1CE4E5B9ull;
            v ^= v >> 27; v *= 0x94D049BB133111EBull;
            return v ^ (v >> 31);
        };
        const unsigned long long a = mix(z), b = mix(z ^ 0xD1B54A32D192ED03ull), e = mix(z + 17);
        unsigned long long ma = a & 0xFFFFFFFFFFFFFull, mb = b & 0xFFFFFFFFFFFFFull;
        if ((e & 15) == 0) mb = 0xFFFFFFFFFFFFFull;
        if ((e & 15) == 1) ma = 0xFFFFFFFFFFFFFull;
        const int ea = (int)((e >> 8) % 81) - 40, eb = (int)((e >> 20) % 81) - 40;
        const unsigned long long sa = (e >> 40) & 1ull;
        const double x = __longlong_as_double((long long)((sa << 63) | ((unsigned long long)(1023 + ea) << 52) | ma));
        const double y = __longlong_as_double((long long)(((unsigned long long)(1023 + eb) << 52) | mb));
        check(x, y);
        check_root(y, x);
    }
}

// Virial stress at particles, main.cpp:2057-2302: four sums (PressureP,
// PressureA, ViscosityV, DiffuseInterface) added in that order.  Only the trace
// of the stress enters VirialPressureAtParticle, so the diagonal alone is summed,
// all four terms in one walk of the list, each sum in list order with the
// reference's expressions.  Without surface tension PressureA's and
// DiffuseInterface's terms are signed zeros added to sums that start at +0.
// One walk with the exact shortened divisions instead of four with the hardware's:
// 4.1 -> 0.36 ms on the 258,392-particle dam break, bound by the FP64 pipe.
template <bool ST>
__global__ void __launch_bounds__(128, ST ? 3 : 4)
k_virial(SimConst c, const double4* __restrict__ pos, const double4* __restrict__ vel,
         const double4* __restrict__ velp, const double4* __restrict__ gc, const int* __restrict__ ncount,
         const int* __restrict__ nlist, double* __restrict__ virial_p) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    const double4 pi = pos[i];
    const double4 vi = vel[i];
    const int ti = type_of(pi);
    const double ppi = velp[i].w;                            // PressureP
    const double4 gci = ST ? gc[i] : make_double4(0, 0, 0, 0);  // .w = PressureA
    const double ai = ST ? c.a_k[ti] : 0.0;
    const Recip ivol = recip_const(c.inv_vol, c.inv_vol_lo);
    double sp[3] = {0.0, 0.0, 0.0}, sa[3] = {0.0, 0.0, 0.0}, sv[3] = {0.0, 0.0, 0.0}, sd[3] = {0.0, 0.0, 0.0};
    struct Rec {
        double4 p, v;
    };
    walk_list(nlist, (size_t)c.n, i, ncount[i],
              [&](int j) { return Rec{ld_d4(pos, j), ld_d4(vel, j)}; },
              [&](int j, const Rec& rj) {
        double x[3];
        disp(c, pi, rj.p, x);
        const double r2 = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
        const bool in_p = r2 < c.rp2, in_v = r2 < c.rv2, in_a = ST && r2 < c.ra2, in_g = ST && r2 < c.rg2;
        double r;
        Recip ri;
        if (!pair_root(r2, in_p || in_v || in_a || in_g, j == i, r, ri)) return;
        const int tj = type_of(rj.p);
        if (in_p) {
            const double dw = s_dwp(c, div_q(r, c.rp, recip_const(c.inv_rp, c.inv_rp_lo)));
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const double f = ppi * div_q(dw * x[d], r, ri) * c.vol;
                sp[d] += div_q(f * x[d], c.vol, ivol);
            }
        }
        if (ST && in_a) {
            const double dw = c.ratio[ti][tj] * s_dwa(c, div_q(r, c.ra, recip_const(c.inv_ra, c.inv_ra_lo)));
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const double f = gci.w * div_q(dw * x[d], r, ri) * c.vol;
                sa[d] += div_q(f * x[d], c.vol, ivol);
            }
        }
        if (in_v) {
            const double dw = -s_dwv(c, div_q(r, c.rv, recip_const(c.inv_rv, c.inv_rv_lo)));
            const double e0 = div_q(x[0], r, ri), e1 = div_q(x[1], r, ri), e2 = div_q(x[2], r, ri);
            const double u0 = rj.v.x - vi.x, u1 = rj.v.y - vi.y, u2 = rj.v.z - vi.z;
            const double k = c.visc_mu[ti][tj] * (u0 * e0 + u1 * e1 + u2 * e2);
            const double e[3] = {e0, e1, e2};
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const double f = div_q(k * e[d] * dw, r, ri) * c.vol;
                sv[d] += div_q(0.5 * f * x[d], c.vol, ivol);
            }
        }
        if (ST && in_g) {
            const Recip ir2g = recip_const(c.inv_r2g, c.inv_r2g_lo);
            const double ratio = c.ratio[ti][tj];
            const double qg = div_q(r, c.rg, recip_const(c.inv_rg, c.inv_rg_lo));
            const double w = ratio * s_wg(c, qg), dw = ratio * s_dwg(c, qg);
            const double gv[3] = {gci.x, gci.y, gci.z};
            double gr = 0.0;
#pragma unroll
            for (int d = 0; d < 3; ++d) gr += (-gv[d]) * x[d];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const double f = div_q(-ai * (-gv[d]) * w, c.r2g, ir2g) * c.rg * c.vol_over_l0;
                sd[d] += div_q(f * x[d], c.vol, ivol);
                const double f2 = div_q(-ai * gr * div_q(dw * x[d], r, ri), c.r2g, ir2g) * c.rg * c.vol_over_l0;
                sd[d] += div_q(f2 * x[d], c.vol, ivol);
            }
        }
    });
    double S[3];
    for (int d = 0; d < 3; ++d) {
        S[d] = 0.0;
        S[d] += sp[d];
        S[d] += sa[d];
        S[d] += sv[d];
        S[d] += sd[d];
    }
    if (c.dim == 2) virial_p[i] = -1.0 / 2.0 * (S[0] + S[1]);
    else virial_p[i] = -1.0 / 3.0 * (S[0] + S[1] + S[2]);
}

// Fluid mass, momentum, kinetic energy: per-block partial sums in a fixed
// order (deterministic), summed on the host.
__global__ void __launch_bounds__(256)
k_conserved(SimConst c, const int* __restrict__ cellstart, const double4* __restrict__ pos,
            const double4* __restrict__ vel, double* __restrict__ partial) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double s[5] = {0, 0, 0, 0, 0};
    if (i < c.n && i < cellstart[c.tot]) {
        const double m = c.density[type_of(pos[i])] * c.vol;
        const double4 v = vel[i];
        s[0] = m;
        s[1] = m * v.x;
        s[2] = m * v.y;
        s[3] = m * v.z;
        s[4] = 0.5 * m * (v.x * v.x + v.y * v.y + v.z * v.z);
    }
    __shared__ double sh[5][256];
    for (int k = 0; k < 5; ++k) sh[k][threadIdx.x] = s[k];
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o)
            for (int k = 0; k < 5; ++k) sh[k][threadIdx.x] += sh[k][threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        for (int k = 0; k < 5; ++k) partial[5 * (size_t)blockIdx.x + k] = sh[k][0];
}

inline int blocks(long long n, int t) { return (int)((n + t - 1) / t); }

// Lanes per particle of a sweep over m particles (1: the thread-per-particle
// kernels): enough threads to fill the GPU, and no more, since every lane added
// splits the list finer and adds the ordered sums' trips.  Set by measurement
// (sweep A / force sweep in us at 1, 4, 8, 16, 32 lanes; long: lists of ~190
// entries, 3-D whole lists; short: ~40 and fewer, 2-D, and sweep A without surface
// tension):
//   long, force sweep, 2,736 fluid     70 / 27 / 20 / 17 / 18
//                      6,400           70 / 29 / 23 / 29 / 29
//                     16,940           76 / 45 / 42 / 48 / 56
//                     43,200           93 / 82 / 88 / 106 / 130
//                    102,400          171 / 183 / 200 / 245 / 293
//   long, surface tension, 4,096      136 / 52 / 35 / 29 / 31
//                         39,304      178 / 171 / 172 / 177 / 215
//                        110,592      365 / 416 / 463 / 500 / 638
//   short, 2-D force sweep, 1,600      37 / 19 / 15 / 13 / 13
//                          10,000      39 / 22 / 23 / 25 / 35
//                          22,500      42 / 35 / 37 / 42 / 65
//                          48,400      49 / 56 / 66 / 80 / 130
//   short, sweep A, 14,724             18 / 14 / 13 / 15 / 16
//                   26,128             18 / 14 / 15 / 18 / 22
//                   52,724             18 / 19 / 21 / 27 / 35
inline int group_lanes(const SimConst& c, int m, bool long_lists) {
    if (c.sweep_layout == 1) return 1;
    if (c.sweep_layout == 2) return 32;
    if (long_lists) return m <= 2000 ? 32 : m <= 4500 ? 16 : m <= 20000 ? 8 : m <= 60000 ? 4 : 1;
    return m <= 6000 ? 16 : m <= 16000 ? 8 : m <= 35000 ? 4 : 1;
}

// ---- learned form ----------------------------------------------------------

// exclusive prefix of ncount[i], i < nf, within blocks of 1024; block totals to bsum
__global__ void __launch_bounds__(1024) k_edge_scan1(const int* __restrict__ ncount, int nf, int* __restrict__ eoff,
                                                     int* __restrict__ bsum) {
    __shared__ int wsum[32];
    const int i = blockIdx.x * 1024 + threadIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int v = i < nf ? ncount[i] : 0;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[w] = x;
    __syncthreads();
    if (w == 0) {
        int t = wsum[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        wsum[lane] = t;
    }
    __syncthreads();
    const int before = (w > 0 ? wsum[w - 1] : 0) + x - v;
    if (i < nf) eoff[i] = before;
    if (threadIdx.x == 1023) bsum[blockIdx.x] = before + v;
}

// exclusive prefix of the block totals (one block, chunks of 1024 with a carry)
__global__ void __launch_bounds__(1024) k_edge_scan2(int* __restrict__ bsum, int nb) {
    __shared__ int wsum[32];
    __shared__ int carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int base = 0; base < nb; base += 1024) {
        const int i = base + threadIdx.x;
        const int v = i < nb ? bsum[i] : 0;
        int x = v;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) wsum[w] = x;
        __syncthreads();
        if (w == 0) {
            int t = wsum[lane];
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, t, o);
                if (lane >= o) t += y;
            }
            wsum[lane] = t;
        }
        __syncthreads();
        const int before = carry + (w > 0 ? wsum[w - 1] : 0) + x - v;
        if (i < nb) bsum[i] = before;
        __syncthreads();
        if (threadIdx.x == 1023) carry = before + v;
        __syncthreads();
    }
    if (threadIdx.x == 0) bsum[nb] = carry;
}

__global__ void __launch_bounds__(1024) k_edge_scan3(int* __restrict__ eoff, const int* __restrict__ bsum, int nf,
                                                     int nb) {
    const int i = blockIdx.x * 1024 + threadIdx.x;
    if (i < nf) eoff[i] += bsum[blockIdx.x];
    if (i == 0) eoff[nf] = bsum[nb];
}

// The fluid's lists as CSR edges.  32 particles a block: the rows of the table
// (512 bytes a warp) go through shared memory, 64 entries of each particle at a time,
// and leave as consecutive entries of one particle.  (A thread per particle wrote
// 4 bytes to 32 lines at once: 451 us for 23.1 M edges, now 78; 51 us for 0.2 M, now 14.)
constexpr int kFillEntries = 64;

__global__ void __launch_bounds__(128) k_edge_fill(const int* __restrict__ ncount, const int* __restrict__ nlist,
                                                   int n, int nf, const int* __restrict__ eoff, int* __restrict__ ei,
                                                   int* __restrict__ ej) {
    __shared__ __align__(16) int tile[32][kFillEntries + 4];  // rows 4 banks apart
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int i0 = blockIdx.x * 32, i = i0 + lane;
    const int cnt = i < nf ? ncount[i] : 0, b = i < nf ? eoff[i] : 0;
    const int most = __reduce_max_sync(0xffffffffu, cnt);
    for (int k0 = 0; k0 < most; k0 += kFillEntries) {
        for (int r = 4 * warp; r < kFillEntries; r += 16)
            if (k0 + r < cnt)
                *reinterpret_cast<int4*>(&tile[lane][r]) =
                    reinterpret_cast<const int4*>(nlist)[(size_t)((k0 + r) >> 2) * n + i];
        __syncthreads();
        for (int q = warp; q < 32; q += 4) {
            const int c = min(kFillEntries, __shfl_sync(0xffffffffu, cnt, q) - k0);
            const int to = __shfl_sync(0xffffffffu, b, q) + k0;
            for (int u = lane; u < c; u += 32) {
                ei[to + u] = i0 + q;
                ej[to + u] = tile[q][u];
            }
        }
        __syncthreads();
    }
}

__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// One training sample per thread: a random CSR edge (i, j), its inputs and
// the FP64 PressureA + DiffuseInterface + ViscosityV force of j on i, with the
// expressions of k_sweep_b (main.cpp:1742-1828, 1941-1985).
template <bool ST, bool RATIO>
__global__ void __launch_bounds__(128)
k_collect(SimConst c, const double4* __restrict__ pos, const double4* __restrict__ velp,
          const double4* __restrict__ gcpa, const int* __restrict__ ei, const int* __restrict__ ej, long long ne,
          long long count, unsigned long long seed, float4* __restrict__ out) {
    const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= count) return;
    const long long g = (long long)(mix64(seed ^ mix64((unsigned long long)q)) % (unsigned long long)ne);
    const int i = ei[g], j = ej[g];
    const double4 pi = pos[i], pj = pos[j];
    double x[3];
    disp(c, pi, pj, x);
    const double r2 = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
    const bool in_a = ST && (c.ra2 - r2 > 0);
    const bool in_g = ST && (c.rg2 - r2 > 0);
    const bool in_v = c.rv2 - r2 > 0;
    const int ti = type_of(pi), tj = type_of(pj);
    const double4 vi = velp[i], vj = velp[j];
    double f0 = 0.0, f1 = 0.0, f2 = 0.0;
    const bool valid = i != j && (in_a || in_g || in_v);
    const double r = sqrt(r2);
    if (valid) {
        const double ri = __drcp_rn(r);
        const double e0 = div_rn(x[0], r, ri), e1 = div_rn(x[1], r, ri), e2 = div_rn(x[2], r, ri);
        const double qa = div_rn(r, c.ra, c.inv_ra);
        double rij = 1.0, rji = 1.0;
        if (RATIO) { rij = c.ratio[ti][tj]; rji = c.ratio[tj][ti]; }
        if (in_a) {
            const double dwa = s_dwa(c, qa);
            const double s = gcpa[i].w * (RATIO ? rij * dwa : dwa) + gcpa[j].w * (RATIO ? rji * dwa : dwa);
            f0 += s * e0 * c.vol;
            f1 += s * e1 * c.vol;
            f2 += s * e2 * c.vol;
        }
        if (ST && in_g) {
            const double4 gci = gcpa[i], gcj = gcpa[j];
            const double ai = c.a_k[ti], aj = ai;
            const double qg = c.rg_eq_ra ? qa : div_rn(r, c.rg, c.inv_rg);
            const double wg = s_wg(c, qg);
            const double wij = RATIO ? rij * wg : wg, wji = RATIO ? rji * wg : wg;
            f0 -= div_rn(aj * gcj.x * wji - ai * gci.x * wij, c.r2g, c.inv_r2g) * c.rg * c.vol_over_l0;
            f1 -= div_rn(aj * gcj.y * wji - ai * gci.y * wij, c.r2g, c.inv_r2g) * c.rg * c.vol_over_l0;
            f2 -= div_rn(aj * gcj.z * wji - ai * gci.z * wij, c.r2g, c.inv_r2g) * c.rg * c.vol_over_l0;
            const double dg = s_dwg(c, qg);
            const double dwij = RATIO ? rij * dg : dg, dwji = RATIO ? rji * dg : dg;
            double gr = 0.0;
            gr += (aj * gcj.x * dwji - ai * gci.x * dwij) * x[0];
            gr += (aj * gcj.y * dwji - ai * gci.y * dwij) * x[1];
            gr += (aj * gcj.z * dwji - ai * gci.z * dwij) * x[2];
            f0 -= div_rn(gr * e0, c.r2g, c.inv_r2g) * c.rg * c.vol_over_l0;
            f1 -= div_rn(gr * e1, c.r2g, c.inv_r2g) * c.rg * c.vol_over_l0;
            f2 -= div_rn(gr * e2, c.r2g, c.inv_r2g) * c.rg * c.vol_over_l0;
        }
        if (in_v) {
            const double qv = c.rv_eq_ra ? qa : div_rn(r, c.rv, c.inv_rv);
            const double dw = -s_dwv(c, qv);
            const double u0 = vj.x - vi.x, u1 = vj.y - vi.y, u2 = vj.z - vi.z;
            const double dot = u0 * e0 + u1 * e1 + u2 * e2;
            const double cm = c.visc_mu[ti][tj];
            f0 += div_rn(cm * dot * e0 * dw, r, ri) * c.vol;
            f1 += div_rn(cm * dot * e1 * dw, r, ri) * c.vol;
            f2 += div_rn(cm * dot * e2 * dw, r, ri) * c.vol;
        }
    }
    const double il0 = 1.0 / c.l0;
    out[3 * q + 0] = make_float4((float)(x[0] * il0), (float)(x[1] * il0), (float)(x[2] * il0), (float)(r * il0));
    out[3 * q + 1] = make_float4((float)(vj.x - vi.x), (float)(vj.y - vi.y), (float)(vj.z - vi.z),
                                 (float)(ti + 4 * tj));
    out[3 * q + 2] = make_float4((float)f0, (float)f1, (float)f2, valid ? 1.f : 0.f);
}

__global__ void __launch_bounds__(256)
k_force_compare(int nf, const double4* __restrict__ fa, const double4* __restrict__ fb,
                const float4* __restrict__ lsum, double* __restrict__ sums) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double s0 = 0.0, s1 = 0.0, s2 = 0.0;
    if (i < nf) {
        const double4 a = fa[i], b = fb[i];
        const float4 l = lsum[i];
        const double d0 = a.x - b.x, d1 = a.y - b.y, d2 = a.z - b.z;
        s0 = d0 * d0 + d1 * d1 + d2 * d2;
        s1 = b.x * b.x + b.y * b.y + b.z * b.z;
        const double v0 = (double)l.x - d0, v1 = (double)l.y - d1, v2 = (double)l.z - d2;
        s2 = v0 * v0 + v1 * v1 + v2 * v2;
    }
    for (int o = 16; o > 0; o >>= 1) {
        s0 += __shfl_xor_sync(0xffffffffu, s0, o);
        s1 += __shfl_xor_sync(0xffffffffu, s1, o);
        s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&sums[0], s0);
        atomicAdd(&sums[1], s1);
        atomicAdd(&sums[2], s2);
    }
}

}  // namespace

void launch_move(const SimConst& c, const int* cellstart, double4* pos, double4* vel, double2* xv,
                 const double4* snap, const double* wall_center, StepScalars* scal, cudaStream_t s) {
    k_move<false><<<blocks(c.n, 256), 256, 0, s>>>(c, cellstart, pos, vel, xv, snap, wall_center, scal);
}

void launch_move_ahead(const SimConst& c, const int* cellstart, double4* pos, double4* vel, double2* xv,
                       const double4* snap, const double* wall_center, StepScalars* scal, cudaStream_t s) {
    k_move<true><<<blocks(c.n, 256), 256, 0, s>>>(c, cellstart, pos, vel, xv, snap, wall_center, scal);
}

void launch_sweep_a(const SimConst& c, const double2* xv, const int* type, const int* ncount, const int* nlist,
                    const int* ncount_s, const int* nlist_s, double* dens_a, double* strain_p, double* div_p,
                    double4* press, double4* gc, double* wall_center, cudaStream_t s, const StepScalars* skip) {
    const int g = group_lanes(c, c.n, c.dim == 3 && c.has_st);
    if (g > 1) {
        const int nb = blocks(c.n, kGroupWarps * (32 / g));
#define SWEEP_AG(G, ST, RATIO)                                                                                    \
    k_sweep_a_g<G, ST, RATIO><<<nb, 32 * kGroupWarps, 0, s>>>(c, xv, type, ncount, nlist, ncount_s, nlist_s, dens_a, \
                                                              strain_p, div_p, press, gc, wall_center, skip)
#define SWEEP_AG2(G)                                  \
    if (!c.has_st) SWEEP_AG(G, false, false);         \
    else if (c.ratio_all_one) SWEEP_AG(G, true, false); \
    else SWEEP_AG(G, true, true)
        switch (g) {
            case 4: SWEEP_AG2(4); break;
            case 8: SWEEP_AG2(8); break;
            case 16: SWEEP_AG2(16); break;
            default: SWEEP_AG2(32);
        }
#undef SWEEP_AG2
#undef SWEEP_AG
        return;
    }
    const int nb = blocks(c.n, 128);
#define SWEEP_A(ST, RATIO)                                                                                      \
    k_sweep_a<ST, RATIO><<<nb, 128, 0, s>>>(c, xv, type, ncount, nlist, ncount_s, nlist_s, dens_a, strain_p,    \
                                            div_p, press, gc, wall_center, skip)
    if (!c.has_st) SWEEP_A(false, false);  // the ratios weigh surface-tension sums alone
    else if (c.ratio_all_one) SWEEP_A(true, false);
    else SWEEP_A(true, true);
#undef SWEEP_A
}

void launch_density_a(const SimConst& c, const double4* pos, const int* ncount, const int* nlist, double* dens_a,
                      double4* gc, cudaStream_t s) {
    const int nb = blocks(c.n, 128) > 0 ? blocks(c.n, 128) : 1;
    if (c.ratio_all_one)
        k_density_a<false><<<nb, 128, 0, s>>>(c, pos, ncount, nlist, dens_a, gc);
    else
        k_density_a<true><<<nb, 128, 0, s>>>(c, pos, ncount, nlist, dens_a, gc);
}

void launch_sweep_b(const SimConst& c, const int* cellstart, const double2* xv, const int* type, double4* vel_out,
                    const double4* press, const double4* gc, const int* ncount, const int* nlist,
                    const int* ncount_s, const int* nlist_s, double4* force, StepScalars* scal, cudaStream_t s,
                    const int* eoff, const float4* eforce, float4* lsum, int part,
                    double* vel_host, const StepScalars* skip) {
    // the ratios weigh surface-tension terms alone
    const bool ratio = c.has_st && !c.ratio_all_one;
    // the particles whose pairs this launch evaluates
    const int b0 = part == 2 ? c.nf : 0, b1 = part == 1 ? c.nf : c.n;
    const int g = !eforce ? group_lanes(c, b1 - b0, c.dim == 3) : 1;
    if (g > 1) {
        const int gb = blocks(b1 - b0, kGroupWarps * (32 / g));
        const int nw = gb + (part == 1 ? blocks(c.n - c.nf, 32 * kGroupWarps) : 0);
        if (nw == 0) return;
#define SWEEP_BG(G, ST, RATIO)                                                                                    \
    k_sweep_b_g<G, ST, RATIO><<<nw, 32 * kGroupWarps, 0, s>>>(c, xv, type, press, part == 2 ? nullptr : vel_out, gc, \
                                                              ncount, nlist, ncount_s, nlist_s, force, scal, b0, b1, \
                                                              gb, vel_host, skip)
#define SWEEP_BG2(G)                                  \
    if (!c.has_st) SWEEP_BG(G, false, false);         \
    else if (!ratio) SWEEP_BG(G, true, false);        \
    else SWEEP_BG(G, true, true)
        switch (g) {
            case 4: SWEEP_BG2(4); break;
            case 8: SWEEP_BG2(8); break;
            case 16: SWEEP_BG2(16); break;
            default: SWEEP_BG2(32);
        }
#undef SWEEP_BG2
#undef SWEEP_BG
        return;
    }
    const int nb = blocks(c.n, 128);
#define SWEEP_B(ST, RATIO, LRN, MU1)                                                                             \
    k_sweep_b<ST, RATIO, LRN, MU1><<<nb, 128, 0, s>>>(c, cellstart, xv, type, press, vel_out, gc, ncount, nlist, \
                                                      ncount_s, nlist_s, force, scal, eoff, eforce, lsum, part,  \
                                                      vel_host, skip)
    if (eforce) SWEEP_B(false, false, true, true);
    else if (!c.has_st) { if (c.mu_uniform) SWEEP_B(false, false, false, true); else SWEEP_B(false, false, false, false); }
    else if (ratio) SWEEP_B(true, true, false, false);
    else if (c.mu_uniform) SWEEP_B(true, false, false, true);
    else SWEEP_B(true, false, false, false);
#undef SWEEP_B
}

void launch_virial(const SimConst& c, const double4* pos, const double4* vel, const double4* press,
                   const double4* gc, const int* ncount, const int* nlist, double* virial_p, cudaStream_t s) {
    const int nb = blocks(c.n, 128);
    if (c.has_st) k_virial<true><<<nb, 128, 0, s>>>(c, pos, vel, press, gc, ncount, nlist, virial_p);
    else k_virial<false><<<nb, 128, 0, s>>>(c, pos, vel, press, gc, ncount, nlist, virial_p);
}

int check_division(unsigned long long seed, long long n, unsigned long long* d_count, double* d_first,
                   cudaStream_t s) {
    k_check_division<<<148 * 8, 256, 0, s>>>(seed, n, d_count, d_first);
    return 1;
}

void launch_conserved(const SimConst& c, const int* cellstart, const double4* pos, const double4* vel,
                      double* partial, cudaStream_t s) {
    k_conserved<<<blocks(c.n, 256), 256, 0, s>>>(c, cellstart, pos, vel, partial);
}

int edge_scan_blocks(int nf) { return (nf + 1023) / 1024 + 1; }

void launch_edge_offsets(const int* ncount, int nf, int* eoff, int* bsum, cudaStream_t s) {
    const int nb = (nf + 1023) / 1024;
    if (nb == 0) {
        cudaMemsetAsync(eoff, 0, sizeof(int), s);
        return;
    }
    k_edge_scan1<<<nb, 1024, 0, s>>>(ncount, nf, eoff, bsum);
    k_edge_scan2<<<1, 1024, 0, s>>>(bsum, nb);
    k_edge_scan3<<<nb, 1024, 0, s>>>(eoff, bsum, nf, nb);
}

void launch_edge_fill(const int* ncount, const int* nlist, int n, int nf, const int* eoff, int* ei, int* ej,
                      cudaStream_t s) {
    if (nf > 0) k_edge_fill<<<blocks(nf, 32), 128, 0, s>>>(ncount, nlist, n, nf, eoff, ei, ej);
}

void launch_collect(const SimConst& c, const double4* pos, const double4* press, const double4* gc, const int* ei,
                    const int* ej, long long ne, long long count, unsigned long long seed, float4* out,
                    cudaStream_t s) {
    if (count <= 0 || ne <= 0) return;
    const unsigned nb = (unsigned)((count + 127) / 128);
#define COLLECT(ST, RATIO) k_collect<ST, RATIO><<<nb, 128, 0, s>>>(c, pos, press, gc, ei, ej, ne, count, seed, out)
    if (c.has_st) {
        if (c.ratio_all_one) COLLECT(true, false); else COLLECT(true, true);
    } else {
        if (c.ratio_all_one) COLLECT(false, false); else COLLECT(false, true);
    }
#undef COLLECT
}

void launch_force_compare(int nf, const double4* fa, const double4* fb, const float4* lsum, double* sums3,
                          cudaStream_t s) {
    if (nf > 0) k_force_compare<<<blocks(nf, 256), 256, 0, s>>>(nf, fa, fb, lsum, sums3);
}

}  // namespace mph
