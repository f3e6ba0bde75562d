// mph_pair32.cuh — FP32 pair terms shared by the mixed-precision sweeps
// (k_mixed.cu) and the batched sweeps (k_batch.cu).
//
// K is any constants struct with the FP32 fields used below (ratio, ra2,
// inv_ra, ca, ca_inv, rg2, inv_rg, cg, cg_m2, inv_r2g_rg, vol, vol_over_l0),
// all evaluated on the host from the FP64 set-up constants.
#pragma once
#include <cuda_runtime.h>

namespace mph {

// Kahan-compensated accumulation (Kahan 1965): s + t with the lost low-order
// part carried in c; the compensated value is s - c.
__device__ __forceinline__ void kahan_add(float& s, float& c, float t) {
    const float y = t - c;
    const float u = s + y;
    c = (u - s) - y;
    s = u;
}

// 1/sqrt(r2) with one Newton step (rsqrtf is within 2 ulp; the step brings it
// to about 1 ulp), for the pressure terms.
__device__ __forceinline__ float rsqrt_nr(float r2) {
    const float y = rsqrtf(r2);
    return y * fmaf(-0.5f * r2 * y, y, 1.5f);
}

// 1/sqrt(r2) in FP64 from an FP32 seed plus one Newton step (relative error
// ~1e-14), for the FP64 density pairs.
__device__ __forceinline__ double rsqrt_dnr(double r2) {
    const double y = (double)rsqrtf((float)r2);
    return y * (1.5 - 0.5 * r2 * y * y);
}

// Surface-tension sums of the density sweep for one pair: DensityA
// (main.cpp:1665-1692) and GravityCenter (main.cpp:1695-1727).
template <bool RATIO, class K>
__device__ __forceinline__ void st_density(const K& m, int ti, int tj, float r2, float r, float dx, float dy,
                                           float dz, float& sa, float& cak, float& g0, float& g1, float& g2) {
    const float ratio = RATIO ? m.ratio[ti][tj] : 1.0f;
    if (r2 <= m.ra2) {
        const float q = r * m.inv_ra;
        kahan_add(sa, cak, ratio * m.ca * q * (1.0f - q) * (1.0f - q));
    }
    if (r2 <= m.rg2) {
        const float q = 1.0f - r * m.inv_rg;
        const float wgt = ratio * m.cg * q * q * m.inv_r2g_rg;
        g0 += dx * wgt;
        g1 += dy * wgt;
        g2 += dz * wgt;
    }
}

// Surface-tension terms of one pair (PressureA, DiffuseInterface with aj the
// a of i as the reference has it, main.cpp:1742-1828); returns the radial
// part and adds the tangential part to t.  The difference of the two gravity
// centres, scaled by a of i, is formed once per axis (exact product, one rounding) and
// shared by the kernel's and its derivative's term.
template <bool RATIO, int DIM = 3, class K>
__device__ __forceinline__ float st_terms(const K& m, int ti, int tj, float r2, float r, float rinv, float dx,
                                          float dy, float dz, const float4& gi, const float4& gj, float ai,
                                          float3& t) {
    const float rij = RATIO ? m.ratio[ti][tj] : 1.0f, rji = RATIO ? m.ratio[tj][ti] : 1.0f;
    float s = 0.0f;
    if (r2 < m.ra2) {
        const float q = r * m.inv_ra;
        const float dwa = (m.ca_inv * m.vol) * (1.0f - q) * fmaf(-3.0f, q, 1.0f);
        s = (RATIO ? fmaf(gi.w, rij, gj.w * rji) : gi.w + gj.w) * dwa * rinv;
    }
    if (r2 < m.rg2) {
        const float q = 1.0f - r * m.inv_rg;
        const float k1 = m.inv_r2g_rg * m.vol_over_l0;
        const float wg = (m.cg * k1) * q * q, dwg = (m.cg_m2 * k1) * q;
        const float bi = RATIO ? ai * rij : ai, bj = RATIO ? ai * rji : ai;
        const float d0 = fmaf(bj, gj.x, -(bi * gi.x)), d1 = fmaf(bj, gj.y, -(bi * gi.y));
        t.x = fmaf(-d0, wg, t.x);
        t.y = fmaf(-d1, wg, t.y);
        float gr = fmaf(d0, dx, d1 * dy);
        if (DIM == 3) {  // in 2-D every z part is zero
            const float d2 = fmaf(bj, gj.z, -(bi * gi.z));
            t.z = fmaf(-d2, wg, t.z);
            gr = fmaf(d2, dz, gr);
        }
        s = fmaf(-gr, dwg * rinv, s);
    }
    return s;
}

}  // namespace mph
