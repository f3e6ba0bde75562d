// mph_internal.h — device constants, context layout and kernel launchers of the
// B200 MPH-WC explicit step.  Shared by the host orchestration (mph_host.cpp)
// and the CUDA translation units (k_cells.cu, k_fp64.cu, k_mixed.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <string>
#include "mph_b200.h"

namespace mph {

// Everything a step kernel needs that is fixed between rebuilds, passed by
// value (kernel parameter space) so no constant-memory upload is needed.
// The kernel-shape prefactors are evaluated on the host in the reference's
// operation order (main.cpp:214-284): e.g. wa = ((ca*q)*(1-q))*(1-q) with
// ca = (1/Swa)/h^D and q = r/h.
struct SimConst {
    int n;                 // particle count
    int nf;                // fluid particles (sorted first)
    int dim;
    int tot;               // TotalCellCount
    int cc[3];             // CellCount
    int range[3];          // stencil half-width per axis (1, or 0 for z in 2-D)
    int pow2;              // PowerParticleCount
    int has_st;            // any surface tension -> diffuse-interface terms
    int ratio_all_one;     // InteractionRatio == 1 everywhere
    int mu_uniform;        // visc_mu is one number for every pair of types
    double dmin[3], width[3], half_width[3], cell_width[3];
    unsigned q75_hi[3];  // high word of 0.75*width: Mod(x, w) needs no division when 0 <= x < 0.75 w
    double dt, l0, vol, vol_over_l0;
    double n0a, n0p, r2g, cof_k;
    double ra, rg, rp, rv;             // radii
    double ra2, rg2, rp2, rv2;         // radius*radius
    double rm2;                        // (MaxRadius+MARGIN)^2, neighbour cut-off
    double rs2;                        // ((RadiusP+MARGIN)(1+1e-9))^2, cut-off of the short sublist
    double ca, cg, cp, cv;             // (1/Sw)/h^D for wa, wg/dwg, wp/dwp, dwv
    double inv_ra, inv_rg, inv_rp, inv_rv;  // 1.0/h
    double m2_rg, m2_rp, m2_rv;        // -2.0/h
    double visc_c;                     // 8 (2-D) or 10 (3-D)
    double inv_r2g;                    // RN(1/R2g)
    // what RN(1/h) lacks to 1/h, for the exact divisions by a constant (div_q)
    double inv_ra_lo, inv_rg_lo, inv_rp_lo, inv_rv_lo, inv_r2g_lo;
    double inv_vol, inv_vol_lo;        // the same for the particle volume
    int rg_eq_ra, rv_eq_ra;            // radii equal: r/h shared
    int sweep_layout;                  // FP64 sweeps: 0 by size, 1 thread per particle, 2 warp per particle
    // visc_c * muij per type pair, muij = 2*(mu_i*mu_j)/(mu_i+mu_j) (main.cpp:1968)
    double visc_mu[MPH_TYPE_COUNT][MPH_TYPE_COUNT];
    double shift_thr;                  // 0.5*MARGIN*0.5*MARGIN
    double density[MPH_TYPE_COUNT], bulk_modulus[MPH_TYPE_COUNT];
    double bulk_viscosity[MPH_TYPE_COUNT], shear_viscosity[MPH_TYPE_COUNT];
    double cof_a[MPH_TYPE_COUNT], a_k[MPH_TYPE_COUNT];  // a_k = CofA*CofK*CofK
    double ratio[MPH_TYPE_COUNT][MPH_TYPE_COUNT];
    double gravity[3];
    double wall_velocity[MPH_TYPE_COUNT][3], wall_omega[MPH_TYPE_COUNT][3];
    double wall_rot[MPH_TYPE_COUNT][3][3];
};

// Warps that share a key (a cell's fluid, or its walls) in the list builds of the FP64
// and the mixed form: enough to fill the GPU in small scenes.  us a build at 1, 2, 4 warps
// (FP64): 3-D, 20,116 particles 360 / 186 / 106; 213,868 474 / 333 / 311; 2,779,256 4403 /
// 4368 / 4607 (each warp sorts its key's particles anew); 2-D (13 particles a key), 22,500
// 50 / 36 / 37; 90,000 84 / 85 / 103.  Mixed: 3-D, 21,924 279 / - / 83; 258,392 429 / 347 /
// 335; 1,526,488 2100 / 2049 / 2150; 2-D, 3,600 22 / 14 / 15; 90,000 62 / - / 86.
// A warp without particles costs 0.14 ns, so a mostly empty grid gets no more of them: 8,000
// particles in 432,000 keys 354 / 198 / 248, in 2,000,000 382 / 562 / 1109; 2-D, 3,600 in 180,000
// 43 / 60 / 109.  The kernels number the warps in 32 bits: at most 2^30 (make_simconst takes up
// to 2^29 cells, two keys each).
constexpr int kListWarps = 4;  // warps per block
inline int list_key_warps(int dim, int n, int tot) {
    const long long keys = 2LL * tot, most = dim == 2 ? 1 << 17 : 1 << 20;
    int w = dim == 2 ? (n <= 50000 ? 2 : 1) : (n <= 250000 ? 4 : 2);
    while (w > 1 && keys * w > most) w /= 2;
    return w;
}

// Entry k of particle i's neighbour list: the tables hold rows of four entries,
// [cap / 4][n][4].
__host__ __device__ inline size_t list_at(int k, size_t n, int i) {
    return ((size_t)(k >> 2) * n + (size_t)i) * 4 + (size_t)(k & 3);
}

// Small per-step device scalars (one cache line, read back with one copy).
struct StepScalars {
    unsigned long long max_shift2_bits;  // max |shift|^2 as ordered bits (>= 0)
    unsigned long long last_shift2_bits; // steps launched ahead: the last moved step's maximum
    int flags;                           // MPH_DEVFLAG_*
    int max_neighbors;                   // longest list of the last build
    int max_short, max_long;             // longest short / long part (mixed table)
    int stop;                            // steps launched ahead: a step asked for a rebuild, the later ones do nothing
    int steps_done;                      // steps launched ahead: steps moved so far
    unsigned blocks_done;                // steps launched ahead: move blocks finished in this launch
    int move_flags;                      // steps launched ahead: `flags` at the last moved step's end of the move
    int pad[4];
};

enum : int {
    DEVFLAG_NEIGHBOR_OVERFLOW = 1,
    DEVFLAG_NONFINITE = 2,
    DEVFLAG_CELL_RANGE = 4,
};

// Device buffers of the FP64 form.  Arrays are in cell-sorted order.
struct DevFP64 {
    char* slab = nullptr;                   // the one allocation of every array but the two lists
    int* pidx[2] = {nullptr, nullptr};
    int* type[2] = {nullptr, nullptr};
    double4* pos[2] = {nullptr, nullptr};   // x,y,z,(double)type
    double4* vel[2] = {nullptr, nullptr};   // vx,vy,vz,0
    int cur = 0;                            // index of the current pos/type/pidx
    int vcur = 0;                           // index of the current velocity
    double2* xv = nullptr;                  // {x, y}, {z, vx}, {vy, vz}: the FP64 sweeps' gathers
    double4* snap = nullptr;                // NeighborCalculatedPosition
    float4* pos32 = nullptr;                // FP32 x - dmin for the list build's prefilter
    double4* force = nullptr;
    double* dens_a = nullptr;
    double* strain_p = nullptr;
    double* div_p = nullptr;
    double4* press = nullptr;               // {vx, vy, vz, PressureP} before the acceleration
    double4* gc = nullptr;                  // {GravityCenter, PressureA}
    double* virial_p = nullptr;
    int* keys = nullptr;                    // CellIndex (sorted), pow2 entries
    int* vals = nullptr;                    // CellParticle, pow2 entries
    int* cellstart = nullptr;               // 2*tot+1: #keys below each key value
    int* ncount = nullptr;                  // NeighborCount
    int* nlist = nullptr;                   // [cap / 4][n][4] (list_at)
    int cap = 0;
    int* ncount_s = nullptr;                // short sublist: the entries
    int* nlist_s = nullptr;                 // within rs2, in list order, [cap_s / 4][n][4]
    int cap_s = 0;
    double* wall_center = nullptr;          // [4][3], advanced on the device
    double* staging = nullptr;              // [n][3] pack/unpack buffer
    StepScalars* scal = nullptr;
};

// ---- kernel launchers (k_cells.cu) ----------------------------------------
void launch_cell_index(const SimConst& c, const double4* pos, const int* type, int* keys,
                       int* vals, cudaStream_t s);
int launch_bitonic_sort(const SimConst& c, int* keys, int* vals, cudaStream_t s);  // returns #launches
void launch_cell_ranges(const SimConst& c, const int* keys, int* cellstart, cudaStream_t s);
// xv: the sweeps' records of the reordered particles (nullptr: not wanted)
void launch_reorder(const SimConst& c, const int* vals, const int* pidx_in, const int* type_in,
                    const double4* pos_in, const double4* vel_in, int* pidx_out, int* type_out,
                    double4* pos_out, double4* vel_out, double2* xv, double4* snap, cudaStream_t s);
// FP32 prefilter of the neighbour-list build: per axis whether it takes part,
// the domain width, and the FP32 distance squared above which no candidate
// can pass the exact FP64 test.
struct Prefilter {
    int use[3];
    float width[3];
    float cell_width[3];
    float r2_hi;   // per pair: FP32 distance squared at or below it for every pair within rm
    float r2_box;  // per candidate: FP32 distance squared to the box around a warp's particles
    float r2_lo;   // FP32 distance squared at or below it: within rm in FP64 for certain (-1: never)
    float rs2_lo, rs2_hi;  // the same two bounds for the short radius rs
};
Prefilter make_prefilter(const SimConst& c);
// FP32 positions relative to the domain origin (the prefilter's input).
void launch_pos32(const SimConst& c, const double4* pos, float4* pos32, cudaStream_t s);
// nlist_s != nullptr: also the short sublist (entries within rs2, in list
// order; its longest length in scal->max_short).  pos32 (launch_pos32) feeds
// the FP32 prefilter that skips candidates surely beyond the cut-off (the
// list is the same).
void launch_neighbor_list(const SimConst& c, const double4* pos, const float4* pos32, const int* cellstart,
                          int* ncount, int* nlist, int cap, int* ncount_s, int* nlist_s, int cap_s,
                          StepScalars* scal, cudaStream_t s);
void launch_pack3(int n, const double4* src, double* dst, cudaStream_t s);

// the move of a step launched ahead of the host (k_fp64.cu): as launch_move, and
// its last block makes the rebuild test of main.cpp:1102 (when it fires, scal->stop
// makes this step's sweeps and every later step's kernels do nothing), counts the
// step and clears the maximum shift for the next step
void launch_move_ahead(const SimConst& c, const int* cellstart, double4* pos, double4* vel, double2* xv,
                       const double4* snap, const double* wall_center, StepScalars* scal, cudaStream_t s);
void launch_unpack3(int n, const double* src, double4* dst, const int* type, cudaStream_t s);

// ---- kernel launchers (k_fp64.cu) -----------------------------------------
// xv receives the moved particles' {x, y}, {z, vx}, {vy, vz}
void launch_move(const SimConst& c, const int* cellstart, double4* pos, double4* vel, double2* xv,
                 const double4* snap, const double* wall_center, StepScalars* scal, cudaStream_t s);
// Sweep A's DensityP and DivergenceP visit the short sublist (ncount_s,
// nlist_s); with surface tension DensityA and GravityCenter the whole list.
// skip: the sweep does nothing when skip->stop is set (steps launched ahead)
void launch_sweep_a(const SimConst& c, const double2* xv, const int* type, const int* ncount, const int* nlist,
                    const int* ncount_s, const int* nlist_s, double* dens_a, double* strain_p, double* div_p,
                    double4* press, double4* gc, double* wall_center, cudaStream_t s,
                    const StepScalars* skip = nullptr);
// DensityA and PressureA alone (into dens_a and gc[].w), in k_sweep_a's
// order: what sweep A leaves out when there is no surface tension.
void launch_density_a(const SimConst& c, const double4* pos, const int* ncount, const int* nlist, double* dens_a,
                      double4* gc, cudaStream_t s);
// eforce != nullptr: the learned form (edge-MLP pair forces replace the
// PressureA, DiffuseInterface and ViscosityV terms; see k_sweep_b; it visits
// the short sublist alone).
// part: 0 every particle; 1 the fluid (walls copy their velocity, their
// force is not written); 2 the walls' forces alone (vel_out unused).
// ncount_s / nlist_s: the short sublist, over which the PressureP force runs
// as its own loop (same result).  xv: positions and velocities of the step.
// vel_host (part 1): a device-accessible [n][3] view of pinned host memory that
// also receives each particle's new velocity.
void launch_sweep_b(const SimConst& c, const int* cellstart, const double2* xv, const int* type, double4* vel_out,
                    const double4* press, const double4* gc, const int* ncount, const int* nlist,
                    const int* ncount_s, const int* nlist_s, double4* force, StepScalars* scal, cudaStream_t s,
                    const int* eoff = nullptr, const float4* eforce = nullptr, float4* lsum = nullptr,
                    int part = 0, double* vel_host = nullptr, const StepScalars* skip = nullptr);

// ---- learned form (k_fp64.cu) ---------------------------------------------
// CSR edges of the fluid particles' lists (i < nf): eoff[0..nf] = exclusive
// prefix of ncount (bsum: scratch of edge_scan_blocks(nf) ints), then
// ei/ej = (i, list entry) for every edge, self entries included.
int edge_scan_blocks(int nf);
void launch_edge_offsets(const int* ncount, int nf, int* eoff, int* bsum, cudaStream_t s);
void launch_edge_fill(const int* ncount, const int* nlist, int n, int nf, const int* eoff, int* ei, int* ej,
                      cudaStream_t s);
// `count` training samples (3 float4 each) of edges drawn at random from the
// ne CSR edges: features of the pair and its FP64 PressureA + DiffuseInterface
// + ViscosityV force on i as target (valid = 0 outside every radius or j == i)
void launch_collect(const SimConst& c, const double4* pos, const double4* press, const double4* gc,
                    const int* ei, const int* ej, long long ne, long long count, unsigned long long seed,
                    float4* out, cudaStream_t s);
// sums over fluid particles of |F_a - F_b|^2, |F_b|^2, |F_b - F_a + L|^2
void launch_force_compare(int nf, const double4* fa, const double4* fb, const float4* lsum, double* sums3,
                          cudaStream_t s);
void launch_virial(const SimConst& c, const double4* pos, const double4* vel, const double4* press,
                   const double4* gc, const int* ncount, const int* nlist, double* virial_p,
                   cudaStream_t s);
int check_division(unsigned long long seed, long long n, unsigned long long* d_count, double* d_first,
                   cudaStream_t s);
void launch_conserved(const SimConst& c, const int* cellstart, const double4* pos,
                      const double4* vel, double* out5, cudaStream_t s);

// Kernel constants of one scene from its parameters, header and set-up
// constants (mph_compute_constants), evaluated in the reference's order
// (mph_host.cpp); on failure returns the status and sets msg.
int make_simconst(const mph_params& p, const mph_grid_header& h, const mph_constants& c, int dim, int n,
                  SimConst& s, std::string& msg);

// Sets the calling thread's message for mph_last_error(NULL, ...) and returns code.
int set_thread_error(int code, const std::string& msg);

}  // namespace mph
