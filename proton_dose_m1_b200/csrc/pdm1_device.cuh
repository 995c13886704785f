// pdm1_device.cuh -- device-side data of a plan and helpers shared by the
// double-precision march (pdm1_march.cu) and the single-precision stencil
// kernels (pdm1_stage_fp32.cu).
#pragma once

#include "../../include/pdm1.h"
#include "pdm1_math.cuh"
#include "pdm1_fp64.cuh"

#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace pdm1 {

constexpr int kMaxMat = 16;
constexpr int kTileCounters = 3;   // behind the tile offsets: one per stage

// Learned moving box: proposer network 16 -> 64 -> 64 -> 6 (ReLU).
constexpr int kFeat = 16, kHid = 64, kOut = 6, kOutPad = 8;
constexpr int kParams = kHid * kFeat + kHid + kHid * kHid + kHid + kOut * kHid + kOut;

// Device form of a box model: BF16 weights [out][in] (the column-major B
// operand of mma.m16n8k16), FP32 biases, input normalisation and the map of
// the network's outputs to margins in cells.
struct BoxModelDev {
    __nv_bfloat16 W1[kHid * kFeat];
    __nv_bfloat16 W2[kHid * kHid];
    __nv_bfloat16 W3[kOutPad * kHid];
    float b1[kHid], b2[kHid], b3[kOutPad];
    float x_mean[kFeat], x_inv_std[kFeat];
    float y_scale[kOut], y_offset[kOut];
    int margin_min, margin_max, grow_cells, extra_max;
    double leak_tol;
};

int pack_box_model(const pdm1_box_model *m, BoxModelDev &out);

// Spacings whose quotients pdm1_fp64.cuh may take without the IEEE routine.
inline bool near_spacing(double h) { return h >= 0x1p-200 && h <= 0x1p200; }

enum { ERR_DEV_RANGE = 1, ERR_DEV_MAXSTEPS = 2, ERR_DEV_NONFINITE = 4, ERR_DEV_CAPACITY = 8, ERR_DEV_TIMEOUT = 16 };
// ---------------------------------------------------------------------------
// Device-side plan data
// ---------------------------------------------------------------------------
struct MatDev {
    TableView sp, tr, nuc;
    double density, X0;
};

// A rectangular domain of the full grid: the whole grid, or the moving active box
// (numerics/moving_active_domain.py), with its tile decomposition.
struct DomainDev {
    int i0, j0, k0;          // origin in the full grid
    int nx, ny, nz;          // extent
    int tx, ty, tz;          // tile shape of the stage kernels
    int tiles_y, tiles_z, ntiles;
    int inflow;              // the domain's z-min face is the beam entrance (k0 == 0)
};

// Tile shape (cells) of the stage kernels.
struct TileDims {
    int x, y, z;
};

// One pencil beam of a march (numerics/boundary.py:63-114): spectrum, angular
// spread, transverse profile on the grid's z-min face, initial moving box.
struct BeamDev {
    double E_beam, sigma_E, rf;     // rf = exp(-angular_spread^2)
    const double *spatial;          // (nx, ny): n_protons * normalised profile
    DomainDev init_box;             // moving_active_domain.py:35-60
};

constexpr int kStepsPerGraph = 32;

// What the host polls between graph replays.
struct MarchSummary {
    int active;         // beams that marched in the last step
    int error;          // OR of the beams' error flags
    // per step of the replay: the nanosecond clock when the first stage's first CTA begins
    // and when the last stage's last CTA ends
    unsigned long long begin_ns[kStepsPerGraph], end_ns[kStepsPerGraph];
};

struct ConfigDev {
    int nx, ny, nz;
    double dx, dy, dz;
    double inv_dx, inv_dy, inv_dz;   // their reciprocals, for the divergence
    int spacing_near;                // the spacings are in the range of quotient()
    int nm;
    int scattering, nuclear, interp, scheme, unit_speeds;
    int cfl_floor;       // moving box: CFL bound at least the phantom's vacuum bound
    unsigned present;    // bit m: material m occurs in the phantom
    int spatial;         // PDM1_SPATIAL_*: the reconstruction
    int stencil_radius;  // its ghost width (vacuum-aware CFL masks)
    int use_if;          // integrating factors active (IF_SSPRK3 with sources)
    int strang;          // Strang-split sources around an SSPRK3 / Euler step
    double cfl, max_dE, Emin;
    int max_steps;
    int step_limit;      // >= 0: stop (without error) after this many steps
    int n_targets;
    const int32_t *ids;
    const double *targets;      // descending
    // beams: per-beam buffers hold `cap` cells each (the beam's domain)
    int nbeams;
    size_t cap;
    const BeamDev *beams;
    int *tile_off;              // (nbeams + 1) prefix sums of the active beams' tiles, then the
                                // tiles handed out beyond the grid's first in stages A, B, C
    MarchSummary *summary;
    // moving active box
    int moving, vacuum_aware, guard;
    double tol;                 // exp(-sigma_trunc^2 / 2)
    double *bufA, *bufB;        // compact-state ping-pong, 4*cap per beam
    unsigned long long *slab;   // max phi per x | y | z slab of the box (double bits), per beam
    unsigned char *active;      // vacuum-aware activity mask on the box, cap per beam
    int grid_ctas;              // persistent grid of the stage kernels
    TileDims tile;              // tile shape of the stage kernels (kTiles[tile_id])
    int tile_id;
    int fp32;                   // FP32-stencil form: float eigenvalues in the CFL bound (not with cfl_floor)
    int bulk_stage;             // FP32 form: stages B and C stage their float4 source by bulk copies
    const double *schedule;     // prescribed energies E_0 .. E_{n-1} (replaces the CFL step), or NULL
    int n_schedule;
    // learned moving box and training-data recorder
    int learned;                // a box model proposes the margins
    const BoxModelDev *model;
    double *acc;                // per beam kAcc doubles: fluence moments and face currents of the box
    double *plane;              // per beam nz doubles: current through each z plane of the box
    float *rec;                 // recorder rows (one-beam full-domain plans), or NULL
    int rec_max;
    double rec_tail_tol[2];     // recorder: the two fluence-tail thresholds
    double density[kMaxMat];
    MatDev mats[kMaxMat];
};

// Layout of a beam's accumulator (cell coordinates are global cell centres,
// in cells): sums over the box of phi, phi x, phi y, phi z, phi x^2, phi y^2,
// phi z^2, Jx, Jy, Jz, |Jx|, |Jy|, then the current |J.n| summed over the
// cells of the box faces x-, x+, y-, y+, z-, z+ that lie inside the phantom
// (the entrance face excluded), then max phi.
enum { ACC_M = 0, ACC_X = 1, ACC_X2 = 4, ACC_J = 7, ACC_JABS = 10, ACC_FACE = 12, ACC_MAX = 18, kAcc = 20 };

struct Coeffs {
    double E, dE, E_next;
    int active;
    int snap_slot;
    double S0[kMaxMat], S1[kMaxMat], S2[kMaxMat];
    double c1p[kMaxMat], c1c[kMaxMat], c1ip[kMaxMat], c1ic[kMaxMat];
    double c2p[kMaxMat], c2c[kMaxMat], c2ip[kMaxMat], c2ic[kMaxMat];
    double Sb[4][kMaxMat];                  // S at E, E-dE/3, E-2dE/3, E-dE
    double fip[4][kMaxMat], fic[4][kMaxMat];   // inverse factors at those depths
    double ed[4];                           // spectrum at those energies
    double ed_next;                         // spectrum at E_next (CFL inflow)
    double hn[kMaxMat], hs[kMaxMat];        // Strang half-step factors
    double S_cfl[kMaxMat];                  // moving box: S at the step's start energy
    double ed_cfl;                          // moving box: spectrum at that energy
};

struct MarchState {
    double E;
    unsigned long long inv_bits;   // CFL max (non-negative double bits)
    double forced_dE;              // > 0: one step with this dE (pdm1_advance)
    int step, done, ti, taken, error;
    DomainDev dom;                 // the domain the stage kernels work on
    DomainDev prev;                // moving box before this step's rebox
    double *Ua;                    // state on `dom`
    double *Uprev;                 // state on `prev`
    int reboxed;
    unsigned long long newmax_bits;   // max phi over the new box (vacuum-aware CFL)
    double pin_max;                // max inflow phi over the new box
    double cell_steps;             // sum over steps of the cells marched (domain volume)
    double max_cells;              // largest domain marched in one step
    // learned box
    int sig[6];                    // significant box (global, half-open); sig[1] < 0: none
    double sig_scale;              // max(phi, phi_in) the threshold was taken from
    int extra[6];                  // growth per face from the outgoing-flux check
    int fallback;                  // 0 learned, 1 full domain, 2 heuristic box
    int grows;                     // faces grown by the check
    int margin[6];                 // margins of the last box
};

__host__ __device__ inline DomainDev make_domain(int i0, int j0, int k0, int nx, int ny, int nz, int inflow,
                                                 TileDims t);


// ---------------------------------------------------------------------------
// Material coefficients (device), mirroring physics/*.py
// ---------------------------------------------------------------------------
// A table at E, clipped to it (false: outside): PCHIP or numpy.interp.  The loads of
// the guessed interval go out together with those of the table's ends; a guess
// that misses (rounding of the logarithm) takes the general evaluation.
__device__ inline bool table_dev(const TableView &view, bool pchip, double E, double &out) {
    const TableView t = view;
    const int last = t.n - 1;
    int i = t.inv_log_step > 0.0 && E > 0.0 ? interval_guess(t, E) : search_right(t, E);
    i = i < 0 ? 0 : (i > last - 1 ? last - 1 : i);
    const double lo = t.E[0], hi = t.E[last], v_last = t.v[last];
    const double e0 = t.E[i], e1 = t.E[i + 1], v0 = t.v[i], v1 = t.v[i + 1];
    const double s0 = t.slope[i], s1 = t.slope[i + 1];
    if (!clip_energy(lo, hi, E)) return false;
    if (E >= hi) out = v_last;
    else if (!(e0 <= E && E < e1)) out = pchip ? pchip_eval(t, E) : linear_eval(t, E);
    else out = pchip ? pchip_interval(e0, e1, v0, v1, s0, s1, E) : linear_interval(e0, e1, v0, v1, E);
    return true;
}

__device__ inline bool stopping_power_dev(const MatDev &m, double E, double &out) {
    return table_dev(m.sp, true, E, out);
}

__device__ inline bool transport_dev(const ConfigDev &cf, const MatDev &m, double E, double &out) {
    if (cf.scattering == PDM1_SCATTERING_OFF) { out = 0.0; return true; }
    if (cf.scattering == PDM1_SCATTERING_ROSSI) {
        double e = E > 1.0e-8 ? E : 1.0e-8;
        double M = kProtonRestMev;
        double pv = e * (e + 2.0 * M) / (e + M);
        double r = kRossiEsMev / pv;
        out = r * r / m.X0;
        return true;
    }
    return table_dev(m.tr, cf.interp != PDM1_INTERP_LINEAR, E, out);
}

__device__ inline bool nuclear_dev(const ConfigDev &cf, const MatDev &m, double E, double &out) {
    return table_dev(m.nuc, cf.interp != PDM1_INTERP_LINEAR, E, out);
}

// numerics/boundary.py:82-114 spectrum factor
__device__ __forceinline__ double energy_density(const BeamDev &bm, double E) {
    double de = E - bm.E_beam;
    double s = bm.sigma_E;
    return dd_exp(-(de * de) / (2.0 * (s * s))) / (sqrt(2.0 * 3.141592653589793) * s);
}

__device__ __forceinline__ void source_factor(double ts, double tn, bool inverse, double &fp, double &fc) {
    double sign = inverse ? 1.0 : -1.0;
    double a = tn < kExpClamp ? tn : kExpClamp;
    double tsum = tn + ts;
    double b = tsum < kExpClamp ? tsum : kExpClamp;
    fp = dd_exp(sign * a);
    fc = dd_exp(sign * b);
}

// ---------------------------------------------------------------------------
// The fused stage kernel
// ---------------------------------------------------------------------------
constexpr int NT = 256;   // threads of a stage CTA

// A tile shape: the tile's cells, its cross-shaped 3-cell WENO halo (no
// corners: WENO reads along one axis at a time) and its faces.  Shared memory
// holds three arms per component, each the core plus the halo along one axis
// (the core stored three times), so every 6-point stencil is a strided run in
// one arm.
template <int X, int Y, int Z>
struct Tile {
    static constexpr int CELLS = X * Y * Z;
    static_assert(CELLS <= NT, "at most one cell per thread");
    static constexpr int TX = X, TY = Y, TZ = Z;
    static constexpr int NFX = (X + 1) * Y * Z, NFY = X * (Y + 1) * Z, NFZ = X * Y * (Z + 1);
    static constexpr int NF = NFX + NFY + NFZ;
    static constexpr int SX = (X + 6) * Y * Z;   // x-arm loads (core and x halo)
    static constexpr int SY = X * 6 * Z;         // y halo loads
    static constexpr int SZ = X * Y * 6;         // z halo loads
    static constexpr int AX = (X + 6) * Y * Z;   // arm sizes per component
    static constexpr int AY = X * (Y + 6) * Z;
    static constexpr int AZ = X * Y * (Z + 6);
    template <typename T>
    static constexpr size_t arm_bytes() {
        return sizeof(T) * 4 * (AX + AY + AZ + NF);
    }
};

// The tile shapes the stage kernels are built for, the autotuner's candidates.
// (An 8x8x8 tile of 512 threads, 3.375 faces per cell against 3.5-3.7, was
// measured slower: 0.674 against 0.606 ns per cell-step on a 51-spot pelvis batch
// in the FP32 form, with half as many CTAs per SM and twice the warps per barrier.)
constexpr int kNumTiles = 3;
using Tile0 = Tile<4, 8, 8>;
using Tile1 = Tile<8, 8, 4>;
using Tile2 = Tile<2, 8, 16>;
constexpr TileDims kTiles[kNumTiles] = {{4, 8, 8}, {8, 8, 4}, {2, 8, 16}};
constexpr int kMaxTileZ = 16;

// Plans whose grids all fit one wave of the resident CTAs in 4x4x4 tiles take
// those: 240 faces for 256 threads, one round instead of the 4x8x8 tile's three and
// a half, and four times the CTAs.  Measured, one FP64 energy step: 225 small tiles
// (12x12x100) 175 -> 118 us; 480 (16x16x120, two waves) 143 -> 153 us, so the line
// lies at one wave.  FP32 form, four CTAs per SM: 480 small tiles 132 -> 101 us; 875
// (1.5 waves) 116 -> 126 us.
using SmallTile = Tile<4, 4, 4>;
constexpr int kSmallTileId = kNumTiles;
constexpr TileDims kSmallTile = {4, 4, 4};

__host__ __device__ inline DomainDev make_domain(int i0, int j0, int k0, int nx, int ny, int nz, int inflow,
                                                 TileDims t) {
    DomainDev d;
    d.i0 = i0; d.j0 = j0; d.k0 = k0;
    d.nx = nx; d.ny = ny; d.nz = nz;
    d.tx = t.x; d.ty = t.y; d.tz = t.z;
    d.tiles_y = (ny + t.y - 1) / t.y;
    d.tiles_z = (nz + t.z - 1) / t.z;
    d.ntiles = ((nx + t.x - 1) / t.x) * d.tiles_y * d.tiles_z;
    d.inflow = inflow;
    return d;
}

enum StageMode { MODE_A = 0, MODE_B = 1, MODE_C = 2, MODE_EULER = 3, MODE_RHS = 4,
                 MODE_C_LEARN = 5 };   // launch selector: stage C with the learned box's moments

struct StageArgs {
    const ConfigDev *cf;
    const Coeffs *co;   // per beam
    MarchState *st;     // per beam
    double *U1;         // stage states (on the beam's domain), 4*cap per beam
    double *U2;
    double *V;          // marched variable of stage 1 / 2
    double *qpart;      // (q0 + q1)/6 quadrature part
    double *dose;       // accumulated dose (full grid), or NULL
    double *edep;       // when non-NULL: energy deposition written instead of dose
    double *snap;       // snapshot buffer base (slot * 4N, full grid)
    unsigned long long *begin_ns, *end_ns;   // stage timing of this step, or NULL
    double *rhs_out;    // MODE_RHS output
    const double *bc_plane;   // MODE_RHS: explicit z-min boundary state (4,nx,ny)
    double rhs_energy_density;
};

template <typename T>
struct SmemT {
    T *X, *Y, *Z, *F;
};


__device__ __forceinline__ size_t global_cell(const ConfigDev &cf, const DomainDev &d, int li, int lj, int lk) {
    return ((size_t)(d.i0 + li) * cf.ny + (d.j0 + lj)) * cf.nz + (d.k0 + lk);
}

// Stencil source value at a domain cell; indices outside the domain are
// clamped (zero-gradient ghosts, numerics/boundary.py:327-397).
template <int MODE>
__device__ __forceinline__ void load_cell(const ConfigDev &cf, const Coeffs &co, const DomainDev &d,
                                          const double *src, int li, int lj, int lk, double out[4]) {
    const int nx = d.nx, ny = d.ny, nz = d.nz;
    const size_t N = (size_t)nx * ny * nz;
    li = li < 0 ? 0 : (li >= nx ? nx - 1 : li);
    lj = lj < 0 ? 0 : (lj >= ny ? ny - 1 : lj);
    lk = lk >= nz ? nz - 1 : lk;
    size_t o = ((size_t)li * ny + lj) * nz + lk;
#pragma unroll
    for (int c = 0; c < 4; ++c) out[c] = src[c * N + o];
    if ((MODE == MODE_A || MODE == MODE_EULER) && cf.strang) {
        int m = cf.ids[global_cell(cf, d, li, lj, lk)];
        double hn = co.hn[m], hs = co.hs[m];
        if (cf.nuclear)
#pragma unroll
            for (int c = 0; c < 4; ++c) out[c] *= hn;
        if (cf.scattering != PDM1_SCATTERING_OFF)
#pragma unroll
            for (int c = 1; c < 4; ++c) out[c] *= hs;
    }
}

// z-min boundary value of component c at domain column (li, lj) for this stage.
// A moving box away from the entrance has zero inflow (moving_active_domain.py:85-95).
template <int MODE>
__device__ __forceinline__ double boundary_value(const StageArgs &a, const ConfigDev &cf, const BeamDev &bm,
                                                 const Coeffs &co, const DomainDev &d, int c, int li, int lj) {
    if (MODE == MODE_RHS && a.bc_plane)
        return a.bc_plane[((size_t)c * d.nx + li) * d.ny + lj];
    if (!d.inflow || c == 1 || c == 2) return 0.0;
    const int gi = d.i0 + li, gj = d.j0 + lj;
    double sp = bm.spatial[(size_t)gi * cf.ny + gj];
    if (MODE == MODE_A || MODE == MODE_EULER || MODE == MODE_RHS) {
        double ed = MODE == MODE_RHS ? a.rhs_energy_density : co.ed[0];
        double phi = sp * ed;
        return c == 0 ? phi : bm.rf * phi;
    }
    // RK-consistent stage traces, numerics/energy.py:348-455 (107-231 without sources)
    int m = cf.ids[((size_t)gi * cf.ny + gj) * cf.nz];
    double V[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        double phi = sp * co.ed[q];
        double x = c == 0 ? phi : bm.rf * phi;
        double B = co.Sb[q][m] * x;
        if (q > 0 && cf.use_if) B *= (c == 0 ? co.fip[q][m] : co.fic[q][m]);
        V[q] = B;
    }
    if (MODE == MODE_B) {
        double vs1 = 0.5 * (-9.0 * V[0] + 18.0 * V[1] - 9.0 * V[2] + 2.0 * V[3]);
        if (cf.use_if) vs1 *= (c == 0 ? co.c1p[m] : co.c1c[m]);
        return vs1 / co.S1[m];
    }
    double vs2 = 0.25 * (11.0 * V[0] - 27.0 * V[1] + 27.0 * V[2] - 7.0 * V[3]);
    if (cf.use_if) vs2 *= (c == 0 ? co.c2p[m] : co.c2c[m]);
    return vs2 / co.S2[m];
}

// One cell's CFL term (numerics/energy.py:539-660): sum over axes of a/(S d).
// `entrance`: the cell is on the domain's z-min layer, where the inflow state
// (zero for a box away from the entrance) joins the z speeds.
// T: the precision of the eigenvalues -- double for the FP64 march, float for
// the FP32-stencil form (its step sequence need not match the FP64 one).
template <typename T>
__device__ __forceinline__ double cfl_term(const ConfigDev &cf, double rf, const double u[4], double s,
                                           bool entrance, double phi_in, const bool use[3]) {
    double a0, a1, a2;
    if (cf.unit_speeds) {
        a0 = a1 = a2 = 1.0;
    } else {
        const T p = T(u[0]), x = T(u[1]), y = T(u[2]), z = T(u[3]);
        T a[3];
        if constexpr (sizeof(T) == sizeof(double)) speeds3_64(u, a);
        else max_abs_speeds3(p, x, y, z, a);
        a0 = double(a[0]);
        a1 = double(a[1]);
        a2 = double(a[2]);
        if (entrance) {
            T pin = T(phi_in);
            T jz = T(rf) * pin;
            double ain = double(max_abs_speed(pin, T(0), T(0), jz, 2));
            if (ain > a2) a2 = ain;
        }
    }
    if (!use[0]) a0 = 0.0;
    if (!use[1]) a1 = 0.0;
    if (!use[2]) a2 = 0.0;
    const double b0 = s * cf.dx, b1 = s * cf.dy, b2 = s * cf.dz;
    if constexpr (sizeof(T) == sizeof(double)) {
        // speeds are 0 (masked) or above 1e-6, so the quotients are in range when the divisors are
        auto in = [](double b) { return abs_hi(b) - exp_word(-200) < exp_word(200) - exp_word(-200); };
        if (in(b0) && in(b1) && in(b2) && a0 <= 2.0 && a1 <= 2.0 && a2 <= 2.0)
            return quotient(a0, b0, rcp_near(b0)) + quotient(a1, b1, rcp_near(b1)) + quotient(a2, b2, rcp_near(b2));
    }
    return a0 / b0 + a1 / b1 + a2 / b2;
}

template <int THREADS = NT>
__device__ __forceinline__ void block_max_atomic(double v, unsigned long long *target) {
    // v >= 0 or NaN; NaN never wins (fmax), like the oracle's comparison loop
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    __shared__ double wmax[THREADS / 32];
    int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) wmax[w] = v;
    __syncthreads();
    if (w == 0) {
        v = l < THREADS / 32 ? wmax[l] : 0.0;
        for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (l == 0 && v > 0.0) atomicMax(target, (unsigned long long)__double_as_longlong(v));
    }
}

__device__ __forceinline__ void atomic_max_double(unsigned long long *target, double v) {
    if (v > 0.0) atomicMax(target, (unsigned long long)__double_as_longlong(v));
}

// The recorder's per-slab maxima of phi over one tile: cell values in `buf`
// (one per cell of the tile, (i, j, k) with k fastest; -1 outside the box).
__device__ __forceinline__ void tile_slab_max(const ConfigDev &cf, unsigned long long *slab, const DomainDev &d,
                                              const double *buf, int i0, int j0, int k0) {
    int t = threadIdx.x;
    const int TX = d.tx, TY = d.ty, TZ = d.tz;
    unsigned long long *sx = slab, *sy = slab + cf.nx, *sz = slab + cf.nx + cf.ny;
    if (t < TX) {
        double m = 0.0;
        for (int e = 0; e < TY * TZ; ++e) m = fmax(m, buf[t * TY * TZ + e]);
        if (i0 + t < d.nx) atomic_max_double(&sx[i0 + t], m);
    } else if (t < TX + TY) {
        int j = t - TX;
        double m = 0.0;
        for (int i = 0; i < TX; ++i)
            for (int k = 0; k < TZ; ++k) m = fmax(m, buf[(i * TY + j) * TZ + k]);
        if (j0 + j < d.ny) atomic_max_double(&sy[j0 + j], m);
    } else if (t < TX + TY + TZ) {
        int k = t - TX - TY;
        double m = 0.0;
        for (int i = 0; i < TX; ++i)
            for (int j = 0; j < TY; ++j) m = fmax(m, buf[(i * TY + j) * TZ + k]);
        if (k0 + k < d.nz) atomic_max_double(&sz[k0 + k], m);
    }
}

// Per-slab maxima of phi over one stage tile (moving box) from each thread's value
// (-1 outside the box): warp maxima over k, over j and k, and over j, then the few
// values per slab from shared memory.  (One thread per slab reading the tile's 64
// values in turn held the CTA for about 2000 cycles a tile.)
template <class Tl>
struct SlabScratch {
    static constexpr int JL = Tl::TY < 32 / Tl::TZ ? Tl::TY : 32 / Tl::TZ;   // j values of a warp
    double x[Tl::CELLS / (Tl::TZ * JL)], y[Tl::TX * Tl::TY], z[Tl::CELLS / 32][Tl::TZ];
};
template <class Tl>
__device__ __forceinline__ void stage_slab_max(const ConfigDev &cf, unsigned long long *slab, const DomainDev &d,
                                               double phi, int i0, int j0, int k0, SlabScratch<Tl> &s) {
    constexpr int TX = Tl::TX, TY = Tl::TY, TZ = Tl::TZ, JL = SlabScratch<Tl>::JL;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (Tl::CELLS == NT || warp < Tl::CELLS / 32) {
        double row = phi, z = phi;
#pragma unroll
        for (int w = 1; w < TZ; w <<= 1) row = fmax(row, __shfl_xor_sync(0xffffffffu, row, w));
        double x = row;
#pragma unroll
        for (int w = TZ; w < TZ * JL; w <<= 1) x = fmax(x, __shfl_xor_sync(0xffffffffu, x, w));
#pragma unroll
        for (int w = TZ; w < 32; w <<= 1) z = fmax(z, __shfl_xor_sync(0xffffffffu, z, w));
        if (lane % TZ == 0) s.y[t / TZ] = row;
        if (lane % (TZ * JL) == 0) s.x[t / (TZ * JL)] = x;
        if (lane < TZ) s.z[warp][lane] = z;
    }
    __syncthreads();
    double m = 0.0;
    if (t < TX) {
#pragma unroll
        for (int e = 0; e < TY / JL; ++e) m = fmax(m, s.x[t * (TY / JL) + e]);
        if (i0 + t < d.nx) atomic_max_double(&slab[i0 + t], m);
    } else if (t >= 32 && t < 32 + TY) {
        const int j = t - 32;
#pragma unroll
        for (int i = 0; i < TX; ++i) m = fmax(m, s.y[i * TY + j]);
        if (j0 + j < d.ny) atomic_max_double(&slab[cf.nx + j0 + j], m);
    } else if (t >= 64 && t < 64 + TZ) {
        const int k = t - 64;
#pragma unroll
        for (int w = 0; w < Tl::CELLS / 32; ++w) m = fmax(m, s.z[w][k]);
        if (k0 + k < d.nz) atomic_max_double(&slab[cf.nx + cf.ny + k0 + k], m);
    }
}

// Beam owning global tile t of the step: tile_off holds the exclusive prefix
// sums of the beams' tile counts (beams that do not march have none).
__device__ __forceinline__ int beam_of_tile(const int *tile_off, int nbeams, int t) {
    int lo = 0, hi = nbeams - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (tile_off[mid] <= t) lo = mid; else hi = mid - 1;
    }
    return lo;
}

__device__ __forceinline__ unsigned long long *beam_slab(const ConfigDev &cf, int b) {
    return cf.slab + (size_t)b * (cf.nx + cf.ny + cf.nz);
}

// Learned box: one tile's contribution to the beam's fluence moments, face
// currents and z-plane currents (acc, plane) from the state u of each cell
// (cell (li, lj, lk) of domain d, `valid` inside it; the tile begins at (i0, j0, k0)).
// Called by every thread of a CTA of THREADS threads laid out as the stage tile (k
// fastest, a power of two); `part` and `pl` are shared scratch.  The twelve sums go
// through one butterfly that halves the values a lane holds as it doubles the lanes
// they cover (16 exchanges of a double instead of 5 per sum); the face currents are
// summed only in tiles that touch a face; a plane's current by the lanes that share k.
// With 19 separate warp sums and one shared-memory atomic per cell the learned
// stage C took 1.36 times the time of stage B on the 256x256x320 field.
template <int THREADS = NT>
__device__ __forceinline__ void tile_moments_cta(const ConfigDev &cf, int b, const DomainDev &d, int i0, int j0,
                                                 int k0, bool valid, int li, int lj, int lk, const double u[4],
                                                 double (*part)[ACC_MAX + 1], double (*pl)[kMaxTileZ]) {
    constexpr int kSums = ACC_MAX, kPlain = ACC_FACE, WARPS = THREADS / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool faces = (i0 == 0 && d.i0 > 0) || (i0 + d.tx >= d.nx && d.i0 + d.nx < cf.nx) ||
                       (j0 == 0 && d.j0 > 0) || (j0 + d.ty >= d.ny && d.j0 + d.ny < cf.ny) ||
                       (k0 == 0 && d.k0 > 0) || (k0 + d.tz >= d.nz && d.k0 + d.nz < cf.nz);
    const double phi = valid ? u[0] : 0.0, jx = valid ? u[1] : 0.0, jy = valid ? u[2] : 0.0, jz = valid ? u[3] : 0.0;
    double m = phi;
    {
        const double gx = d.i0 + li + 0.5, gy = d.j0 + lj + 0.5, gz = d.k0 + lk + 0.5;
        const double px = phi * gx, py = phi * gy, pz = phi * gz;
        double v[16] = {phi, px, py, pz, px * gx, py * gy, pz * gz, jx, jy, jz, fabs(jx), fabs(jy), 0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int w = 8; w > 0; w >>= 1) {
            const bool up = (lane & w) != 0;
#pragma unroll
            for (int q = 0; q < w; ++q) {
                const double keep = up ? v[q + w] : v[q], send = up ? v[q] : v[q + w];
                v[q] = keep + __shfl_xor_sync(0xffffffffu, send, w);
            }
        }
        v[0] += __shfl_xor_sync(0xffffffffu, v[0], 16);   // lane l: the warp's sum of value l & 15
        if (lane < kPlain) part[warp][lane] = v[0];
    }
    for (int w = 16; w > 0; w >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, w));
    if (lane == 0) part[warp][kSums] = m;
    if (faces) {
        double f[6];
        f[0] = li == 0 && d.i0 > 0 ? fabs(jx) : 0.0;
        f[1] = li == d.nx - 1 && d.i0 + d.nx < cf.nx ? fabs(jx) : 0.0;
        f[2] = lj == 0 && d.j0 > 0 ? fabs(jy) : 0.0;
        f[3] = lj == d.ny - 1 && d.j0 + d.ny < cf.ny ? fabs(jy) : 0.0;
        f[4] = lk == 0 && d.k0 > 0 ? fabs(jz) : 0.0;
        f[5] = lk == d.nz - 1 && d.k0 + d.nz < cf.nz ? fabs(jz) : 0.0;
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            for (int w = 16; w > 0; w >>= 1) f[q] += __shfl_xor_sync(0xffffffffu, f[q], w);
            if (lane == 0) part[warp][ACC_FACE + q] = f[q];
        }
    }
    double z = jz;
    for (int w = d.tz; w < 32; w <<= 1) z += __shfl_xor_sync(0xffffffffu, z, w);
    if (lane < d.tz) pl[warp][lane] = z;
    __syncthreads();
    double *acc = cf.acc + (size_t)b * kAcc;
    if (tid < (faces ? kSums : kPlain)) {
        double s = 0.0;
        for (int w = 0; w < WARPS; ++w) s += part[w][tid];
        if (s != 0.0) atomicAdd(&acc[tid], s);
    } else if (tid == kSums) {
        m = 0.0;
        for (int w = 0; w < WARPS; ++w) m = fmax(m, part[w][kSums]);
        atomic_max_double(reinterpret_cast<unsigned long long *>(&acc[ACC_MAX]), m);
    } else if (tid >= 32 && tid < 32 + d.tz) {
        const int k = tid - 32;
        double s = 0.0;
        for (int w = 0; w < WARPS; ++w) s += pl[w][k];
        if (k0 + k < d.nz && s != 0.0) atomicAdd(&cf.plane[(size_t)b * cf.nz + d.k0 + k0 + k], s);
    }
    __syncthreads();
}

// The significant box of desired_box (moving_active_domain.py:107-151):
// scale = max(max phi, max phi_in) (phi_in only while the domain touches
// z = 0), then the first and last x / y / z slab of `d` whose max phi exceeds
// tol * scale (the plan's tolerance for the moving box), an inflow cell above
// it joining the k = 0 layer.  Called by all threads of a CTA of 256 (8
// warps) with `red` = 16 doubles of shared memory; results (local indices,
// hi < 0 when none) in the caller's shared memory.
__device__ inline void significant_box_cta(const ConfigDev &cf, const BeamDev &bm, const DomainDev &d,
                                           const unsigned long long *slab, double ed, double *red, int *s_lo,
                                           int *s_hi, double *s_scale, double tol) {
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const unsigned long long *sx = slab, *sy = slab + cf.nx, *sz = slab + cf.nx + cf.ny;
    auto as_d = [](unsigned long long b) { return __longlong_as_double((long long)b); };
    auto inflow = [&](int i, int j) { return bm.spatial[(size_t)(d.i0 + i) * cf.ny + (d.j0 + j)] * ed; };
    // the state's maximum (slab maxima) and the inflow's over the box's entrance
    double m = 0.0, mi = 0.0;
    for (int i = t; i < d.nx; i += 256) m = fmax(m, as_d(sx[i]));
    if (d.inflow)
        for (int i = warp; i < d.nx; i += 8)
            for (int j = lane; j < d.ny; j += 32) mi = fmax(mi, inflow(i, j));
    for (int w = 16; w > 0; w >>= 1) {
        m = fmax(m, __shfl_xor_sync(0xffffffffu, m, w));
        mi = fmax(mi, __shfl_xor_sync(0xffffffffu, mi, w));
    }
    if (lane == 0) { red[warp] = m; red[8 + warp] = mi; }
    if (t < 3) { s_lo[t] = 0x7fffffff; s_hi[t] = -1; }
    __syncthreads();
    m = mi = 0.0;
    for (int w = 0; w < 8; ++w) { m = fmax(m, red[w]); mi = fmax(mi, red[8 + w]); }
    const double scale = fmax(m, mi);
    if (t == 0) *s_scale = scale;
    const double thr = tol * scale;
    // an inflow cell above the threshold exists iff the inflow's maximum is above it
    const bool inflow_on = d.inflow && mi > thr;
    if (scale != 0.0) {
        // one thread per slab: its maximum above the threshold, or the k = 0 layer under
        // an inflow above it
        auto scan = [&](const unsigned long long *sl, int n, int ax, bool first) {
            for (int base = 32 * warp; base < n; base += 256) {
                const int i = base + lane;
                const bool act = i < n && (as_d(sl[i]) > thr || (first && i == 0));
                const unsigned mask = __ballot_sync(0xffffffffu, act);
                if (lane == 0 && mask) {
                    atomicMin(&s_lo[ax], base + __ffs(mask) - 1);
                    atomicMax(&s_hi[ax], base + 31 - __clz(mask));
                }
            }
        };
        scan(sx, d.nx, 0, false);
        scan(sy, d.ny, 1, false);
        scan(sz, d.nz, 2, inflow_on);
        if (inflow_on) {
            // one warp per x slab (y slab): any inflow cell of its entrance row above the threshold
            for (int i = warp; i < d.nx; i += 8) {
                bool any = false;
                for (int j = lane; j < d.ny; j += 32) any = any || inflow(i, j) > thr;
                if (__any_sync(0xffffffffu, any) && lane == 0) { atomicMin(&s_lo[0], i); atomicMax(&s_hi[0], i); }
            }
            for (int j = warp; j < d.ny; j += 8) {
                bool any = false;
                for (int i = lane; i < d.nx; i += 32) any = any || inflow(i, j) > thr;
                if (__any_sync(0xffffffffu, any) && lane == 0) { atomicMin(&s_lo[1], j); atomicMax(&s_hi[1], j); }
            }
        }
    }
    __syncthreads();
}

// Switch a beam to the box `nb` (one thread): the capacity check, the
// compact-state ping-pong, the spectrum for the CFL bound and, for the
// vacuum-aware CFL (energy.py:496-537), the max inflow over the new box
// (`with_pin`; box_kernel takes that with its whole CTA).
__device__ inline void switch_box(const ConfigDev &cf, const BeamDev &bm, Coeffs *co, MarchState *st, int b,
                                  DomainDev nb, double ed, bool with_pin = true) {
    const DomainDev d = st->dom;
    bool same = nb.i0 == d.i0 && nb.j0 == d.j0 && nb.k0 == d.k0 && nb.nx == d.nx && nb.ny == d.ny && nb.nz == d.nz;
    if (!same && (size_t)nb.nx * nb.ny * nb.nz > cf.cap) {
        st->error |= ERR_DEV_CAPACITY;   // the box outgrew the beam's buffers
        same = true;
    }
    st->reboxed = same ? 0 : 1;
    if (!same) {
        st->prev = d;
        st->Uprev = st->Ua;
        double *a_buf = cf.bufA + 4 * (size_t)b * cf.cap, *b_buf = cf.bufB + 4 * (size_t)b * cf.cap;
        st->Ua = st->Ua == a_buf ? b_buf : a_buf;
        st->dom = nb;
    }
    st->inv_bits = 0ull;
    co->ed_cfl = ed;
    st->newmax_bits = 0ull;
    double pin = 0.0;
    if (with_pin && cf.vacuum_aware && nb.inflow)
        for (int e = 0; e < nb.nx * nb.ny; ++e)
            pin = fmax(pin, bm.spatial[(size_t)(nb.i0 + e / nb.ny) * cf.ny + (nb.j0 + e % nb.ny)] * ed);
    st->pin_max = pin;
}

// Learned box and recorder kernels (pdm1_box.cu).
void launch_box_moments(const ConfigDev *d_cf, const MarchState *d_st, int grid, int record, cudaStream_t stream);
void launch_box_learn(const ConfigDev *d_cf, Coeffs *d_co, MarchState *d_st, int nbeams, cudaStream_t stream);
void launch_record(const ConfigDev *d_cf, const Coeffs *d_co, MarchState *d_st, cudaStream_t stream);

// Record an error message for pdm1_last_error() and return `code`.
int report_error(int code, const char *msg);

// The plans' caching allocator (pdm1_pool.cu): device blocks of the current
// device and pinned host blocks, reused by size; pool_free of a pointer the
// pool did not hand out is ignored.
cudaError_t pool_malloc(void **ptr, size_t bytes);
// The buffers of one call in one block, its size the next power of two: however many
// sizes a program calls with, the blocks kept of them are less than twice the largest
// (one size each kept 311 MB after analytical doses of ten grids, the largest of 49 MB).
cudaError_t pool_malloc_workspace(void **ptr, size_t bytes);
cudaError_t pool_malloc_host(void **ptr, size_t bytes);
void pool_free(void *ptr);

// Single-precision stencil kernels (pdm1_stage_fp32.cu, compiled with fast math).
int stage_fp32_set_attributes();
void launch_stage_fp32(int mode, int tile_id, int grid, const StageArgs &a, cudaStream_t stream);

}  // namespace pdm1
