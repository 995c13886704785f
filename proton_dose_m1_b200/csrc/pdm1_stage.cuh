// pdm1_stage.cuh -- the fused IF-SSPRK3 stage kernel, templated on the
// arithmetic of the stencil (WENO-Z, interface projection, HLL, divergence):
// double in pdm1_march.cu, float in pdm1_stage_fp32.cu.  The stage update,
// cell projection, CFL bound and dose stay in double in both.
#pragma once

#include "pdm1_device.cuh"

namespace pdm1 {

// Element e of component c's copy of an arm of asz elements.  Double arms are
// [c][e]; float arms hold a cell's four components together, [e][c] (one
// float4 per cell, the layout of the FP32 form's stage states in HBM), so a
// 128-bit load brings (phi, Jx) and (Jy, Jz) into two packed f32x2 pairs.
template <typename T>
__device__ __forceinline__ T &arm_at(T *arm, int asz, int c, int e) {
    if constexpr (sizeof(T) == sizeof(float)) return arm[e * 4 + c];
    else return arm[c * asz + e];
}

// The FP32 form keeps its stage states U1, U2 as one float4 (phi, Jx, Jy, Jz)
// per cell: stage A writes U1, stage B reads U1 and writes U2, stage C reads
// U2.  The stencil reads them in float in any case, so storing them rounded
// changes no result; the state itself (U^n, V) and the dose stay in double.
template <typename T, int MODE>
constexpr bool kF4Source = sizeof(T) == sizeof(float) && (MODE == MODE_B || MODE == MODE_C);
template <typename T, int MODE>
constexpr bool kF4Dest = sizeof(T) == sizeof(float) && (MODE == MODE_A || MODE == MODE_B);

// ---------------------------------------------------------------------------
// Bulk staging of a float4 tile (cp.async.bulk, the TMA engine's untiled
// copy, completed on a shared-memory mbarrier).  Every z row of every arm is
// one contiguous copy of 16-byte cells; rows outside the domain in x or y
// are the clamped rows (zero-gradient ghosts, numerics/boundary.py:327-397),
// rows are clipped to [0, nz) in z and the z-max ghosts patched afterwards.
// No multicast: each CTA copies from this GPU's own memory into its own
// shared memory.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned long long *bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(unsigned long long *bar, unsigned bytes) {
    asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(unsigned long long *bar) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" ::"r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(unsigned long long *bar, unsigned parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(smem_u32(bar)), "r"(parity)
                 : "memory");
    return ok != 0;
}

// One row: `bytes` (a multiple of 16) from 16-byte aligned global memory to
// 16-byte aligned shared memory, counted on `bar`.
__device__ __forceinline__ void bulk_row(void *dst, const void *src, unsigned bytes, unsigned long long *bar) {
    mbar_expect_tx(bar, bytes);
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

// Issue the rows of one tile (x arm with its x halo, y arm, z arm), each
// thread its share, then arrive once.  The x and y arms hold the tile's own
// z range k0 .. k0 + TZ - 1, the z arm k0 - 3 .. k0 + TZ + 2.
template <class Tl>
__device__ __forceinline__ void bulk_stage_tile(const float4 *src, const DomainDev &d, int i0, int j0, int k0,
                                                float4 *X, float4 *Y, float4 *Z, unsigned long long *bar) {
    constexpr int TX = Tl::TX, TY = Tl::TY, TZ = Tl::TZ;
    constexpr int RX = (TX + 6) * TY, RY = TX * (TY + 6), RZ = TX * TY;
    const int nx = d.nx, ny = d.ny, nz = d.nz;
    // shared memory read or written by the threads before (the last tile) is
    // overwritten by the async proxy next
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    for (int r = threadIdx.x; r < RX + RY + RZ; r += NT) {
        int li, lj, ka, kb, dst_e;
        float4 *arm;
        if (r < RX) {
            const int j = r % TY, ii = r / TY;
            li = i0 + ii - 3; lj = j0 + j; ka = k0; kb = k0 + TZ;
            arm = X; dst_e = (ii * TY + j) * TZ;
        } else if (r < RX + RY) {
            const int q = r - RX, jj = q % (TY + 6), i = q / (TY + 6);
            li = i0 + i; lj = j0 + jj - 3; ka = k0; kb = k0 + TZ;
            arm = Y; dst_e = (i * (TY + 6) + jj) * TZ;
        } else {
            const int q = r - RX - RY, j = q % TY, i = q / TY;
            li = i0 + i; lj = j0 + j; ka = k0 - 3; kb = k0 + TZ + 3;
            arm = Z; dst_e = (i * TY + j) * (TZ + 6);
        }
        li = li < 0 ? 0 : (li >= nx ? nx - 1 : li);
        lj = lj < 0 ? 0 : (lj >= ny ? ny - 1 : lj);
        const int k_lo = ka < 0 ? 0 : ka, k_hi = kb > nz ? nz : kb;
        if (k_hi > k_lo)
            bulk_row(arm + dst_e + (k_lo - ka), src + ((size_t)li * ny + lj) * nz + k_lo,
                     (unsigned)(k_hi - k_lo) * 16u, bar);
    }
    mbar_arrive(bar);
}

// Wait for the tile's rows; a wait past ~2^31 cycles (about a second) flags
// ERR_DEV_TIMEOUT and lets the march end with an error instead of hanging.
__device__ __forceinline__ void bulk_wait(unsigned long long *bar, unsigned parity, int *error) {
    const long long t0 = clock64();
    while (!mbar_try_wait(bar, parity)) {
        if (clock64() - t0 > (1ll << 31)) {
            atomicOr(error, ERR_DEV_TIMEOUT);
            return;
        }
    }
}

// z-max ghosts of the z arm of a tile whose z range passes nz: the cells
// beyond hold the last cell's value (zero gradient).
template <class Tl>
__device__ __forceinline__ void patch_zmax(const DomainDev &d, int k0, float4 *Z) {
    constexpr int TX = Tl::TX, TY = Tl::TY, TZ = Tl::TZ;
    const int over = k0 + TZ + 3 - d.nz;   // cells of each z-arm row beyond nz
    if (over <= 0) return;
    const int last = d.nz - 1 - (k0 - 3);   // arm index of the domain's last z cell
    for (int e = threadIdx.x; e < TX * TY * over; e += NT) {
        const int row = e / over, kk = last + 1 + e % over;
        Z[row * (TZ + 6) + kk] = Z[row * (TZ + 6) + last];
    }
}

// Shared memory of a stage CTA ahead of the tile's arms and fluxes (all of it
// dynamic).
struct StageShared {
    double slab[208];                // moving box: the tile's slab maxima (SlabScratch)
    double mom_part[NT / 32][ACC_MAX + 1];   // learned box: moments of the new state
    double mom_pl[NT / 32][kMaxTileZ];
    unsigned long long stage_bar;    // FP32 stages B and C: the tile's bulk copies
    int next_tile[2];                // the CTA's next tile, by the parity of the tile it is on
};
static_assert(sizeof(StageShared) % 16 == 0, "the arms behind it are 16-byte aligned");

template <typename T, class Tl>
constexpr size_t stage_smem_bytes() { return sizeof(StageShared) + Tl::template arm_bytes<T>(); }

// One tile of beam b: stage the source, the faces, the stage update.  A tile of
// Tl::CELLS cells is worked on by NT threads.
template <typename T, int MODE, class Tl, bool LEARN>
__device__ __forceinline__ void stage_tile(const StageArgs &a, const ConfigDev &cf, const DomainDev &d, int b, int tile,
                                           unsigned bar_phase, double &cta_inv) {
    constexpr int TX = Tl::TX, TY = Tl::TY, TZ = Tl::TZ;
    constexpr int NF = Tl::NF, NFX = Tl::NFX, NFY = Tl::NFY;
    constexpr int SX = Tl::SX, SY = Tl::SY, SZ = Tl::SZ;
    constexpr int AX = Tl::AX, AY = Tl::AY, AZ = Tl::AZ;
    constexpr bool kNear = sizeof(T) == sizeof(double);   // pdm1_fp64.cuh's branch-free face path
    extern __shared__ __align__(16) unsigned char smem_raw[];
    StageShared &sh = *reinterpret_cast<StageShared *>(smem_raw);
    SmemT<T> s;
    s.X = reinterpret_cast<T *>(smem_raw + sizeof(StageShared));   // [c][i + 3][j][k]  (float: [i + 3][j][k][c], arm_at)
    s.Y = s.X + 4 * AX;    // [c][i][j + 3][k]
    s.Z = s.Y + 4 * AY;    // [c][i][j][k + 3]
    s.F = s.Z + 4 * AZ;
    int tid = threadIdx.x;
    asm volatile("" : "+r"(tid));   // the indices that follow from it are formed per tile: hoisted, they spill
    const bool unit = cf.unit_speeds != 0;
    const bool all_axes[3] = {true, true, true};
    const Coeffs &co = a.co[b];
    MarchState &stb = a.st[b];
    const BeamDev &bm = cf.beams[b];
    double *const Ua = stb.Ua;
    const int nx = d.nx, ny = d.ny, nz = d.nz;
    const size_t N = (size_t)nx * ny * nz;
    const size_t boff = (size_t)b * cf.cap;
    double *const U1 = a.U1 + 4 * boff;
    double *const U2 = a.U2 + 4 * boff;
    double *const Vb = a.V + 4 * boff;
    double *const qb = a.qpart + boff;
    const double *src = (MODE == MODE_B) ? U1 : (MODE == MODE_C ? U2 : Ua);
    const int tz = tile % d.tiles_z, ty = (tile / d.tiles_z) % d.tiles_y, tx = tile / (d.tiles_z * d.tiles_y);
    const int i0 = tx * TX, j0 = ty * TY, k0 = tz * TZ;

    // ---- 1. stage the stencil source + halo (the core into all three arms) ----
    int out_of_range = 0;   // a staged value lies outside weno_range
    if constexpr (kF4Source<T, MODE>) {
        // the float4 stage state: bulk copies, or (bulk_stage == 0) one
        // 128-bit load per cell; the arms receive the same values either way
        const float4 *src4 = reinterpret_cast<const float4 *>(src);
        float4 *X4 = reinterpret_cast<float4 *>(s.X), *Y4 = reinterpret_cast<float4 *>(s.Y);
        float4 *Z4 = reinterpret_cast<float4 *>(s.Z);
        if (cf.bulk_stage) {
            bulk_stage_tile<Tl>(src4, d, i0, j0, k0, X4, Y4, Z4, &sh.stage_bar);
            bulk_wait(&sh.stage_bar, bar_phase, &stb.error);
            patch_zmax<Tl>(d, k0, Z4);
        } else {
            auto cell = [&](int li, int lj, int lk) {
                li = li < 0 ? 0 : (li >= nx ? nx - 1 : li);
                lj = lj < 0 ? 0 : (lj >= ny ? ny - 1 : lj);
                lk = lk >= nz ? nz - 1 : lk;
                return src4[((size_t)li * ny + lj) * nz + lk];
            };
            for (int e = tid; e < SX; e += NT) {
                const int k = e % TZ, j = (e / TZ) % TY, ii = e / (TZ * TY);
                const float4 v = cell(i0 + ii - 3, j0 + j, k0 + k);
                X4[(ii * TY + j) * TZ + k] = v;
                if (ii >= 3 && ii < TX + 3) {
                    Y4[((ii - 3) * (TY + 6) + j + 3) * TZ + k] = v;
                    Z4[((ii - 3) * TY + j) * (TZ + 6) + k + 3] = v;
                }
            }
            for (int e = tid; e < SY; e += NT) {
                const int k = e % TZ, jj = (e / TZ) % 6, i = e / (TZ * 6);
                const int gj = jj < 3 ? j0 + jj - 3 : j0 + TY + jj - 3;
                const int aj = jj < 3 ? jj : TY + jj;
                Y4[(i * (TY + 6) + aj) * TZ + k] = cell(i0 + i, gj, k0 + k);
            }
            for (int e = tid; e < SZ; e += NT) {
                const int kk = e % 6, j = (e / 6) % TY, i = e / (6 * TY);
                const int gk = kk < 3 ? k0 + kk - 3 : k0 + TZ + kk - 3;
                const int ak = kk < 3 ? kk : TZ + kk;
                if (gk < 0) continue;   // z-min ghost, filled below
                Z4[(i * TY + j) * (TZ + 6) + ak] = cell(i0 + i, j0 + j, gk);
            }
        }
    } else {
    for (int e = tid; e < SX; e += NT) {
        int k = e % TZ, j = (e / TZ) % TY, ii = e / (TZ * TY);
        double u[4];
        load_cell<MODE>(cf, co, d, src, i0 + ii - 3, j0 + j, k0 + k, u);
        const bool core = ii >= 3 && ii < TX + 3;
        const int ex = (ii * TY + j) * TZ + k;
        const int ey = ((ii - 3) * (TY + 6) + j + 3) * TZ + k;
        const int ez = ((ii - 3) * TY + j) * (TZ + 6) + k + 3;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const T v = T(u[c]);
            if constexpr (kNear) out_of_range |= !weno_range(u[c]);
            arm_at(s.X, AX, c, ex) = v;
            if (core) {
                arm_at(s.Y, AY, c, ey) = v;
                arm_at(s.Z, AZ, c, ez) = v;
            }
        }
    }
    for (int e = tid; e < SY; e += NT) {
        int k = e % TZ, jj = (e / TZ) % 6, i = e / (TZ * 6);
        int gj = jj < 3 ? j0 + jj - 3 : j0 + TY + jj - 3;
        int aj = jj < 3 ? jj : TY + jj;   // arm index of local j = gj - j0
        double u[4];
        load_cell<MODE>(cf, co, d, src, i0 + i, gj, k0 + k, u);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if constexpr (kNear) out_of_range |= !weno_range(u[c]);
            arm_at(s.Y, AY, c, (i * (TY + 6) + aj) * TZ + k) = T(u[c]);
        }
    }
    for (int e = tid; e < SZ; e += NT) {
        int kk = e % 6, j = (e / 6) % TY, i = e / (6 * TY);
        int gk = kk < 3 ? k0 + kk - 3 : k0 + TZ + kk - 3;
        int ak = kk < 3 ? kk : TZ + kk;
        if (gk < 0) continue;   // z-min ghost, filled below
        double u[4];
        load_cell<MODE>(cf, co, d, src, i0 + i, j0 + j, gk, u);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if constexpr (kNear) out_of_range |= !weno_range(u[c]);
            arm_at(s.Z, AZ, c, (i * TY + j) * (TZ + 6) + ak) = T(u[c]);
        }
    }
    }   // the double-precision source
    bool ieee = false;   // the tile's reconstructions take the IEEE path
    if constexpr (kNear) ieee = __syncthreads_or(out_of_range) != 0;
    else __syncthreads();
    // ---- 2. z-min ghost cells: quartic extrapolation through the inflow ----
    if (k0 == 0) {
        for (int e = tid; e < 4 * TX * TY; e += NT) {
            int j = e % TY, i = (e / TY) % TX, c = e / (TX * TY);
            int li = i0 + i, lj = j0 + j;
            if (li >= nx || lj >= ny) continue;
            T ui = T(boundary_value<MODE>(a, cf, bm, co, d, c, li, lj));
            const int ez = (i * TY + j) * (TZ + 6);
            auto z = [&](int kk) -> T & { return arm_at(s.Z, AZ, c, ez + kk); };
            T u0 = z(3), u1 = z(4), u2 = z(5), u3 = z(6);
            if (cf.spatial == PDM1_SPATIAL_WENO_Z) {   // quartic, boundary.py:247-320
                z(2) = T(5.0) * ui - T(77.0 / 12.0) * u0 + T(43.0 / 12.0) * u1 - T(17.0 / 12.0) * u2 + T(0.25) * u3;
                z(1) = T(25.0) * ui - T(505.0 / 12.0) * u0 + T(335.0 / 12.0) * u1 - T(145.0 / 12.0) * u2 + T(9.0 / 4.0) * u3;
                z(0) = T(75.0) * ui - T(545.0 / 4.0) * u0 + T(395.0 / 4.0) * u1 - T(181.0 / 4.0) * u2 + T(35.0 / 4.0) * u3;
            } else if (cf.spatial == PDM1_SPATIAL_FIRST_ORDER) {   // boundary.py:205-212
                z(2) = ui;
            } else {   // MUSCL / WENO3: quadratic, boundary.py:214-245
                z(2) = T(3.0) * ui - T(2.5) * u0 + T(0.5) * u1;
                z(1) = T(9.0) * ui - T(10.5) * u0 + T(2.5) * u1;
            }
            if constexpr (kNear) {   // the ghosts just written; what lies in the others is an earlier tile's
                const int first = cf.spatial == PDM1_SPATIAL_WENO_Z ? 0 : (cf.spatial == PDM1_SPATIAL_FIRST_ORDER ? 2 : 1);
#pragma unroll
                for (int kk = 0; kk < 3; ++kk) out_of_range |= kk >= first && !weno_range(z(kk));
            }
        }
        if constexpr (kNear) ieee = __syncthreads_or(out_of_range) != 0;
        else __syncthreads();
    }
    // ---- 3. every face of the tile's cells inside the domain: WENO-Z, projection, HLL ----
    // A ragged tile (the domain ends inside it) enumerates only those, in the same flux
    // slots: on 45x51x187 the padding is 17 % of the cells.
    const int vx = min(TX, nx - i0), vy = min(TY, ny - j0), vz = min(TZ, nz - k0);
    const bool full = vx == TX && vy == TY && vz == TZ;
    const int nfx = full ? NFX : (vx + 1) * vy * vz, nfy = full ? NFY : vx * (vy + 1) * vz;
    const int nf = full ? NF : nfx + nfy + vx * vy * (vz + 1);
    for (int f = tid; f < nf; f += NT) {
        int axis, i, j, k, slot = f;
        if (full) {
            if (f < NFX) {
                axis = 0; k = f % TZ; j = (f / TZ) % TY; i = f / (TZ * TY);
            } else if (f < NFX + NFY) {
                int u = f - NFX;
                axis = 1; k = u % TZ; j = (u / TZ) % (TY + 1); i = u / (TZ * (TY + 1));
            } else {
                int u = f - NFX - NFY;
                axis = 2; k = u % (TZ + 1); j = (u / (TZ + 1)) % TY; i = u / ((TZ + 1) * TY);
            }
        } else {
            axis = f < nfx ? 0 : (f < nfx + nfy ? 1 : 2);
            const int u = f - (axis == 0 ? 0 : (axis == 1 ? nfx : nfx + nfy));
            const int ez = axis == 2 ? vz + 1 : vz, ey = axis == 1 ? vy + 1 : vy;   // faces along z and y
            const int row = u / ez;
            k = u - row * ez;
            i = row / ey;
            j = row - i * ey;
            slot = axis == 0 ? (i * TY + j) * TZ + k
                             : (axis == 1 ? NFX + (i * (TY + 1) + j) * TZ + k : NFX + NFY + (i * TY + j) * (TZ + 1) + k);
        }
        T L[4], R[4];
        // the six cells along the axis, i - 3 .. i + 2 (face between i - 1 and i),
        // are arm indices i .. i + 5
        T *arm = s.X;
        int e0, stride, cs;
        if (axis == 0) {
            arm = s.X; e0 = (i * TY + j) * TZ + k; stride = TY * TZ; cs = AX;
        } else if (axis == 1) {
            arm = s.Y; e0 = (i * (TY + 6) + j) * TZ + k; stride = TZ; cs = AY;
        } else {
            arm = s.Z; e0 = (i * TY + j) * (TZ + 6) + k; stride = 1; cs = AZ;
        }
        if (cf.spatial == PDM1_SPATIAL_WENO_Z) {
            if constexpr (sizeof(T) == sizeof(float)) {
                // two components per packed reconstruction, L and R from the
                // same six 128-bit loads: (phi, Jx) and (Jy, Jz) of each cell
                const float4 *b4 = reinterpret_cast<const float4 *>(arm) + e0;
                float2 w01[6], w23[6];
#pragma unroll
                for (int q = 0; q < 6; ++q) {
                    const float4 v = b4[q * stride];
                    w01[q] = make_float2(v.x, v.y);
                    w23[q] = make_float2(v.z, v.w);
                }
                float2 l = weno_left_f32x2(w01[0], w01[1], w01[2], w01[3], w01[4]);
                float2 r = weno_left_f32x2(w01[5], w01[4], w01[3], w01[2], w01[1]);
                L[0] = l.x; L[1] = l.y; R[0] = r.x; R[1] = r.y;
                l = weno_left_f32x2(w23[0], w23[1], w23[2], w23[3], w23[4]);
                r = weno_left_f32x2(w23[5], w23[4], w23[3], w23[2], w23[1]);
                L[2] = l.x; L[3] = l.y; R[2] = r.x; R[3] = r.y;
            } else {
                if (!ieee) {
                    // no branch between the components: their chains interleave
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        T w[6];
#pragma unroll
                        for (int q = 0; q < 6; ++q) w[q] = arm[e0 + c * cs + q * stride];
                        weno_pair(w, L[c], R[c]);
                    }
                } else {
                    for (int c = 0; c < 4; ++c) {
                        T w[6];
#pragma unroll
                        for (int q = 0; q < 6; ++q) w[q] = arm[e0 + c * cs + q * stride];
                        const T l = weno_left_ieee(w[0], w[1], w[2], w[3], w[4]);
                        const T r = weno_left_ieee(w[5], w[4], w[3], w[2], w[1]);
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            if (q == c) { L[q] = l; R[q] = r; }
                    }
                }
            }
        } else {
            // the narrower stencils read cells i-2 .. i+1 (arm indices i+1 .. i+4)
            for (int c = 0; c < 4; ++c) {
                const T wm = arm_at(arm, cs, c, e0 + stride), w0 = arm_at(arm, cs, c, e0 + 2 * stride);
                const T w1 = arm_at(arm, cs, c, e0 + 3 * stride), wp = arm_at(arm, cs, c, e0 + 4 * stride);
                if (cf.spatial == PDM1_SPATIAL_FIRST_ORDER) {   // first_order.py:66-111
                    L[c] = w0;
                    R[c] = w1;
                } else if (cf.spatial == PDM1_SPATIAL_MUSCL) {   // muscl.py:86-145
                    T lo, hi;
                    muscl_faces(wm, w0, w1, lo, hi);
                    L[c] = hi;
                    muscl_faces(w0, w1, wp, lo, hi);
                    R[c] = lo;
                } else if constexpr (kNear) {   // WENO3, weno3.py:108-171
                    L[c] = ieee ? weno3_left_ieee(wm, w0, w1) : weno3_near(wm, w0, w1);
                    R[c] = ieee ? weno3_left_ieee(wp, w1, w0) : weno3_near(wp, w1, w0);
                } else {
                    L[c] = weno3_left(wm, w0, w1);
                    R[c] = weno3_left(wp, w1, w0);
                }
            }
        }
        if constexpr (kNear) {
            face_flux64(L, R, axis, unit, s.F + slot, NF);
        } else {
            T F[4];
            face_flux_f32x2(L, R, axis, unit, F);
#pragma unroll
            for (int c = 0; c < 4; ++c) s.F[c * NF + slot] = F[c];
        }
    }
    __syncthreads();
    // ---- 4. divergence and the stage update, one cell per thread ----
    const int k = tid % TZ, j = (tid / TZ) % TY, i = tid / (TZ * TY);
    const int li = i0 + i, lj = j0 + j, lk = k0 + k;
    const bool valid = (Tl::CELLS == NT || tid < Tl::CELLS) && li < nx && lj < ny && lk < nz;
    double phi_new = -1.0;   // for the moving box's slab maxima
    double um[4] = {0.0, 0.0, 0.0, 0.0};   // the new state, for the learned box's moments
    if (valid) {
        const int fx0 = (i * TY + j) * TZ + k, fx1 = ((i + 1) * TY + j) * TZ + k;
        const int fy0 = NFX + (i * (TY + 1) + j) * TZ + k, fy1 = NFX + (i * (TY + 1) + j + 1) * TZ + k;
        const int fz0 = NFX + NFY + (i * TY + j) * (TZ + 1) + k, fz1 = fz0 + 1;
        double L[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const T *F = s.F + c * NF;
            const T ex = F[fx1] - F[fx0], ey = F[fy1] - F[fy0], ez = F[fz1] - F[fz0];
            if constexpr (kNear) {
                // spacings are in range (checked with the plan); a difference that is not: IEEE
                double gx = quotient(ex, cf.dx, cf.inv_dx), gy = quotient(ey, cf.dy, cf.inv_dy);
                double gz = quotient(ez, cf.dz, cf.inv_dz);
                if (!(cf.spacing_near && zero_or_within<-900, 700>(ex) && zero_or_within<-900, 700>(ey) &&
                      zero_or_within<-900, 700>(ez))) {
                    gx = div_ieee(ex, cf.dx); gy = div_ieee(ey, cf.dy); gz = div_ieee(ez, cf.dz);
                }
                L[c] = -(gx + gy + gz);
            } else {
                const T gx = ex / T(cf.dx), gy = ey / T(cf.dy), gz = ez / T(cf.dz);
                L[c] = double(-(gx + gy + gz));
            }
        }
        const size_t o = ((size_t)li * ny + lj) * nz + lk;
        if (MODE == MODE_RHS) {
#pragma unroll
            for (int c = 0; c < 4; ++c) a.rhs_out[c * N + o] = L[c];
        } else {
            const size_t go = global_cell(cf, d, li, lj, lk);
            const int m = cf.ids[go];
            const double dE = co.dE;
            // the accepted state at this cell (with the Strang half step applied)
            double un[4];
            if ((MODE == MODE_A || MODE == MODE_EULER) && sizeof(T) == sizeof(double)) {
#pragma unroll
                for (int c = 0; c < 4; ++c) un[c] = double(s.X[((c * (TX + 6) + (i + 3)) * TY + j) * TZ + k]);
            } else if (MODE == MODE_A || MODE == MODE_EULER) {
                load_cell<MODE>(cf, co, d, Ua, li, lj, lk, un);   // the state in double
            } else {
                load_cell<MODE_A>(cf, co, d, Ua, li, lj, lk, un);
            }
            const double s0 = co.S0[m];
            if (MODE == MODE_A) {
                double u1[4], v1[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    double v0 = s0 * un[c];
                    double v = L[c] * dE + v0;
                    v1[c] = v;
                    u1[c] = v * (c == 0 ? co.c1p[m] : co.c1c[m]);
                }
                div4(u1, co.S1[m]);
                project64(u1);
                if constexpr (kF4Dest<T, MODE>)
                    reinterpret_cast<float4 *>(U1)[o] = make_float4(float(u1[0]), float(u1[1]), float(u1[2]),
                                                                    float(u1[3]));
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    if constexpr (!kF4Dest<T, MODE>) U1[c * N + o] = u1[c];
                    Vb[c * N + o] = v1[c];
                }
                double q0 = un[0] * s0, q1 = u1[0] * co.S1[m];
                qb[o] = 1.0 / 6.0 * q0 + 1.0 / 6.0 * q1;
            } else if (MODE == MODE_B) {
                double u2[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    double r = L[c] * (c == 0 ? co.c1ip[m] : co.c1ic[m]);
                    r = (r * dE + Vb[c * N + o]) * 0.25;
                    double v = 0.75 * (s0 * un[c]) + r;
                    Vb[c * N + o] = v;
                    u2[c] = v * (c == 0 ? co.c2p[m] : co.c2c[m]);
                }
                div4(u2, co.S2[m]);
                project64(u2);
                if constexpr (kF4Dest<T, MODE>) {
                    reinterpret_cast<float4 *>(U2)[o] = make_float4(float(u2[0]), float(u2[1]), float(u2[2]),
                                                                    float(u2[3]));
                    // the dose quadrature's stage-2 term, from the double state
                    // (stage C reads the sum; the same sum, rounded as it would be there)
                    double q2 = u2[0] * co.S2[m];
                    qb[o] = qb[o] + 2.0 / 3.0 * q2;
                } else {
#pragma unroll
                    for (int c = 0; c < 4; ++c) U2[c * N + o] = u2[c];
                }
            } else {
                double unew[4];
                double ed;
                if (MODE == MODE_C) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        double r = L[c] * (c == 0 ? co.c2ip[m] : co.c2ic[m]);
                        r = (r * dE + Vb[c * N + o]) * (2.0 / 3.0);
                        double v = 1.0 / 3.0 * (s0 * un[c]) + r;
                        unew[c] = v * (c == 0 ? co.c1p[m] : co.c1c[m]);
                    }
                    div4(unew, co.S1[m]);
                    project64(unew);
                    if constexpr (sizeof(T) == sizeof(double)) {
                        double u2c = double(s.X[((i + 3) * TY + j) * TZ + k]);
                        double q2 = u2c * co.S2[m];
                        ed = dE * (qb[o] + 2.0 / 3.0 * q2);
                    } else {
                        ed = dE * qb[o];   // stage B added 2/3 q2
                    }
                } else {   // forward Euler, numerics/energy.py:663-722
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        unew[c] = L[c] * dE + s0 * un[c];
                    }
                    div4(unew, co.S1[m]);
                    project64(unew);
                    ed = dE * un[0] * s0;
                }
                if (cf.strang) {
                    if (cf.nuclear)
#pragma unroll
                        for (int c = 0; c < 4; ++c) unew[c] *= co.hn[m];
                    if (cf.scattering != PDM1_SCATTERING_OFF)
#pragma unroll
                        for (int c = 1; c < 4; ++c) unew[c] *= co.hs[m];
                }
                if (MODE == MODE_C)
#pragma unroll
                    for (int c = 0; c < 4; ++c) um[c] = unew[c];
                double *dst = MODE == MODE_C ? Ua : U1;
                bool finite = true;
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    dst[c * N + o] = unew[c];
                    finite = finite && isfinite(unew[c]);
                }
                // a non-finite state ends the march with PDM1_ERR_NONFINITE
                if (!finite) atomicOr(&stb.error, ERR_DEV_NONFINITE);
                if (a.edep) a.edep[o] = ed;
                else atomicAdd(&a.dose[go], ed * kMevToJoule / cf.density[m]);
                if (MODE == MODE_C) {
                    if (co.snap_slot >= 0 && a.snap) {
                        const size_t NG = (size_t)cf.nx * cf.ny * cf.nz;
                        double *sn = a.snap + (size_t)co.snap_slot * 4 * NG;
#pragma unroll
                        for (int c = 0; c < 4; ++c) sn[c * NG + go] = unew[c];
                    }
                    if (!cf.moving) {
                        double phi_in = 0.0;
                        if (lk == 0 && d.inflow)
                            phi_in = bm.spatial[(size_t)(d.i0 + li) * cf.ny + (d.j0 + lj)] * co.ed_next;
                        double v = cfl_term<T>(cf, bm.rf, unew, co.S1[m], lk == 0, phi_in, all_axes);
                        cta_inv = fmax(cta_inv, v);
                    }
                    phi_new = unew[0];
                }
            }
        }
    }
    if (MODE == MODE_C && cf.moving) {
        static_assert(sizeof(SlabScratch<Tl>) <= sizeof(sh.slab), "slab scratch");
        stage_slab_max<Tl>(cf, beam_slab(cf, b), d, phi_new, i0, j0, k0, *reinterpret_cast<SlabScratch<Tl> *>(sh.slab));
    }
    if constexpr (LEARN && MODE == MODE_C) {
        // learned box: the moments of the new state feed the next step's proposer
        tile_moments_cta<NT>(cf, b, d, i0, j0, k0, valid, li, lj, lk, um, sh.mom_part, sh.mom_pl);
    }
}

__device__ __forceinline__ unsigned long long clock_ns() {
    unsigned long long v;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(v));
    return v;
}

// LEARN (stage C of a plan with a learned box): the tile's fluence moments of
// the new state are accumulated for the next step's proposer.
template <typename T, int MODE, class Tl, bool LEARN = false>
__global__ void __launch_bounds__(NT, sizeof(T) == sizeof(double) ? 2 : 4) stage_kernel(const __grid_constant__ StageArgs a) {
    const ConfigDev &cf = *a.cf;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    StageShared &sh = *reinterpret_cast<StageShared *>(smem_raw);
    double cta_inv = 0.0;
    if ((MODE == MODE_A || MODE == MODE_EULER) && a.begin_ns && blockIdx.x == 0 && threadIdx.x == 0)
        *a.begin_ns = *a.end_ns = clock_ns();
    // FP32 stages B and C: bulk copies of the float4 stage state, one mbarrier phase per tile
    unsigned bar_phase = 0;
    if constexpr (kF4Source<T, MODE>) {
        if (cf.bulk_stage) {
            if (threadIdx.x == 0) mbar_init(&sh.stage_bar, NT);
            __syncthreads();
        }
    }
    // tiles of all marching beams, back to back (one beam: its domain's tiles).  A CTA takes
    // the first by its index and, from two waves of tiles on, each further one from the
    // stage's counter while it works on the one before: ragged tiles and those at the entrance
    // cost less and more than the rest (45x51x187 FP64 step, 6.8 waves: 598 us by index, 559
    // by counter).  Below two waves the SM that ends first would take a second wave of its
    // own while others idle (28x14x500 FP32 step, 1.5 waves: 173 us by index, 182 by counter).
    const int total = MODE == MODE_RHS ? a.st[0].dom.ntiles : cf.tile_off[cf.nbeams];
    int *const counter = cf.tile_off + cf.nbeams + 1 + (MODE == MODE_EULER ? 0 : MODE);
    for (int gt = blockIdx.x; gt < total;) {
        const int b = (MODE == MODE_RHS || cf.nbeams == 1) ? 0 : beam_of_tile(cf.tile_off, cf.nbeams, gt);
        const int tile = MODE == MODE_RHS ? gt : gt - cf.tile_off[b];
        int next = gridDim.x + gt;
        if (MODE != MODE_RHS && threadIdx.x == 0 && total >= 2 * (int)gridDim.x) next = gridDim.x + atomicAdd(counter, 1);
        const DomainDev d = a.st[b].dom;
        stage_tile<T, MODE, Tl, LEARN>(a, cf, d, b, tile, bar_phase, cta_inv);
        if (threadIdx.x == 0) sh.next_tile[bar_phase] = next;
        __syncthreads();   // shared memory is reused by the next tile
        gt = sh.next_tile[bar_phase];
        bar_phase ^= 1u;
    }
    if (MODE == MODE_C && !cf.moving) block_max_atomic<NT>(cta_inv, &a.st[0].inv_bits);
    if ((MODE == MODE_C || MODE == MODE_EULER) && a.end_ns && threadIdx.x == 0) atomicMax(a.end_ns, clock_ns());
}

}  // namespace pdm1
