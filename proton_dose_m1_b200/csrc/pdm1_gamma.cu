// pdm1_gamma.cu -- global 3-D gamma index on the GPU.
//
// The reference scores doses with pymedphys.gamma (pymedphys 0.41.0, called at
// proton_solver/metrics.py:581-594 with interp_fraction=10, max_gamma=1.1,
// local_gamma=False, global_normalisation=max(reference),
// lower_percent_dose_cutoff=10, skip_once_passed=True).  This kernel follows
// the published definition (Low et al., Med. Phys. 25 (1998) 656) with those
// parameters: for every reference voxel at or above the cutoff,
//   gamma = min over evaluation points e within max_gamma * DTA of
//           sqrt(|r - e|^2 / DTA^2 + (D_eval(e) - D_ref(r))^2 / dD^2),
// where the evaluation dose is trilinearly interpolated at points on a lattice
// of spacing DTA / interp_fraction around r (points outside the evaluation
// grid are not candidates) and dD = dose_percent/100 * global normalisation.
// Candidates are visited in order of distance, so the search stops as soon as
// the distance term alone exceeds the best value, or once gamma <= 1.
#include "../../include/pdm1.h"
#include "pdm1_device.cuh"

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <exception>
#include <vector>

namespace {

struct Offset {
    double dx, dy, dz;   // mm
    double d2;           // squared distance / DTA^2
};

__device__ __forceinline__ double trilinear(const double *D, int nx, int ny, int nz, double fi, double fj,
                                            double fk) {
    int i = (int)floor(fi), j = (int)floor(fj), k = (int)floor(fk);
    // the lower corner of the cell; an axis of one cell has corner 0 only
    i = max(min(i, nx - 2), 0);
    j = max(min(j, ny - 2), 0);
    k = max(min(k, nz - 2), 0);
    double ti = nx > 1 ? fi - i : 0.0, tj = ny > 1 ? fj - j : 0.0, tk = nz > 1 ? fk - k : 0.0;
    int i1 = nx > 1 ? i + 1 : i, j1 = ny > 1 ? j + 1 : j, k1 = nz > 1 ? k + 1 : k;
    auto at = [&](int a, int b, int c) { return D[((size_t)a * ny + b) * nz + c]; };
    double c00 = at(i, j, k) * (1.0 - tk) + at(i, j, k1) * tk;
    double c01 = at(i, j1, k) * (1.0 - tk) + at(i, j1, k1) * tk;
    double c10 = at(i1, j, k) * (1.0 - tk) + at(i1, j, k1) * tk;
    double c11 = at(i1, j1, k) * (1.0 - tk) + at(i1, j1, k1) * tk;
    double c0 = c00 * (1.0 - tj) + c01 * tj;
    double c1 = c10 * (1.0 - tj) + c11 * tj;
    return c0 * (1.0 - ti) + c1 * ti;
}

// Squared gamma of the candidate `ofs` of voxel (i, j, k) with dose dr; infinite outside the grid.
__device__ __forceinline__ double candidate(const Offset &ofs, const double *eval, int nx, int ny, int nz, double hx,
                                            double hy, double hz, int i, int j, int k, double dr, double inv_dd2) {
    const double fi = i + ofs.dx / hx, fj = j + ofs.dy / hy, fk = k + ofs.dz / hz;
    if (fi < 0.0 || fi > nx - 1 || fj < 0.0 || fj > ny - 1 || fk < 0.0 || fk > nz - 1) return INFINITY;
    const double de = trilinear(eval, nx, ny, nz, fi, fj, fk) - dr;
    return ofs.d2 + de * de * inv_dd2;
}

// A CTA per 256 voxels: each thread takes the nearest candidate (the voxel itself); the
// voxels at or above the cutoff that it does not pass are listed in shared memory and
// searched by one warp each, 32 candidates at a time.  A voxel's gamma is the
// first candidate's that passes (skip_once_passed) or the smallest of all that are nearer
// than it, in whichever way they are evaluated; a thread per voxel walked up to 5575
// candidates in turn, and the few voxels that fail held the kernel for them (80x80x400 at
// 0.5 mm, 1 %/1 mm, whole call: 1.7-5.6 ms by the share that fails -> 0.5 ms).  Where nearly
// all pass at the first candidate, as two close doses without a cutoff do, a warp for each of
// them took 14 ms on 256x256x320, a thread 1.2 ms (2 to 32 candidates by the thread: no
// faster).
constexpr int kGammaThreads = 256;
__global__ void __launch_bounds__(kGammaThreads) gamma_kernel(const double *ref, const double *eval, int nx, int ny,
                                                              int nz, double hx, double hy, double hz,
                                                              const Offset *off, int n_off, double inv_dd2,
                                                              double cutoff, double max_gamma, int skip_once_passed,
                                                              double *gamma, unsigned long long *counts) {
    __shared__ int list[kGammaThreads];
    __shared__ int n_list;
    const size_t N = (size_t)nx * ny * nz, base = (size_t)blockIdx.x * kGammaThreads;
    const int lane = threadIdx.x & 31;
    if (threadIdx.x == 0) n_list = 0;
    __syncthreads();
    unsigned pass = 0, valid = 0;
    auto finish = [&](size_t o, double best) {
        double g = sqrt(best);
        if (g > max_gamma) g = max_gamma > 0.0 ? INFINITY : g;
        gamma[o] = g;
        ++valid;
        pass += g <= 1.0;
    };
    const size_t mine = base + threadIdx.x;
    if (mine < N) {
        const double dr = ref[mine];
        if (dr >= cutoff) {
            const int k = (int)(mine % nz), j = (int)((mine / nz) % ny), i = (int)(mine / ((size_t)nz * ny));
            const double g2 = n_off > 0 ? candidate(off[0], eval, nx, ny, nz, hx, hy, hz, i, j, k, dr, inv_dd2) : INFINITY;
            if (skip_once_passed && g2 <= 1.0) finish(mine, g2);
            else list[atomicAdd(&n_list, 1)] = threadIdx.x;
        } else {
            gamma[mine] = NAN;
        }
    }
    __syncthreads();
    for (int v = threadIdx.x >> 5; v < n_list; v += kGammaThreads / 32) {
        const size_t o = base + list[v];
        const double dr = ref[o];
        const int k = (int)(o % nz), j = (int)((o / nz) % ny), i = (int)(o / ((size_t)nz * ny));
        double best = INFINITY;
        for (int q0 = 0; q0 < n_off; q0 += 32) {
            const int q = q0 + lane;
            double g2 = INFINITY, d2 = INFINITY;
            if (q < n_off) {
                const Offset ofs = off[q];
                d2 = ofs.d2;
                g2 = candidate(ofs, eval, nx, ny, nz, hx, hy, hz, i, j, k, dr, inv_dd2);
            }
            if (__shfl_sync(0xffffffffu, d2, 0) >= best) break;   // farther points cannot win
            const unsigned passed = __ballot_sync(0xffffffffu, skip_once_passed && g2 <= 1.0);
            if (passed) {   // the first in order ends the search
                best = __shfl_sync(0xffffffffu, g2, __ffs(passed) - 1);
                break;
            }
            for (int w = 16; w > 0; w >>= 1) g2 = fmin(g2, __shfl_xor_sync(0xffffffffu, g2, w));
            best = fmin(best, g2);
        }
        if (lane == 0) finish(o, best);
    }
    pass = __reduce_add_sync(0xffffffffu, pass);
    valid = __reduce_add_sync(0xffffffffu, valid);
    if (lane == 0 && valid) {
        atomicAdd(&counts[0], (unsigned long long)pass);
        atomicAdd(&counts[1], (unsigned long long)valid);
    }
}

}  // namespace

extern "C" int pdm1_gamma(const double *dose_ref, const double *dose_eval, int nx, int ny, int nz,
                          double dx_mm, double dy_mm, double dz_mm, double dose_percent,
                          double distance_mm, double lower_cutoff_percent, int interp_fraction,
                          double max_gamma, double global_normalisation, double *gamma_out,
                          double *pass_rate_out, pdm1_stream_t stream_) {
    if (!dose_ref || !dose_eval || !gamma_out || nx <= 0 || ny <= 0 || nz <= 0 || !(dx_mm > 0) ||
        !(dy_mm > 0) || !(dz_mm > 0) || !(dose_percent > 0) || !(distance_mm > 0) || interp_fraction <= 0 ||
        !(global_normalisation > 0))
        return PDM1_ERR_ARGUMENT;
    cudaStream_t stream = (cudaStream_t)stream_;
    // candidate offsets on the interpolation lattice inside the search sphere, by distance
    const double h = distance_mm / interp_fraction;
    const double R = (max_gamma > 0 ? max_gamma : 1.0) * distance_mm;
    const double cells = std::floor(R / h + 1e-9);
    const int m = cells >= 0.0 && cells < 2147483647.0 ? (int)cells : -1;
    // (sorted within the shells of equal a^2 + b^2 + c^2, whose distances differ by rounding only);
    // a radius that the lattice cannot count (infinite: m < 0) has no candidates
    std::vector<Offset> offs;
    try {
        std::vector<std::vector<Offset>> shells(m < 0 ? 0 : 3 * (size_t)m * m + 1);
        for (int a = -m; a <= m; ++a)
            for (int b = -m; b <= m; ++b)
                for (int c = -m; c <= m; ++c) {
                    double x = a * h, y = b * h, z = c * h;
                    double r2 = x * x + y * y + z * z;
                    if (r2 <= R * R * (1.0 + 1e-12))
                        shells[(size_t)((long long)a * a + (long long)b * b + (long long)c * c)].push_back(
                            {x, y, z, r2 / (distance_mm * distance_mm)});
                }
        for (auto &s : shells) {
            std::stable_sort(s.begin(), s.end(), [](const Offset &p, const Offset &q) { return p.d2 < q.d2; });
            offs.insert(offs.end(), s.begin(), s.end());
        }
    } catch (const std::exception &) {   // more candidates than memory holds: no C++ exception leaves a C entry
        return PDM1_ERR_ARGUMENT;
    }
    unsigned long long *d_counts = nullptr;   // the two counts, then the candidates
    const size_t head = 256;
    if (pdm1::pool_malloc_workspace((void **)&d_counts, head + offs.size() * sizeof(Offset)) != cudaSuccess)
        return PDM1_ERR_CUDA;
    Offset *d_off = (Offset *)((unsigned char *)d_counts + head);
    cudaMemcpyAsync(d_off, offs.data(), offs.size() * sizeof(Offset), cudaMemcpyHostToDevice, stream);
    cudaMemsetAsync(d_counts, 0, 2 * sizeof(unsigned long long), stream);
    double dD = dose_percent / 100.0 * global_normalisation;
    double cutoff = lower_cutoff_percent / 100.0 * global_normalisation;
    size_t N = (size_t)nx * ny * nz;
    int blocks = (int)((N + kGammaThreads - 1) / kGammaThreads);
    gamma_kernel<<<blocks, kGammaThreads, 0, stream>>>(dose_ref, dose_eval, nx, ny, nz, dx_mm, dy_mm, dz_mm, d_off,
                                             (int)offs.size(), 1.0 / (dD * dD), cutoff, max_gamma, 1,
                                             gamma_out, d_counts);
    unsigned long long counts[2] = {0, 0};
    cudaError_t e = cudaMemcpyAsync(counts, d_counts, sizeof counts, cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) cudaStreamSynchronize(stream);   // nothing of this call still uses the block
    pdm1::pool_free(d_counts);
    if (e != cudaSuccess) return PDM1_ERR_CUDA;
    if (pass_rate_out) *pass_rate_out = counts[1] ? 100.0 * (double)counts[0] / (double)counts[1] : NAN;
    return PDM1_OK;
}
