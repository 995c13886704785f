// pdm1_analytical.cu -- the analytical CSDA + straight-streaming dose on the GPU.
//
// The reference's reduced-model verifier (proton_solver/analytical.py:64-326):
// without scattering, nuclear removal or angular spread, every proton keeps
// its transverse position and loses energy along z by the continuous-slowing-
// down range relation R(E_out) = R(E_in) - dz, cell by cell.  The dose of a
// cell is the spectrum-weighted energy lost in it (trapezoid rule over the
// incident energies on [energy_min, E0 + window * sigma_E]) times
// MEV_TO_JOULE / (rho dz), scaled by the beam's transverse fluence.
//
// Range tables (analytical.py:64-106): geometric energy grid from the
// stopping-power table's first node to its last, PCHIP stopping power,
// cumulative trapezoid of 1/S, built on the device.  Energy <-> range by linear
// interpolation (numpy.interp semantics: clamp below to 0, above to the last value).
// Identical material columns share one column computation, as the
// reference's column cache does; the energies of a column are marched by one
// thread each, the per-cell sums reduced per CTA and added atomically.
#include "../../include/pdm1.h"
#include "pdm1_device.cuh"

#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <string>
#include <unordered_map>
#include <vector>

namespace pdm1 {
std::vector<double> host_pchip_slopes(const double *E, const double *v, int n);
}

using namespace pdm1;

namespace {

constexpr int kThreads = 256;

struct RangeView {
    const double *E, *R;
    int n;
    double log_a, inv_step;   // the energies are exp(log_a + i / inv_step)
};

// numpy.interp at x in [xs[0], xs[n - 1]] given a guess of the interval: the interval
// is the last one with xs[lo] <= x (at most n - 2), found by steps that double from the
// guess and then halve, two or three loads when the guess is near.
__device__ __forceinline__ double interp_from(double x, const double *xs, const double *ys, int n, int guess, int &at) {
    int lo = min(max(guess, 0), n - 2), hi;
    if (xs[lo] <= x) {
        int w = 1;
        hi = lo + 1;
        while (hi < n - 1 && xs[hi] <= x) { lo = hi; w <<= 1; hi = min(lo + w, n - 1); }
    } else {
        int w = 1;
        hi = lo;
        lo = max(hi - w, 0);
        while (lo > 0 && xs[lo] > x) { hi = lo; w <<= 1; lo = max(hi - w, 0); }
    }
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (xs[mid] <= x) lo = mid; else hi = mid;
    }
    at = lo;
    const double x0 = xs[lo], x1 = xs[hi];
    if (x1 == x0) return ys[hi];
    const double t = (x - x0) / (x1 - x0);
    return ys[lo] + t * (ys[hi] - ys[lo]);
}

// Energy grid and 1/S of a material's range table (grid.y: material).
__global__ void range_grid_kernel(const TableView *sp, RangeView *tabs, double *blob, int n, double *inv_S) {
    const int m = blockIdx.y, i = blockIdx.x * blockDim.x + threadIdx.x;
    const TableView t = sp[m];
    const double a = t.E[0] > 1e-12 ? t.E[0] : 1e-12, b = t.E[t.n - 1];
    const double la = log(a), lb = log(b);
    double *E = blob + 2 * (size_t)m * n;
    if (i == 0) tabs[m] = RangeView{E, E + n, n, la, (n - 1) / (lb - la)};
    if (i >= n) return;
    const double e = i == 0 ? a : (i == n - 1 ? b : exp(la + (lb - la) * i / (n - 1)));
    E[i] = e;
    inv_S[(size_t)m * n + i] = 1.0 / pchip_eval(t, fmax(e, t.E[0]));
}

// Cumulative trapezoid of 1/S: one CTA per material, each thread sums a run of the
// table, the runs' sums are scanned, each thread writes its run.  Sums are carried as
// value and remainder (dd_add), so every R is its terms' sum rounded once: the dose of 170 mm
// of water is 1.8e-14 from extended precision, 2.6e-14 with the sequential sum in double.
constexpr int kScanThreads = 1024;
__global__ void __launch_bounds__(kScanThreads) range_sum_kernel(double *blob, int n, const double *inv_S) {
    __shared__ dd sum[kScanThreads];
    const int m = blockIdx.x, t = threadIdx.x;
    const double *E = blob + 2 * (size_t)m * n, *q = inv_S + (size_t)m * n;
    double *R = blob + (2 * (size_t)m + 1) * n;
    const int run = (n + kScanThreads - 1) / kScanThreads, lo = min(t * run, n), hi = min(lo + run, n);
    auto step = [&](int i) { return dd{i > 0 ? 0.5 * (q[i] + q[i - 1]) * (E[i] - E[i - 1]) : 0.0, 0.0}; };
    dd s = {0.0, 0.0};
    for (int i = lo; i < hi; ++i) s = dd_add(s, step(i));
    sum[t] = s;
    __syncthreads();
    for (int w = 1; w < kScanThreads; w <<= 1) {
        const dd v = t >= w ? sum[t - w] : dd{0.0, 0.0};
        __syncthreads();
        sum[t] = dd_add(sum[t], v);
        __syncthreads();
    }
    s = t > 0 ? sum[t - 1] : dd{0.0, 0.0};
    for (int i = lo; i < hi; ++i) {
        s = dd_add(s, step(i));
        R[i] = s.hi;
    }
}

// Incident energies on [Emin, E0], trapezoid weights times the spectrum (analytical.py:173-269).
struct Incident {
    double Emin, E0, E_beam, sigma, norm;
    int n;
    __device__ double node(int i) const { return i == n - 1 ? E0 : Emin + (E0 - Emin) * i / (double)(n - 1); }
    __device__ double weight(int i) const {
        const double e = node(i), d = e - E_beam;
        const double left = i > 0 ? e - node(i - 1) : 0.0, right = i + 1 < n ? node(i + 1) - e : 0.0;
        return 0.5 * (left + right) * (exp(-(d * d) / (2.0 * sigma * sigma)) / norm);
    }
};

// One column per blockIdx.y; energy nodes over blockIdx.x * blockDim.x + threadIdx.x.
// Energies whose weight underflows to 0 (38 standard deviations off) add nothing: a warp
// of them stops.  Both look-ups start from a guess (the log spacing; the range-energy power
// law E ~ R^(1/1.77) from the interval before), and the warps' sums wait in shared memory for
// kLevels cells at a time.  With binary searches over 200,000 nodes, two barriers a cell,
// every energy marched and the tables built on the host, the whole call took 10.4-13 ms on
// 40x40x200 water; now 2.0 ms.
constexpr int kLevels = 128;
__global__ void __launch_bounds__(kThreads) column_kernel(const RangeView *tabs, const int *col_mats, int nz,
                                                          double dz, Incident in, double *lost_sum) {
    __shared__ double part[kThreads / 32][kLevels];
    const int col = blockIdx.y;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double w = i < in.n ? in.weight(i) : 0.0;
    double E = w != 0.0 ? in.node(i) : 0.0;
    if (!__syncthreads_or(E > 0.0)) return;
    for (int z0 = 0; z0 < nz; z0 += kLevels) {
        const int levels = min(kLevels, nz - z0);
        for (int q = 0; q < levels; ++q) {
            double v = 0.0;
            if (__any_sync(0xffffffffu, E > 0.0)) {
                const RangeView t = tabs[col_mats[(size_t)col * nz + z0 + q]];
                if (E > 0.0) {
                    // numpy.interp: 0 below the table, its last value above
                    double r_in, e_out = 0.0;
                    int at = t.n - 2;
                    if (!(E >= t.E[0])) r_in = 0.0;
                    else if (E > t.E[t.n - 1]) r_in = t.R[t.n - 1];
                    else r_in = interp_from(E, t.E, t.R, t.n, (int)((logf((float)E) - (float)t.log_a) * (float)t.inv_step), at);
                    const double r_out = r_in - dz;
                    if (r_out > 0.0) {
                        const float back = logf((float)(r_out / r_in)) * (1.0f / 1.77f) * (float)t.inv_step;
                        const int guess = at + (int)fmaxf(back, -1.0e9f);
                        if (!(r_out >= t.R[0])) e_out = 0.0;
                        else if (r_out > t.R[t.n - 1]) e_out = t.E[t.n - 1];
                        else e_out = interp_from(r_out, t.R, t.E, t.n, guess, at);
                    }
                    v = w * fmax(E - e_out, 0.0);
                    E = e_out;
                }
                for (int s = 16; s > 0; s >>= 1) v += __shfl_xor_sync(0xffffffffu, v, s);
            }
            if (lane == 0) part[warp][q] = v;
        }
        __syncthreads();
        for (int q = threadIdx.x; q < levels; q += kThreads) {
            double sum = 0.0;
            for (int k = 0; k < kThreads / 32; ++k) sum += part[k][q];
            if (sum != 0.0) atomicAdd(&lost_sum[(size_t)col * nz + z0 + q], sum);
        }
        __syncthreads();
    }
}

__global__ void dose_kernel(const int *col_of, const double *lost_sum, const int32_t *ids, const double *inv_rho,
                            const double *spatial, int nx, int ny, int nz, double scale, double *dose) {
    size_t N = (size_t)nx * ny * nz;
    for (size_t o = (size_t)blockIdx.x * blockDim.x + threadIdx.x; o < N; o += (size_t)gridDim.x * blockDim.x) {
        int k = (int)(o % nz);
        size_t xy = o / nz;
        double f = lost_sum[(size_t)col_of[xy] * nz + k] * scale * inv_rho[ids[o]];
        dose[o] = spatial[xy] * f;
    }
}

#define CUDA_OK(expr)                                                              \
    do {                                                                           \
        cudaError_t e_ = (expr);                                                   \
        if (e_ != cudaSuccess) {                                                   \
            std::string m_ = std::string(#expr ": ") + cudaGetErrorString(e_);     \
            return report_error(PDM1_ERR_CUDA, m_.c_str());                        \
        }                                                                          \
    } while (0)

}  // namespace

extern "C" int pdm1_analytical_csda_dose(const pdm1_problem *p, int energy_points, int range_points, double *dose,
                                         pdm1_stream_t stream_) {
    if (!p || !dose || !p->materials || !p->ids || !p->inflow_spatial)
        return report_error(PDM1_ERR_ARGUMENT, "NULL problem, tables, ids, inflow or dose");
    if (p->scattering != PDM1_SCATTERING_OFF || p->nuclear || p->angular_spread != 0.0)
        return report_error(PDM1_ERR_ARGUMENT, "Analytical reference is not available for this configuration.");
    if (energy_points < 2) return report_error(PDM1_ERR_ARGUMENT, "num_energy_points must be at least 2.");
    if (range_points < 2) return report_error(PDM1_ERR_ARGUMENT, "range_points must be at least 2.");
    if (!(p->energy_spread > 0.0))
        return report_error(PDM1_ERR_ARGUMENT, "Zero energy spread is not supported by the Gaussian inflow.");
    if (p->nx <= 0 || p->ny <= 0 || p->nz <= 0 || p->n_materials < 1 || p->n_materials > kMaxMat)
        return report_error(PDM1_ERR_ARGUMENT, "bad grid or material count");
    cudaStream_t stream = (cudaStream_t)stream_;
    const int nx = p->nx, ny = p->ny, nz = p->nz, nm = p->n_materials;
    const size_t NXY = (size_t)nx * ny, N = NXY * nz;
    for (size_t c = 0; c < N; ++c)
        if (p->ids[c] < 0 || p->ids[c] >= nm) return report_error(PDM1_ERR_ARGUMENT, "material id out of range");
    // stopping-power tables with their PCHIP slopes; the range tables are built from them
    std::vector<double> tables;
    std::vector<TableView> sp(nm);
    std::vector<double> inv_rho(nm);
    for (int m = 0; m < nm; ++m) {
        const pdm1_table &t = p->materials[m].stopping_power;
        if (t.n_nodes < 2) return report_error(PDM1_ERR_ARGUMENT, "stopping-power table needs two nodes");
        std::vector<double> slopes = host_pchip_slopes(t.energy, t.value, t.n_nodes);
        sp[m].n = t.n_nodes;
        sp[m].log_e0 = sp[m].inv_log_step = 0.0;   // the interval by bisection
        tables.insert(tables.end(), t.energy, t.energy + t.n_nodes);
        tables.insert(tables.end(), t.value, t.value + t.n_nodes);
        tables.insert(tables.end(), slopes.begin(), slopes.end());
        inv_rho[m] = 1.0 / p->materials[m].density;
    }
    Incident in;
    in.Emin = p->energy_min;
    in.E0 = p->beam_energy + p->energy_window_sigma * p->energy_spread;
    in.E_beam = p->beam_energy;
    in.sigma = p->energy_spread;
    in.norm = std::sqrt(2.0 * 3.141592653589793) * p->energy_spread;
    in.n = energy_points;
    // distinct material columns (the reference's column cache): by a hash of the column,
    // compared with the columns of that hash
    std::unordered_multimap<uint64_t, int> seen;
    std::vector<int> col_of(NXY), first;
    std::vector<int> col_mats;
    for (size_t xy = 0; xy < NXY; ++xy) {
        const int32_t *c = p->ids + xy * nz;
        uint64_t h = 1469598103934665603ull;
        for (int k = 0; k < nz; ++k) h = (h ^ (uint32_t)c[k]) * 1099511628211ull;
        int found = -1;
        auto r = seen.equal_range(h);
        for (auto it = r.first; it != r.second && found < 0; ++it)
            if (std::memcmp(p->ids + (size_t)first[it->second] * nz, c, nz * sizeof(int32_t)) == 0) found = it->second;
        if (found < 0) {
            found = (int)first.size();
            first.push_back((int)xy);
            seen.emplace(h, found);
            col_mats.insert(col_mats.end(), c, c + nz);
        }
        col_of[xy] = found;
    }
    const int ncol = (int)first.size();
    // one block for the call's buffers
    unsigned char *block = nullptr;
    size_t used = 0;
    auto part = [&](size_t bytes) { const size_t at = used; used = (at + bytes + 255) & ~size_t(255); return at; };
    const size_t o_blob = part(2 * (size_t)nm * range_points * sizeof(double));
    const size_t o_invS = part((size_t)nm * range_points * sizeof(double));
    const size_t o_tab = part(tables.size() * sizeof(double)), o_views = part(nm * sizeof(TableView));
    const size_t o_lost = part((size_t)ncol * nz * sizeof(double)), o_rho = part(nm * sizeof(double));
    const size_t o_sp = part(NXY * sizeof(double)), o_cm = part(col_mats.size() * sizeof(int));
    const size_t o_colof = part(NXY * sizeof(int)), o_ids = part(N * sizeof(int32_t));
    const size_t o_tabs = part(nm * sizeof(RangeView));
    if (pool_malloc_workspace((void **)&block, used) != cudaSuccess)
        return report_error(PDM1_ERR_CUDA, "pdm1_analytical_csda_dose: cudaMalloc failed");
    auto release = [&]() {   // back to the pool: nothing of this call may still use it
        cudaStreamSynchronize(stream);
        pool_free(block);
    };
    double *d_blob = (double *)(block + o_blob), *d_invS = (double *)(block + o_invS), *d_tab = (double *)(block + o_tab);
    double *d_lost = (double *)(block + o_lost), *d_rho = (double *)(block + o_rho), *d_sp = (double *)(block + o_sp);
    int *d_cm = (int *)(block + o_cm), *d_colof = (int *)(block + o_colof);
    int32_t *d_ids = (int32_t *)(block + o_ids);
    TableView *d_views = (TableView *)(block + o_views);
    RangeView *d_tabs = (RangeView *)(block + o_tabs);
    size_t at = 0;
    for (int m = 0; m < nm; ++m) {
        sp[m].E = d_tab + at;
        sp[m].v = d_tab + at + sp[m].n;
        sp[m].slope = d_tab + at + 2 * (size_t)sp[m].n;
        at += 3 * (size_t)sp[m].n;
    }
    cudaError_t e = cudaSuccess;
    auto up = [&](void *dst, const void *src, size_t bytes) {
        if (e == cudaSuccess) e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, stream);
    };
    up(d_tab, tables.data(), tables.size() * sizeof(double));
    up(d_views, sp.data(), nm * sizeof(TableView));
    if (e == cudaSuccess) e = cudaMemsetAsync(d_lost, 0, (size_t)ncol * nz * sizeof(double), stream);
    up(d_rho, inv_rho.data(), nm * sizeof(double));
    up(d_sp, p->inflow_spatial, NXY * sizeof(double));
    up(d_cm, col_mats.data(), col_mats.size() * sizeof(int));
    up(d_colof, col_of.data(), NXY * sizeof(int));
    up(d_ids, p->ids, N * sizeof(int32_t));
    if (e == cudaSuccess) {
        range_grid_kernel<<<dim3((range_points + 255) / 256, nm), 256, 0, stream>>>(d_views, d_tabs, d_blob, range_points, d_invS);
        range_sum_kernel<<<nm, kScanThreads, 0, stream>>>(d_blob, range_points, d_invS);
        dim3 grid((energy_points + kThreads - 1) / kThreads, ncol);
        column_kernel<<<grid, kThreads, 0, stream>>>(d_tabs, d_cm, nz, p->dz, in, d_lost);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) {
        int blocks = (int)std::min<size_t>((N + 255) / 256, 148 * 16);
        dose_kernel<<<blocks, 256, 0, stream>>>(d_colof, d_lost, d_ids, d_rho, d_sp, nx, ny, nz,
                                                kMevToJoule / p->dz, dose);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    release();
    if (e != cudaSuccess) return report_error(PDM1_ERR_CUDA, cudaGetErrorString(e));
    return PDM1_OK;
}
