// Field map of a BEM solution: classification of candidate cells and the cells'
// polynomials (spt_map_classify, spt_map_cells; include/spt_b200.h gives the
// layout, spt_device.cuh the lookup and the evaluation).  Built once per
// geometry; the host (bem_b200/field_map.py) walks the quadtree.
#include "spt_abi.hpp"
#include "spt_device.cuh"

namespace spt {

// One warp per candidate cell, lanes over the panels.
__global__ void __launch_bounds__(kMaxThreads)
map_classify_kernel(const double* cells, int n, const __grid_constant__ SptBem b, double kappa, int* flag,
                    double* far_ratio) {
    const int k = (int)((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (k >= n) return;
    const double r = cells[3 * k], z = cells[3 * k + 1], h = cells[3 * k + 2];
    const double diag = 1.4142135623730951 * h;  // the corners' distance from the centre
    double best = INFINITY;
    int bs = 0;
    bool clear = true, inside = false;  // outside every panel's band; wholly inside one's
    for (int s = lane; s < b.n_seg; s += 32) {
        double proj, d;
        seg_near(b, s, r, z, proj, d);
        const double band = SPT_MAP_BAND * segf(b, 4, s);
        if (!(d - diag >= band)) clear = false;
        if (d + diag < band) inside = true;
        if (d < best) { best = d; bs = s; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int os = __shfl_xor_sync(0xffffffffu, bs, o);
        if (ob < best || (ob == best && os < bs)) { best = ob; bs = os; }
    }
    clear = __all_sync(0xffffffffu, clear);
    inside = __any_sync(0xffffffffu, inside);
    if (lane == 0) {
        const double side = (r - segf(b, 0, bs)) * segf(b, 7, bs) + (z - segf(b, 1, bs)) * segf(b, 8, bs);
        const bool behind = side < 0.0 && best > diag;  // the normals point into the vacuum
        int f = 0;
        if (inside || behind) f = 2;
        else if (clear && best >= kappa * h) f = 1;
        else if (h < 0.125 * segf(b, 4, bs)) f = 2;
        flag[k] = f;
        far_ratio[k] = best / h;
    }
}

// One CTA per cell: its N x N samples, one warp a sample, then the transform
// of both components.  To Chebyshev coefficients first (stable: their rounding
// is that of the samples), then to powers, whose coefficients inherit the
// Chebyshev ones' decay.  Bound by the samples' ring sums, as the direct path.
constexpr int kMapN2 = SPT_MAP_N * SPT_MAP_N;
__global__ void __launch_bounds__(kMaxThreads, 2)
map_cells_kernel(const double* cells, const __grid_constant__ SptBem bem, const double* cheb, const double* dct,
                 const double* mono, double* rec, double* tail) {
    extern __shared__ __align__(16) double smem[];
    __shared__ SptGeometry s_geo;
    __shared__ double s_f[2 * kMapN2], s_t[2 * kMapN2], s_x[SPT_MAP_N], s_d[kMapN2], s_m[kMapN2];
    __shared__ double s_max[2][kMaxWarps];
    __shared__ unsigned long long s_cnt[SPT_N_COUNTERS];
    __shared__ int s_next;
    constexpr int N = SPT_MAP_N;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const double rc = cells[3 * blockIdx.x], zc = cells[3 * blockIdx.x + 1], h = cells[3 * blockIdx.x + 2];
    const bool axis = rc < 1.5 * h;  // nodes in rho^2 / (2 h^2) - 1, E_rho divided by rho / h
    if (tid < N) s_x[tid] = cheb[tid];
    for (int e = tid; e < kMapN2; e += blockDim.x) {
        s_d[e] = dct[e];
        s_m[e] = mono[e];
    }
    if (tid == 0) s_next = 0;
    Ctx c(s_geo, bem);
    c.nt = kMaxThreads;
    c.nw = kMaxWarps;
    c.cnt = s_cnt;
    c.tiles = smem;
    __syncthreads();
    PointCounts cnt;
    for (;;) {
        const int t = next_task(&s_next);
        if (t >= kMapN2) break;
        // rho: row i, z: row j; no panel is near
        PointSums S(0, 1);
        double er, ez, mr, mz, mabs;
        const double u = axis ? sqrt(2.0 * (1.0 + s_x[t / N])) : 1.0;  // rho / h on the axis
        far_adaptive_warp<false>(c, axis ? h * u : rc + h * s_x[t / N], zc + h * s_x[t % N], S, cnt, mr, mz, mabs);
        S.total(er, ez);
        if (lane == 0) {
            s_f[t] = er / u;
            s_f[kMapN2 + t] = ez;
        }
        __syncwarp();
    }
    // value at (node i, node j) -> T_k(x) T_l(y) -> x^i y^j, one axis at a time
    double big = 0.0, high = 0.0;
    for (int pass = 0; pass < 4; ++pass) {
        const double* src = pass & 1 ? s_t : s_f;
        double* dst = pass & 1 ? s_f : s_t;
        __syncthreads();
        for (int e = tid; e < 2 * kMapN2; e += blockDim.x) {
            const int comp = e / kMapN2, k = (e % kMapN2) / N, l = e % N;
            const double* f = src + comp * kMapN2;
            double v = 0.0;
            for (int q = 0; q < N; ++q) {
                if (pass == 0) v = fma(s_d[k * N + q], f[q * N + l], v);
                else if (pass == 1) v = fma(s_d[l * N + q], f[k * N + q], v);
                else if (pass == 2) v = fma(s_m[q * N + k], f[q * N + l], v);
                else v = fma(s_m[q * N + l], f[k * N + q], v);
            }
            dst[e] = v;
            if (pass == 1) {
                big = fmax(big, fabs(v));
                if (k >= N - 2 || l >= N - 2) high = fmax(high, fabs(v));
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        big = fmax(big, __shfl_xor_sync(0xffffffffu, big, o));
        high = fmax(high, __shfl_xor_sync(0xffffffffu, high, o));
    }
    if (lane == 0) {
        s_max[0][warp] = big;
        s_max[1][warp] = high;
    }
    __syncthreads();
    double* out = rec + (size_t)blockIdx.x * SPT_MAP_REC;
    if (tid < 8) out[tid] = tid == 0 ? rc : (tid == 1 ? zc : (tid == 2 ? 1.0 / h : 0.0));
    for (int e = tid; e < 2 * kMapN2; e += blockDim.x) {
        const int comp = e / kMapN2, i = (e % kMapN2) / N, j = e % N;
        out[8 + (2 * j + comp) * N + i] = s_f[e];
    }
    if (tid == 0) {
        double b = 0.0, t = 0.0;
        for (int w = 0; w < kMaxWarps; ++w) {
            b = fmax(b, s_max[0][w]);
            t = fmax(t, s_max[1][w]);
        }
        tail[blockIdx.x] = b > 0.0 ? t / b : 0.0;
    }
}

}  // namespace spt

using spt_abi::cuda_check;
using spt_abi::fail;

extern "C" int spt_map_classify(const double* cells, int32_t n, const SptBem* b, double kappa, int32_t* flag,
                                double* far_ratio, void* stream) {
    if (n <= 0) return SPT_OK;
    if (!cells || !flag || !far_ratio) return fail(SPT_ERR_ARG, "null argument");
    const int rc = spt_abi::check_bem(b);
    if (rc) return rc;
    const long long blocks = (n + spt::kMaxWarps - 1LL) / spt::kMaxWarps;
    spt::map_classify_kernel<<<(unsigned)blocks, spt::kMaxThreads, 0, static_cast<cudaStream_t>(stream)>>>(
        cells, n, *b, kappa, flag, far_ratio);
    return cuda_check(cudaGetLastError(), "map_classify_kernel launch");
}

extern "C" int spt_map_cells(const double* cells, int32_t n, const SptBem* b, const double* cheb, const double* dct,
                             const double* mono, double* rec, double* tail, void* stream) {
    if (n <= 0) return SPT_OK;
    if (!cells || !cheb || !dct || !mono || !rec || !tail) return fail(SPT_ERR_ARG, "null argument");
    const int rc = spt_abi::check_bem(b);
    if (rc) return rc;
    if (b->far_rule != SPT_FAR_ADAPTIVE || b->reserved)
        return fail(SPT_ERR_ARG, "spt_map_cells: needs the adaptive far rule's tables, without a map");
    const size_t smem = spt::kMaxWarps * spt::kWarpScratchInts * 4;
    spt::map_cells_kernel<<<(unsigned)n, spt::kMaxThreads, smem, static_cast<cudaStream_t>(stream)>>>(
        cells, *b, cheb, dct, mono, rec, tail);
    return cuda_check(cudaGetLastError(), "map_cells_kernel launch");
}
