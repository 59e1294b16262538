// Float64 perturbation field at listed points, by either far rule: the kernels
// behind spt_bem_field and the first pass of spt_accel.
#include "spt_device.cuh"

namespace spt {

// First point of the launch and the end of its points.
__device__ __forceinline__ long long field_range(const FieldMask& m, long long n, long long& end) {
    if (!m.active) {
        end = n;
        return 0;
    }
    end = m.group_offset[m.n_groups];
    return m.group_offset[0];
}

// Points the caller wants: all of them, or (spt_accel) the active particles in
// the valid region with blend weight > 0.  The others get a zero field:
// spt_accel's second launch makes this test again, compiled by itself, and a
// point on the threshold to the last bit must not find there what the caller's
// memory held.
__device__ __forceinline__ bool field_wanted(const FieldMask& m, long long i, double x, double y, double z) {
    if (!m.active) return true;
    if (!m.active[i] || !(blend_weight(z, m.g.z_handoff) > 0.0)) return false;
    if (m.g.kind == SPT_GEOM_TIP_BEM) return bem_valid<SPT_GEOM_TIP_BEM>(x, y, z, m.g);
    if (m.g.kind == SPT_GEOM_WELL_BEM) return bem_valid<SPT_GEOM_WELL_BEM>(x, y, z, m.g);
    return bem_valid<SPT_GEOM_POST_BEM>(x, y, z, m.g);
}

// The adaptive rule: a CTA takes `chunk` points (1 to 256: fewer than its warps
// while that leaves SMs free, so that a point's direct sums are shared).  Every thread finds its point's cell
// of the field map; mapped points are evaluated by the warp they sit in, the
// others (near the surface, or no map) go to a task list that all warps of the
// CTA draw from, one warp a point.
__global__ void __launch_bounds__(kMaxThreads, 2)
field_points_kernel(const double* x, const double* y, const double* z, long long n, int chunk,
                    const __grid_constant__ SptBem bem, const __grid_constant__ FieldMask mask, double* ex, double* ey,
                    double* ez) {
    extern __shared__ __align__(16) double smem[];
    __shared__ SptGeometry s_geo;
    __shared__ double s_p[3 * kMaxThreads], s_rec[kMaxWarps][8];
    __shared__ int s_task[kMaxThreads];
    __shared__ int s_n, s_next;
    __shared__ unsigned long long s_cnt[SPT_N_COUNTERS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) s_n = s_next = 0;
    __syncthreads();
    Ctx c(s_geo, bem);
    c.nt = kMaxThreads;
    c.nw = kMaxWarps;
    c.cnt = s_cnt;
    c.tiles = smem;
    c.wrec = s_rec[warp];
    const double* const map = field_map(bem);
    // point of this thread: lane + 32 warp of a full chunk, fewer lanes a warp in a small one
    const int per_warp = (chunk + kMaxWarps - 1) / kMaxWarps;
    long long end;
    const long long first = field_range(mask, n, end) + blockIdx.x * (long long)chunk;
    const long long i = first + warp * per_warp + lane;
    bool in = lane < per_warp && warp * per_warp + lane < chunk && i < end;
    double px = 0.0, py = 0.0, pz = 0.0;
    int leaf = -1;
    if (in) {
        px = x[i];
        py = y[i];
        pz = z[i];
        in = field_wanted(mask, i, px, py, pz);
        if (!in) ex[i] = ey[i] = ez[i] = 0.0;
    }
    if (map) {
        const double rho = hypot(px, py);
        if (in) leaf = map_find(map, rho, pz);
        double er = 0.0, fx, fy, fz = 0.0;
        map_field_lanes(map, leaf, rho, pz, er, fz);
        if (leaf >= 0) {
            rotate_rho(px, py, rho, er, fx, fy);
            ex[i] = fx;
            ey[i] = fy;
            ez[i] = fz;
        }
    }
    if (in && leaf < 0) {
        s_p[tid] = px;
        s_p[kMaxThreads + tid] = py;
        s_p[2 * kMaxThreads + tid] = pz;
        s_task[atomicAdd(&s_n, 1)] = tid;
    }
    __syncthreads();
    const int n_direct = s_n, shares = chunk < kMaxWarps ? split_shares(n_direct, kMaxWarps) : 1;
    double* const part = smem + kMaxWarps * (kWarpScratchInts / 2);
    PointCounts pts;
    auto store = [&](int k, double er, double fz) {  // lane 0
        double fx, fy;
        rotate_rho(s_p[k], s_p[kMaxThreads + k], hypot(s_p[k], s_p[kMaxThreads + k]), er, fx, fy);
        const long long o = first + (k >> 5) * per_warp + (k & 31);
        ex[o] = fx;
        ey[o] = fy;
        ez[o] = fz;
    };
    for (;;) {
        const int t = next_task(&s_next);
        if (t >= n_direct * shares) break;
        const int k = s_task[t / shares];
        PointSums S(t & (shares - 1), shares);
        direct_sums<SPT_FORM_FP64>(c, s_p[k], s_p[kMaxThreads + k], s_p[2 * kMaxThreads + k], S, pts);
        if (shares == 1) {
            double er, fz;
            S.total(er, fz);
            if (lane == 0) store(k, er, fz);
        } else {
            split_store(S, part + 256 * (t / shares));
        }
    }
    if (shares == 1) return;
    __syncthreads();
    for (int t = warp; t < n_direct; t += kMaxWarps) {
        double er, fz;
        split_total(part + 256 * t, er, fz);
        if (lane == 0) store(s_task[t], er, fz);
    }
}

// The reference rule: every far segment on its sub-panel nodes.  A point's
// segments are split, in runs of 32, over S warps (1 to 64: up to eight of one
// CTA, then over a cluster), so that a call of one point and one of a million
// both fill the SMs; with S = 1 a warp needs nobody else.  Each warp takes its
// run's near flags as one ballot, then two nodes a lane at a time straight
// from L1/L2 (24 bytes for ~100 FP64 instructions: the rings bound it), sums
// in registers, and the partial sums are added in a fixed order.  The near
// quadrature is the first warp's.  1500 points of the 64,000-ring tip: 0.82 ms,
// 118 G rings/s (6.7 ms as 24 CTAs of 64 points that stream the nodes through
// shared memory); 4000 points of the 39-panel hemisphere 0.16 ms (0.32).
__global__ void __launch_bounds__(kMaxThreads, 2)
field_quad_kernel(const double* x, const double* y, const double* z, long long n, int in_cta, int ranks,
                  unsigned nps_inv, const __grid_constant__ SptBem bem, const __grid_constant__ FieldMask mask,
                  double* ex, double* ey, double* ez) {
    __shared__ SptGeometry s_geo;
    __shared__ double s_rec[kMaxWarps][12];
    __shared__ double s_part[2 * kMaxWarps * 8];  // [rank][warp][component] on rank 0
    __shared__ unsigned long long s_cnt[SPT_N_COUNTERS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int slot = warp / in_cta, sub = warp - slot * in_cta;   // this CTA's point, this warp's share of it
    const int rank = (int)(blockIdx.x % ranks), per_cta = kMaxWarps / in_cta;
    long long end;
    const long long i = field_range(mask, n, end) + (long long)(blockIdx.x / ranks) * per_cta + slot;
    Ctx c(s_geo, bem);
    c.nt = kMaxThreads;
    c.nw = kMaxWarps;
    c.cnt = s_cnt;
    c.bpt = s_rec[slot];  // the record of the point, shared by its warps
    c.ntmp = c.bpt + 8;
    // (a CTA of the cluster may write to another's shared memory only once that one has started)
    if (ranks > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    double px = 0.0, py = 0.0, pz = 0.0;
    bool in = i < end;
    if (in) {
        px = x[i];
        py = y[i];
        pz = z[i];
        in = field_wanted(mask, i, px, py, pz);
        if (!in && sub == 0 && rank == 0 && lane == 0) ex[i] = ey[i] = ez[i] = 0.0;
    }
    PointCounts cnt;
    if (in && sub == 0) {
        if (lane == 0) {
            c.bpt[0] = px;
            c.bpt[1] = py;
            c.bpt[2] = pz;
            c.bpt[7] = c.ntmp[2] = 0.0;
        }
        __syncwarp();
        closest_point(c, c.bpt, 0, false);
        __syncwarp();
    }
    if (in_cta > 1) __syncthreads();
    double ar = 0.0, az = 0.0;
    if (in) {
        const int nseg = bem.n_seg, nps = bem.nodes_per_seg;
        const int n_run = (nseg + 31) / 32, share = in_cta * ranks, part = rank * in_cta + sub;
        const int q0 = (int)((long long)n_run * part / share), q1 = (int)((long long)n_run * (part + 1) / share);
        const double rho = c.bpt[3], zz = c.bpt[4], inv = rho > 0.0 ? 1.0 / rho : 0.0;
        const double* nr = bem.node;
        const double* nz = bem.node + bem.node_stride;
        const double* nw = bem.node + 2 * bem.node_stride;
        for (int q = q0; q < q1; ++q) {
            const int s = 32 * q + lane, ns = min(32, nseg - 32 * q);
            unsigned m = 0;
            if (!(bem.blk && blk_lower(bem, q, rho, zz) >= blk_lmax(bem, q))) {
                double proj, dist;
                m = __ballot_sync(0xffffffffu, s < nseg && seg_near(bem, s, rho, zz, proj, dist));
            }
            const size_t base = (size_t)32 * q * nps;
            for (int k = lane; k < ns * nps; k += 64) {
                const int k1 = k + 32 < ns * nps ? k + 32 : k;
                const double r0 = __ldg(nr + base + k), z0 = __ldg(nz + base + k);
                const double r1 = __ldg(nr + base + k1), z1 = __ldg(nz + base + k1);
                double w0 = __ldg(nw + base + k), w1 = __ldg(nw + base + k1);
                // near segments and the padding of the last pair count nothing (their field may be anything)
                const bool on0 = !((m >> __umulhi((unsigned)k, nps_inv)) & 1u);
                const bool on1 = k1 != k && !((m >> __umulhi((unsigned)k1, nps_inv)) & 1u);
                double er0, ez0, er1, ez1;
                ring_field_far<false, false>(rho, inv, zz - z0, r0, er0, ez0);
                ring_field_far<false, false>(rho, inv, zz - z1, r1, er1, ez1);
                if (on0) {
                    ar = fma(w0, er0, ar);
                    az = fma(w0, ez0, az);
                }
                if (on1) {
                    ar = fma(w1, er1, ar);
                    az = fma(w1, ez1, az);
                }
            }
        }
        ar = warp_sum(ar);
        az = warp_sum(az);
        if (part == 0) near_point(c, c.bpt, 0, cnt);
    }
    if (in_cta > 1) {
        // partial sums to the first rank's shared memory
        if (ranks > 1) {
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
            if (lane == 0) {
                const uint32_t at = smem_u32(s_part + 2 * (rank * kMaxWarps + warp));
                uint32_t remote;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(at), "r"(0));
                asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(remote), "d"(ar) : "memory");
                asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(remote + 8), "d"(az) : "memory");
            }
            asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
        } else {
            if (lane == 0) {
                s_part[2 * warp] = ar;
                s_part[2 * warp + 1] = az;
            }
            __syncthreads();
        }
        if (sub != 0 || rank != 0) return;
        ar = az = 0.0;
        for (int r = 0; r < ranks; ++r)
            for (int w = 0; w < in_cta; ++w) {
                ar += s_part[2 * (r * kMaxWarps + slot * in_cta + w)];
                az += s_part[2 * (r * kMaxWarps + slot * in_cta + w) + 1];
            }
    }
    __syncwarp();
    if (in && lane == 0) {
        double fx, fy;
        rotate_rho(px, py, hypot(px, py), ar + c.bpt[7], fx, fy);
        ex[i] = fx;
        ey[i] = fy;
        ez[i] = az + c.ntmp[2];
    }
}

// Launches the field of about n points (the work split is chosen for n, the
// grid covers `most`; what lies past the masked range returns at once); 0, a
// cudaError_t, or -1 for too many points.
int launch_field(const double* x, const double* y, const double* z, long long n, long long most, const SptBem& b,
                 const FieldMask& mask, double* ex, double* ey, double* ez, cudaStream_t st) {
    constexpr long long kWarps = 148 * 2 * kMaxWarps;  // resident warps: two CTAs of 128 registers a thread on each SM
    if (b.far_rule == SPT_FAR_ADAPTIVE) {
        // 1, 2, 4 points a CTA while every CTA finds a place at once, then chunks of 8 a resident warp
        constexpr long long kCtas = 148 * 2;
        long long chunk = n <= kCtas ? 1 : (n <= 2 * kCtas ? 2 : (n <= 4 * kCtas ? 4 : 8 * ((n + kWarps - 1) / kWarps)));
        if (chunk > kMaxThreads) chunk = kMaxThreads;
        const size_t smem = kMaxWarps * (kWarpScratchInts * 4) + (chunk < kMaxWarps ? split_doubles(kMaxWarps) * 8 : 0);
        const long long grid = (most + chunk - 1) / chunk;
        if (grid > 0x7fffffffLL) return -1;
        // (under the 48 KiB that need no attribute: one set per call would be two threads' to race for)
        field_points_kernel<<<(unsigned)grid, kMaxThreads, smem, st>>>(x, y, z, n, (int)chunk, b, mask, ex, ey, ez);
        return (int)cudaGetLastError();
    }
    // Enough shares for four rounds of every resident warp (at one the last,
    // part-filled round costs up to half the time), no more than the runs;
    // clusters of up to 8 CTAs.
    const int n_run = (b.n_seg + 31) / 32;
    int shares = 1;
    while (shares < 64 && n * shares < 4 * kWarps && 2 * shares <= n_run) shares *= 2;
    const int in_cta = shares < kMaxWarps ? shares : kMaxWarps, ranks = shares / in_cta;
    const long long grid = (most * in_cta + kMaxWarps - 1) / kMaxWarps * ranks;
    if (grid > 0x7fffffffLL) return -1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(kMaxThreads);
    cfg.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)ranks;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = ranks > 1 ? 1 : 0;
    // floor(k / nps) = umulhi(k, nps_inv) for k below 32 nps <= 8192
    const unsigned nps_inv = (unsigned)(0x100000000ULL / b.nodes_per_seg) + 1u;
    return (int)cudaLaunchKernelEx(&cfg, field_quad_kernel, x, y, z, n, in_cta, ranks, nps_inv, b, mask, ex, ey, ez);
}

}  // namespace spt
