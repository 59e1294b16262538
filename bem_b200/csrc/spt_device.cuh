// Device code of the B200 (sm_100a) tracer, shared by the translation units
// that instantiate the trace kernel per geometry kind (spt_trace_<kind>.cu)
// and by the C ABI (spt_kernels.cu).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>
#include <math.h>
#include <type_traits>

#include "../../include/spt_b200.h"
#include "spt_image.cuh"
#include "spt_math.cuh"
#include "spt_umma.cuh"

namespace spt {

// A CTA is one team of nt = blockDim.x threads (32, 64, 128 or 256) working on
// one group at a time; its width is a launch parameter (smaller CTAs for
// smaller groups: more CTAs per SM, fewer warps per barrier).  Static shared
// arrays are sized for the widest CTA.
constexpr int kMaxThreads = 256;
constexpr int kMaxWarps = kMaxThreads / 32;
constexpr int kRound = 4;           // points per far-sum round (largest; the register tile of the far sums)
constexpr double kKappa = 16.0;     // default conditioning bound of the mixed form's float32 sums
constexpr int kTileNodes = 2048;    // nodes per TMA tile row (largest; halved while shared memory is short)
constexpr size_t kMaxSmem = 226 * 1024;  // dynamic part; the static __shared__ scalars take the rest of 227 KB
constexpr int kSmallGroup = 256;    // groups above this keep slopes in global memory

// Dormand-Prince 5(4) tableau (batched_rk45.py:30-50).
static __device__ __constant__ double kA[6][5] = {
    {0, 0, 0, 0, 0},
    {1.0 / 5, 0, 0, 0, 0},
    {3.0 / 40, 9.0 / 40, 0, 0, 0},
    {44.0 / 45, -56.0 / 15, 32.0 / 9, 0, 0},
    {19372.0 / 6561, -25360.0 / 2187, 64448.0 / 6561, -212.0 / 729, 0},
    {9017.0 / 3168, -355.0 / 33, 46732.0 / 5247, 49.0 / 176, -5103.0 / 18656}};
static __device__ __constant__ double kB[6] = {35.0 / 384, 0.0, 500.0 / 1113, 125.0 / 192, -2187.0 / 6784, 11.0 / 84};
static __device__ __constant__ double kE[7] = {71.0 / 57600, 0.0, -71.0 / 16695, 71.0 / 1920, -17253.0 / 339200, 22.0 / 525, -1.0 / 40};

constexpr double kSpeedOfLight = 299792458.0;
constexpr double kTiny = 2.2250738585072014e-308;  // np.finfo(float).tiny

// ---------------------------------------------------------------------------
// small helpers
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ void tma_load_1d(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

// Bounded wait on an mbarrier phase.  Returns false when the iteration limit
// ran out (the caller flags the group instead of spinning forever).
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t phase) {
    uint32_t done = 0;
    for (int it = 0; it < (1 << 22); ++it) {
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(smem_u32(bar)), "r"(phase)
            : "memory");
        if (done) return true;
    }
    return false;
}

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// ---------------------------------------------------------------------------
// geometry helpers (fields.py, geometry.py, bem/fields.py, bem/geometry.py)

__device__ __forceinline__ bool well_contains(double rho, double z, const SptGeometry& g) {
    const double R = g.R, H = g.H;
    const double eps = 1e-6 * R;
    bool solid = (rho >= R * (1.0 - 1e-6)) ? (z <= 0.0) : (z <= -H * (1.0 + 1e-6));
    if (g.rim_fillet > 0.0) {
        const double rf = g.rim_fillet, cr = R + rf, cz = -rf;
        if (rho >= R - eps && rho <= R + rf + eps && z >= -rf - eps && z <= eps) solid = hypot(rho - cr, z - cz) <= rf;
    }
    if (g.bottom_fillet > 0.0) {
        const double bf = g.bottom_fillet, cr = R - bf, cz = -H + bf;
        if (rho <= R + eps && rho >= R - bf - eps && z <= -H + bf + eps && z >= -H - eps)
            solid = hypot(rho - cr, z - cz) >= bf;
    }
    return solid;
}

__device__ __forceinline__ bool post_inside(double x, double y, double z, const SptGeometry& g) {
    const double rk = g.R * (1.0 - 1e-6);
    const double r2 = x * x + y * y;
    const double zc = z - g.L;
    return (r2 <= rk * rk && z <= g.L) || (r2 + zc * zc <= rk * rk);
}

template <int KIND>
__device__ __forceinline__ bool kill_test(double x, double y, double z, const SptGeometry& g) {
    bool k = false;
    if (KIND == SPT_GEOM_FLAT) {
        k = g.has_kill_below && z <= g.kill_z_below;
    } else if (KIND == SPT_GEOM_TIP || KIND == SPT_GEOM_TIP_BEM) {
        const double rk = g.R * (1.0 - 1e-6);
        k = (x * x + y * y + z * z) <= rk * rk;
        if (g.has_kill_below) k = k || (z <= g.kill_z_below);
    } else if (KIND == SPT_GEOM_WELL_BEM) {
        k = well_contains(sqrt(x * x + y * y), z, g);
    } else {
        k = post_inside(x, y, z, g);
        if (g.has_kill_below) k = k || (z <= g.kill_z_below);
    }
    if (g.has_z_max) k = k || (z >= g.z_max);
    return k;
}

// analytic tip field (fields.py:119-160)
__device__ __forceinline__ void tip_field(double x, double y, double z, double Ez, double R, double& ex, double& ey,
                                          double& ez) {
    const double r = sqrt(x * x + y * y + z * z);
    const bool ok = (r >= R * (1.0 - 1e-6)) && (z >= 0.0);
    if (!ok) {
        ex = ey = ez = 0.0;
        return;
    }
    const double r3 = r * r * r;
    const double r5 = r3 * r * r;
    const double R3 = R * R * R;
    ex = 3.0 * Ez * R3 * x * z / r5;
    ey = 3.0 * Ez * R3 * y * z / r5;
    ez = Ez * (1.0 - R3 / r3 + 3.0 * R3 * z * z / r5);
}

// BEM geometries: is the point in the field's valid (vacuum) region
template <int KIND>
__device__ __forceinline__ bool bem_valid(double x, double y, double z, const SptGeometry& g) {
    if (KIND == SPT_GEOM_TIP_BEM) return (sqrt(x * x + y * y + z * z) >= g.R * (1.0 - 1e-6)) && (z >= 0.0);
    if (KIND == SPT_GEOM_WELL_BEM) return !well_contains(sqrt(x * x + y * y), z, g);
    return !post_inside(x, y, z, g) && (z >= 0.0);
}

__device__ __forceinline__ double blend_weight(double z, double zh) {
    const double zlo = 0.5 * zh;
    double s = (zh - z) / (zh - zlo);
    s = fmin(fmax(s, 0.0), 1.0);
    return s * s * (3.0 - 2.0 * s);
}

// ---------------------------------------------------------------------------
// shared-memory layout of one CTA

struct Layout {
    // offsets in doubles from the start of dynamic shared memory
    int y0, nw, sp, kp, kv;   // y0: 6E, nw: 6E, sp: 3E, kp/kv: 21E each
    int tb, td, q, m, cps;    // E each
    int fld;                  // 3E field
    int img;                  // 4E sphere images
    int bpt;                  // 8E per BEM list entry: x y z rho_e z_e near_r near_z (+1 pad)
    int imgs;                 // scratch of the BEM image-charge force (geometries with z0), or 0 doubles
    int sur;                  // surrogate region: act (4096), wt (4096), sout 2E, sseg E, st E, sd E, feat 128; -1 if none
    int tiles;                // reference far rule: 2 * 3 * tile_cap node tiles; adaptive: per-warp scratch
    int tile_cap;             // nodes per TMA tile row (reference far rule)
    int red;                  // kMaxWarps * 3 * kRound (far-round reduction: E_rho, E_z, sum of |terms|)
    int ints;                 // int region start (in doubles)
    int total_doubles;
    int list_off, lidx_off, live_off, flags_off;  // in ints from ints start
    size_t bytes;
    bool big;                 // slopes/y0/nw in global memory
};

// The adaptive far rule classifies 32 runs of SPT_BLOCK_SEGS segments at a time
// (a lane each) and the segments of up to kWarpChunk / SPT_BLOCK_SEGS of them
// before their nodes are summed.  Each warp keeps its lists in a private
// scratch of kWarpScratchInts ints: four segment lists and the near masks of
// the first (kWarpChunk bytes each: a segment by its place among the runs at
// hand), four run lists and the bits of the runs that cluster expansions cover.
constexpr int kWarpChunk = 256;
constexpr int kWarpRuns = 32;
constexpr int kWarpScratchInts = 5 * kWarpChunk / 4 + 4 * kWarpRuns + SPT_MAX_CLUSTER_RUNS / 32;
static_assert(kWarpScratchInts % 2 == 0, "per-warp scratch keeps 8-byte alignment");
// Shared slots of the points that several warps share (split_shares: at most
// half as many points as warps), per point 4 slots x 2 components x 32 lanes.
__host__ __device__ constexpr int split_doubles(int warps) { return warps / 2 * 256; }

// Shared-memory layout of one CTA for groups of up to E particles.  The far
// rule decides the big region: node tiles for the reference rule (the TMA
// bulk engine streams the node table through them), segment lists for the
// adaptive rule (which reads its few nodes through L1/L2), one scratch per
// warp of a CTA of `warps` warps.  want_tiles false: neither (paths that
// evaluate no far sum).
__host__ __device__ inline Layout make_layout(int E, int far_rule, bool want_sur = false, bool want_tiles = true,
                                              int warps = kMaxWarps, int img_doubles = 0, bool slopes = true) {
    Layout L;
    const bool big = E > kSmallGroup;
    int o = 0;
    L.big = big;
    if (!slopes) {  // one stage only: its result
        L.y0 = L.nw = L.kp = 0;
        L.kv = o; o += 3 * E;
    } else if (!big) {
        L.y0 = o; o += 6 * E;
        L.nw = o; o += 6 * E;
        L.kp = o; o += 21 * E;
        L.kv = o; o += 21 * E;
    } else {
        L.y0 = L.nw = L.kp = L.kv = -1;
    }
    L.sp = o; o += 3 * E;
    L.tb = o; o += E;
    L.td = o; o += E;
    L.q = o; o += E;
    L.m = o; o += E;
    L.cps = o; o += E;
    L.fld = o; o += 3 * E;
    L.img = o; o += 4 * E;
    L.bpt = o; o += 8 * E;
    L.imgs = o; o += img_doubles;
    if (want_sur) {
        o = (o + 127) & ~127;  // 1 KiB alignment for the tensor-core operand tiles
        L.sur = o; o += 8192 + 5 * E + 128;
    } else {
        L.sur = -1;
    }
    o = (o + 1) & ~1;  // 16-byte alignment for the TMA tiles
    const int base = o;
    // list (ints), live list (16 bits each), live (bytes), near flags (bytes), redo flag, live count: no more
    // than two ints a particle, as the group sizes that a CTA holds are part of the interface
    L.list_off = 0;
    L.lidx_off = E;
    L.live_off = L.lidx_off + (E + 1) / 2;
    L.flags_off = L.live_off + (E + 3) / 4;
    const int n_ints = L.flags_off + kRound * 256 / 4 + 3;
    const bool tiles = want_tiles && far_rule == SPT_FAR_REFERENCE;
    const bool lists = want_tiles && far_rule != SPT_FAR_REFERENCE;
    for (int cap = kTileNodes; cap >= 256; cap >>= 1) {
        o = base;
        L.tile_cap = tiles ? cap : 0;
        L.tiles = o; o += tiles ? 2 * 3 * cap : (lists ? warps * (kWarpScratchInts / 2) + split_doubles(warps) : 0);
        L.red = o; o += kMaxWarps * 3 * kRound;
        L.ints = o;
        L.total_doubles = o + (n_ints + 1) / 2;
        L.bytes = (size_t)L.total_doubles * 8 + 64;  // + mbarriers
        if (L.bytes <= kMaxSmem || !tiles) break;
    }
    return L;
}

// Partial right-hand sides of the image-charge solve per profile node: as
// many source subsets as the CTA has threads per node, 1 to 4.
__host__ __device__ inline int image_chunks(int P, int threads) {
    const int c = threads / (P > 0 ? P : 1);
    return c < 1 ? 1 : (c > 4 ? 4 : c);
}

// Shared doubles the BEM image-charge force needs for groups of up to E
// particles on a CTA of `threads` threads: 0 unless the geometry is a BEM
// tip or well built with z0 and the image tables are given.
__host__ __device__ inline int image_scratch(const SptGeometry& g, const SptBem& b, int E, int threads) {
    if (!(g.kind == SPT_GEOM_TIP_BEM || g.kind == SPT_GEOM_WELL_BEM) || !g.has_image || b.image.n_nodes < 2) return 0;
    return (int)spt_img::scratch_doubles(E, b.image.mirror_symmetric, b.image.n_nodes, b.image.n_max,
                                         image_chunks(b.image.n_nodes, threads));
}

// global per-CTA slot for big groups: y0 6E, nw 6E, kp 21E, kv 21E
__host__ __device__ inline size_t big_slot_doubles(int E) { return (size_t)54 * E; }

struct Ctx {
    // the kernel's parameter blocks (__grid_constant__: referenced in place, never copied)
    const SptGeometry& g;
    const SptBem& bem;
    __device__ Ctx(const SptGeometry& g_, const SptBem& b_) : g(g_), bem(b_) {}
    int nt, nw;      // threads and warps of this CTA (blockDim.x, a multiple of 32)
    double cm;       // charge_to_mass
    double kc;       // Coulomb constant 1/(4 pi eps0)
    double soft2;    // plummer^2
    int round_pts;           // points per far-sum round, 1..kRound
    double kappa;            // mixed form: float32 sums whose sum of |terms| exceeds kappa x |result| are redone in float64
    int* redo;               // shared flag of that test
    int E;
    double* base;    // dynamic smem
    Layout L;
    double *y0, *nw_, *sp, *kp, *kv, *tb, *td, *q, *m, *cps, *fld, *img, *bpt, *tiles, *red, *imgs;
    double* ntmp;    // reference rule: near sums' E_z per record (stride 3)
    double* wrec;    // adaptive rule: this warp's record (8 doubles)
    unsigned char* live;
    int* list;
    uint16_t* lidx;  // live particles in order
    int* nl;         // and their number
    unsigned char* nflag;
    uint64_t* bars;
    uint32_t phase[3];          // parity of the next phase to wait for on bars[0..2] (identical in every thread)
    unsigned long long* cnt;    // shared-memory counter partials of the CTA (flushed by flush_counters)
    unsigned long long pairs = 0;  // this thread's pair interactions since the last group
    // learned form
    uint8_t *act, *wt;          // BF16 operand tiles (activations, weights), canonical K-major, 32 KiB each
    double *sout, *st, *sd;     // surrogate E (rho, z) per record; closest-point parameter and distance
    int* sseg;                  // closest segment per record
    float* feat;                // features of the current 128-row chunk
    const float* sw;            // FP32 (BF16-rounded) parameters
    const __nv_bfloat16* sw16;  // BF16 parameters
    const double *s_start, *log_scale;
    double s_end, sig_floor, band, spot, dmin, dmax;
    unsigned long long* sstats;
    uint32_t tmem;
    uint32_t key;               // hash key of the current stage evaluation (spot checks)
};

// add v (a per-thread partial) to the CTA's counter k: warp sum, one shared atomic per warp
__device__ __forceinline__ void count_add(Ctx& c, int k, unsigned long long v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(c.cnt + k, v);
}

__device__ inline void bind(Ctx& c, double* smem, int E, int far_rule, double* slot, unsigned long long* s_cnt,
                            bool sur = false, bool tiles = true, bool slopes = true) {
    c.base = smem;
    c.E = E;
    c.nt = blockDim.x;
    c.nw = blockDim.x >> 5;
    c.L = make_layout(E, far_rule, sur, tiles, blockDim.x >> 5, image_scratch(c.g, c.bem, E, blockDim.x), slopes);
    c.round_pts = kRound;
    c.kappa = kKappa;
    c.cnt = s_cnt;
    const Layout& L = c.L;
    if (!L.big) {
        c.y0 = smem + L.y0;
        c.nw_ = smem + L.nw;
        c.kp = smem + L.kp;
        c.kv = smem + L.kv;
    } else {
        c.y0 = slot;
        c.nw_ = slot + 6 * E;
        c.kp = slot + 12 * E;
        c.kv = slot + 33 * E;
    }
    c.sp = smem + L.sp;
    c.tb = smem + L.tb;
    c.td = smem + L.td;
    c.q = smem + L.q;
    c.m = smem + L.m;
    c.cps = smem + L.cps;
    c.fld = smem + L.fld;
    c.ntmp = c.fld;
    c.img = smem + L.img;
    c.bpt = smem + L.bpt;
    c.imgs = smem + L.imgs;
    c.tiles = smem + L.tiles;
    c.red = smem + L.red;
    c.wrec = c.red + 8 * (threadIdx.x >> 5);  // (the adaptive rule has no block reduction)
    int* ib = reinterpret_cast<int*>(smem + L.ints);
    c.list = ib + L.list_off;
    c.lidx = reinterpret_cast<uint16_t*>(ib + L.lidx_off);
    c.live = reinterpret_cast<unsigned char*>(ib + L.live_off);
    c.nflag = reinterpret_cast<unsigned char*>(ib + L.flags_off);
    c.redo = ib + L.flags_off + kRound * 256 / 4;  // first spare int after the near-flag bytes
    c.nl = c.redo + 1;
    c.bars = reinterpret_cast<uint64_t*>(smem + L.total_doubles + 1);
    for (int k = threadIdx.x; k < SPT_N_COUNTERS; k += blockDim.x) s_cnt[k] = 0;
    if (L.sur >= 0) {
        double* r = smem + L.sur;
        c.act = reinterpret_cast<uint8_t*>(r);
        c.wt = reinterpret_cast<uint8_t*>(r + 4096);
        c.sout = r + 8192;
        c.st = c.sout + 2 * E;
        c.sd = c.st + E;
        c.sseg = reinterpret_cast<int*>(c.sd + E);
        c.feat = reinterpret_cast<float*>(c.sd + 2 * E);
    }
}

// ---------------------------------------------------------------------------
// BEM: segment table access

struct Seg {
    double p0r, p0z, tr, tz, len, ur, uz, nr, nz, s0, s1;
};

__device__ __forceinline__ double segf(const SptBem& b, int f, int s) { return __ldg(b.seg + (size_t)f * b.seg_stride + s); }

// closest-point distance^2 of (rq, zq) to segment s (bem/axisymmetric.py:117-133,
// 374-381), with no FMA contraction: the on-surface offset below is a
// threshold test on this value, so it is rounded like the reference's.
__device__ __forceinline__ double seg_dist2(const SptBem& b, int s, double rq, double zq) {
    const double p0x = segf(b, 0, s), p0y = segf(b, 1, s), ax = segf(b, 2, s), ay = segf(b, 3, s);
    const double ab = __dadd_rn(__dmul_rn(ax, ax), __dmul_rn(ay, ay));
    double t = __ddiv_rn(__dadd_rn(__dmul_rn(__dadd_rn(rq, -p0x), ax), __dmul_rn(__dadd_rn(zq, -p0y), ay)), ab);
    t = fmin(fmax(t, 0.0), 1.0);
    const double cr = __dadd_rn(p0x, __dmul_rn(t, ax)), cz = __dadd_rn(p0y, __dmul_rn(t, ay));
    const double dr = __dadd_rn(rq, -cr), dz = __dadd_rn(zq, -cz);
    return __dadd_rn(__dmul_rn(dr, dr), __dmul_rn(dz, dz));
}

// Distance from its components, branch-free: 1e-300 keeps the square off zero (it
// rounds away beside any real one), and a NaN stays a NaN, which is near no
// panel (fmax in its place gave the bound for a NaN).
__device__ __forceinline__ double dist_pos(double x, double y) { return sqrt_pos(fma(x, x, fma(y, y, 1e-300))); }

// near test of bem/axisymmetric.py:566-570 -> (near, projection, distance)
// FAST (the adaptive rule): a branch-free root, exact to the last bit or two.
template <bool FAST = false>
__device__ __forceinline__ bool seg_near(const SptBem& b, int s, double re, double ze, double& proj, double& dist) {
    const double p0r = segf(b, 0, s), p0z = segf(b, 1, s), L = segf(b, 4, s), ur = segf(b, 5, s), uz = segf(b, 6, s);
    const double dr = re - p0r, dz = ze - p0z;
    const double along = dr * ur + dz * uz;
    proj = fmin(fmax(along, 0.0), L);
    const double ar = dr - proj * ur, az = dz - proj * uz;
    if constexpr (FAST) dist = dist_pos(ar, az);
    else dist = sqrt(ar * ar + az * az);
    return dist < L;
}

// Runs of SPT_BLOCK_SEGS consecutive segments (SptBem.blk): a lower bound of
// the distance from (r, z) to every segment of run q, less a relative margin
// that covers the rounding of this bound and of the table, and the run's
// largest segment length.
__device__ __forceinline__ double blk_lower(const SptBem& b, int q, double r, double z) {
    const double cr = __ldg(b.blk + q), cz = __ldg(b.blk + b.blk_stride + q), rad = __ldg(b.blk + 2 * b.blk_stride + q);
    const double dr = r - cr, dz = z - cz;
    const double dc = dist_pos(dr, dz);
    return dc - rad - 1e-9 * (dc + rad);
}
__device__ __forceinline__ double blk_lmax(const SptBem& b, int q) { return __ldg(b.blk + 3 * b.blk_stride + q); }


// Fixed-order block reduction of a far round's accumulators into record
// slots 5, 6 (far + near sums).  Mixed form: the Kahan sums are folded in,
// and when the sum of |float32 terms| at a point exceeds kappa times the
// whole field there (uniform + perturbation), *c.redo is set -- the float32
// result is then ill-conditioned (shielded regions, where the perturbation
// cancels the uniform field) and the caller recomputes the round in float64.
template <int NP, bool MIX>
__device__ __forceinline__ void round_reduce(Ctx& c, int r0, int np_, double* ar, double* az, const float* fr,
                                             const float* fz, const float* kr, const float* kz, const float* sa) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double* P = c.bpt;
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        if (MIX) {
            ar[p] += (double)fr[p] - (double)kr[p];
            az[p] += (double)fz[p] - (double)kz[p];
        }
        const double vr = warp_sum(ar[p]);
        const double vz = warp_sum(az[p]);
        const double va = MIX ? warp_sum((double)sa[p]) : 0.0;
        if (lane == 0) {
            c.red[warp * 3 * kRound + p] = vr;
            c.red[warp * 3 * kRound + kRound + p] = vz;
            c.red[warp * 3 * kRound + 2 * kRound + p] = va;
        }
    }
    __syncthreads();
    if (tid < np_) {
        double sr = 0.0, sz = 0.0, sabs = 0.0;
        for (int w = 0; w < c.nw; ++w) {
            sr += c.red[w * 3 * kRound + tid];
            sz += c.red[w * 3 * kRound + kRound + tid];
            sabs += c.red[w * 3 * kRound + 2 * kRound + tid];
        }
        const int k = r0 + tid;
        const double er = sr + P[8 * k + 7], ez = sz + c.ntmp[3 * k + 2];
        P[8 * k + 5] = er;
        P[8 * k + 6] = ez;
        if (MIX) {
            const double tz = ez + c.g.E_gun;
            if (!(sabs <= c.kappa * sqrt(er * er + tz * tz))) atomicOr(c.redo, 1);
        }
    }
    __syncthreads();
}

// One far-sum round for points r0..r0+np_-1 of the list (np_ <= NP): the
// node table streams through shared memory in TMA tiles (double buffered);
// each thread takes NQ nodes at a time, strided by the CTA width, against
// all NP points (NP * NQ independent ring evaluations per iteration).
template <int NP, int NQ, bool MIX>
__device__ void far_round(Ctx& c, int r0, int np_, int n_tiles, int segs_per_tile, bool& ok,
                          unsigned long long& far_evals) {
    const SptBem& b = c.bem;
    const int tid = threadIdx.x;
    const int nseg = b.n_seg, nps = b.nodes_per_seg;
    const int tile_cap = c.L.tile_cap;
    double* P = c.bpt;
    double* tile[2] = {c.tiles, c.tiles + 3 * tile_cap};
    uint64_t* bars = c.bars;
    double pr[NP], pinv[NP], pz[NP], ar[NP], az[NP];
    float fr[NP], fz[NP], kr[NP], kz[NP], prf[NP], pinvf[NP];  // mixed form: Kahan sums and float copies
    float sa[NP];                                               // mixed form: sum of |float32 terms|
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        const int k = r0 + (p < np_ ? p : 0);
        pr[p] = P[8 * k + 3];
        pinv[p] = pr[p] > 0.0 ? 1.0 / pr[p] : 0.0;
        pz[p] = P[8 * k + 4];
        ar[p] = 0.0;
        az[p] = 0.0;
        fr[p] = fz[p] = kr[p] = kz[p] = sa[p] = 0.0f;
        prf[p] = (float)pr[p];
        pinvf[p] = (float)pinv[p];
    }
    if (MIX && tid == 0) *c.redo = 0;  // ordered before the reduction's writes by the barriers between
    auto issue = [&](int t, int buf) {
        const int s_first = t * segs_per_tile;
        const int nn = min(segs_per_tile, nseg - s_first) * nps;
        const uint32_t bytes = (uint32_t)nn * 8u;
        mbar_expect_tx(&bars[buf], 3u * bytes);
        for (int row = 0; row < 3; ++row)
            tma_load_1d(tile[buf] + row * tile_cap, b.node + (size_t)row * b.node_stride + (size_t)s_first * nps, bytes,
                        &bars[buf]);
    };
    if (tid == 0) {
        issue(0, 0);
        if (n_tiles > 1) issue(1, 1);
    }
    for (int t = 0; t < n_tiles; ++t) {
        const int buf = t & 1;
        const int s_first = t * segs_per_tile;
        const int ns = min(segs_per_tile, nseg - s_first);
        for (int idx = tid; idx < np_ * ns; idx += c.nt) {
            const int p = idx / ns, sl = idx - p * ns;
            double proj, dist;
            c.nflag[p * 256 + sl] = seg_near(b, s_first + sl, P[8 * (r0 + p) + 3], P[8 * (r0 + p) + 4], proj, dist);
        }
        if (!mbar_wait(&bars[buf], c.phase[buf])) ok = false;
        c.phase[buf] ^= 1u;
        __syncthreads();
        if (ok) {
            const double* tr = tile[buf];
            const double* tz = tr + tile_cap;
            const double* tw = tz + tile_cap;
            const int nn = ns * nps;
            for (int q0 = tid; q0 < nn; q0 += c.nt * NQ) {
                double rq[NQ], zq[NQ], wq[NQ];
                int sl[NQ];
                bool in[NQ];
#pragma unroll
                for (int j = 0; j < NQ; ++j) {
                    const int q = q0 + j * c.nt;
                    in[j] = q < nn;
                    const int qq = in[j] ? q : 0;
                    rq[j] = tr[qq];
                    zq[j] = tz[qq];
                    wq[j] = tw[qq];
                    sl[j] = qq / nps;
                }
                if (MIX) {
                    // float32 Kahan sums; pairs the float path declines (p < 1e-3 or
                    // near the axis) are evaluated in float64
#pragma unroll
                    for (int p = 0; p < NP; ++p) {
#pragma unroll
                        for (int j = 0; j < NQ; ++j) {
                            if (p < np_ && in[j] && !c.nflag[p * 256 + sl[j]]) {
                                const double dz = pz[p] - zq[j];
                                float er, ez;
                                if (ring_far_f(prf[p], pinvf[p], (float)(pr[p] - rq[j]), (float)(pr[p] + rq[j]),
                                               (float)dz, (float)rq[j], er, ez)) {
                                    const float w = (float)wq[j];
                                    kahan_add(fr[p], kr[p], w * er);
                                    kahan_add(fz[p], kz[p], w * ez);
                                    sa[p] += fabsf(w * er) + fabsf(w * ez);
                                } else {
                                    // close to the ring: the term in float64, summed like the others
                                    double e64r, e64z;
                                    ring_field_far_cold(pr[p], 1.0 / pr[p], dz, rq[j], e64r, e64z);
                                    const float ter = (float)(wq[j] * e64r), tez = (float)(wq[j] * e64z);
                                    kahan_add(fr[p], kr[p], ter);
                                    kahan_add(fz[p], kz[p], tez);
                                    sa[p] += fabsf(ter) + fabsf(tez);
                                }
                                ++far_evals;
                            }
                        }
                    }
                } else {
                // a point's NQ terms are added first: one step of the running sum's chain for all of them
#pragma unroll
                for (int p = 0; p < NP; ++p) {
                    double tr_ = 0.0, tz_ = 0.0;
#pragma unroll
                    for (int j = 0; j < NQ; ++j) {
                        if (p < np_ && in[j] && !c.nflag[p * 256 + sl[j]]) {
                            const double dz = pz[p] - zq[j];
                            double er, ez;
                            ring_field_far<false, false>(pr[p], pinv[p], dz, rq[j], er, ez);
                            tr_ = fma(wq[j], er, tr_);
                            tz_ = fma(wq[j], ez, tz_);
                            ++far_evals;
                        }
                    }
                    ar[p] += tr_;
                    az[p] += tz_;
                }
                }
            }
        }
        __syncthreads();
        if (tid == 0 && t + 2 < n_tiles) issue(t + 2, buf);
    }
    // fixed-order block reduction of the round's accumulators
    round_reduce<NP, MIX>(c, r0, np_, ar, az, fr, fz, kr, kz, sa);
}

// Recurrence constants of the Legendre polynomials, P_(n+1) = a_n u P_n - b_n P_(n-1).
static __device__ __constant__ double kLegA[64] = {
#define SPT_LA(n) (2.0 * (n) + 1.0) / ((n) + 1.0)
    SPT_LA(0), SPT_LA(1), SPT_LA(2), SPT_LA(3), SPT_LA(4), SPT_LA(5), SPT_LA(6), SPT_LA(7), SPT_LA(8), SPT_LA(9),
    SPT_LA(10), SPT_LA(11), SPT_LA(12), SPT_LA(13), SPT_LA(14), SPT_LA(15), SPT_LA(16), SPT_LA(17), SPT_LA(18),
    SPT_LA(19), SPT_LA(20), SPT_LA(21), SPT_LA(22), SPT_LA(23), SPT_LA(24), SPT_LA(25), SPT_LA(26), SPT_LA(27),
    SPT_LA(28), SPT_LA(29), SPT_LA(30), SPT_LA(31), SPT_LA(32), SPT_LA(33), SPT_LA(34), SPT_LA(35), SPT_LA(36),
    SPT_LA(37), SPT_LA(38), SPT_LA(39), SPT_LA(40), SPT_LA(41), SPT_LA(42), SPT_LA(43), SPT_LA(44), SPT_LA(45),
    SPT_LA(46), SPT_LA(47), SPT_LA(48), SPT_LA(49), SPT_LA(50), SPT_LA(51), SPT_LA(52), SPT_LA(53), SPT_LA(54),
    SPT_LA(55), SPT_LA(56), SPT_LA(57), SPT_LA(58), SPT_LA(59), SPT_LA(60), SPT_LA(61), SPT_LA(62), SPT_LA(63)};
#undef SPT_LA
static __device__ __constant__ double kLegB[64] = {
#define SPT_LB(n) (n) / ((n) + 1.0)
    SPT_LB(0), SPT_LB(1), SPT_LB(2), SPT_LB(3), SPT_LB(4), SPT_LB(5), SPT_LB(6), SPT_LB(7), SPT_LB(8), SPT_LB(9),
    SPT_LB(10), SPT_LB(11), SPT_LB(12), SPT_LB(13), SPT_LB(14), SPT_LB(15), SPT_LB(16), SPT_LB(17), SPT_LB(18),
    SPT_LB(19), SPT_LB(20), SPT_LB(21), SPT_LB(22), SPT_LB(23), SPT_LB(24), SPT_LB(25), SPT_LB(26), SPT_LB(27),
    SPT_LB(28), SPT_LB(29), SPT_LB(30), SPT_LB(31), SPT_LB(32), SPT_LB(33), SPT_LB(34), SPT_LB(35), SPT_LB(36),
    SPT_LB(37), SPT_LB(38), SPT_LB(39), SPT_LB(40), SPT_LB(41), SPT_LB(42), SPT_LB(43), SPT_LB(44), SPT_LB(45),
    SPT_LB(46), SPT_LB(47), SPT_LB(48), SPT_LB(49), SPT_LB(50), SPT_LB(51), SPT_LB(52), SPT_LB(53), SPT_LB(54),
    SPT_LB(55), SPT_LB(56), SPT_LB(57), SPT_LB(58), SPT_LB(59), SPT_LB(60), SPT_LB(61), SPT_LB(62), SPT_LB(63)};
#undef SPT_LB

// Field (E_rho, E_z) at (rho, z) of a cluster from its record (z_c, r_max,
// M_0 .. M_(nt-1)): with r, u = cos(theta), s = sin(theta) about (0, z_c) and
// x = r_max / r, the potential (1/4 pi) sum_n M_n x^n P_n(u) / r gives
// E_r = (1/4 pi r^2) sum (n+1) M_n x^n P_n(u), E_theta = (s/4 pi r^2) sum
// M_n x^n P_n'(u), turned into (rho, z) components.  P_n' by
// P'_(n+1) = P'_(n-1) + (2n+1) P_n.
__device__ __forceinline__ void cluster_field(const double* rec, int nt, double rho, double z, double& er,
                                              double& ez) {
    const double dz = z - __ldg(rec);
    const double r2 = rho * rho + dz * dz;
    const double ir = rsqrt(r2);
    const double u = dz * ir, s = rho * ir, x = __ldg(rec + 1) * ir;
    double p0 = 1.0, p1 = u, d0 = 0.0, d1 = 1.0;
    double A = __ldg(rec + 2), B = 0.0;
    double xn = x, n1 = 2.0;  // n + 1, as a double: conversions are slower than the sum
    auto term = [&](int n, double moment) {
        const double m = moment * xn;
        A = fma(n1 * m, p1, A);
        B = fma(m, d1, B);
        const double p2 = fma(kLegA[n] * u, p1, -kLegB[n] * p0);
        const double d2 = fma(fma(2.0, n1, -1.0), p1, d0);
        n1 += 1.0;
        p0 = p1;
        p1 = p2;
        d0 = d1;
        d1 = d2;
        xn *= x;
    };
    // moments loaded four terms ahead of the recurrence that consumes them
    int n = 1;
    for (; n + 3 < nt; n += 4) {
        const double m0 = __ldg(rec + 2 + n), m1 = __ldg(rec + 3 + n), m2 = __ldg(rec + 4 + n),
                     m3 = __ldg(rec + 5 + n);
        term(n, m0);
        term(n + 1, m1);
        term(n + 2, m2);
        term(n + 3, m3);
    }
    for (; n < nt; ++n) term(n, __ldg(rec + 2 + n));
    const double sc = ir * ir * 0.07957747154594767;  // 1 / (4 pi r^2)
    const double e_r = A * sc, e_t = s * B * sc;
    er = e_r * s + e_t * u;
    ez = e_r * u - e_t * s;
}

// ---------------------------------------------------------------------------
// Field map (SptBem.reserved, spt_map.cu): square cells of a quadtree over the
// (rho, z) half plane, each holding (E_rho, E_z) as polynomials of degree
// SPT_MAP_N - 1 in either coordinate (cells on the axis in rho^2, and E_rho
// there as rho times a polynomial: E_rho is odd in rho, and a polynomial that
// only comes close to 0 on the axis is off by 1e-14 of E_z there, which is 7 %
// of E_rho 1e-9 of the surface's distance from the axis).  The field is analytic away from the
// surface, so cells a few half-widths from it converge to rounding; cells
// within SPT_MAP_BAND panel lengths of a panel hold none, and points there
// take the direct sum.
__device__ __forceinline__ const double* field_map(const SptBem& b) {
    return ((unsigned)b.reserved >> 16) == SPT_MAP_TAG ? b.clusters + (size_t)(b.reserved & 0xffff) * SPT_MAP_UNIT
                                                       : nullptr;
}

// Cell that holds (rho, z), or -1: one table for the first SPT_MAP_ROOT_BITS
// quadtree levels and tables of SPT_MAP_BITS levels below it, so a point's cell
// is three or four dependent loads away (with three levels a table throughout it
// was seven, at L2's latency most of a stage); one lane per point.
__device__ __forceinline__ int map_find(const double* map, double rho, double z) {
    const double u = rho * __ldg(map), v = (z - __ldg(map + 1)) * __ldg(map);
    if (!(u < 1.0 && v >= 0.0 && v < 1.0)) return -1;
    const unsigned iu = (unsigned)(u * 1073741824.0), iv = (unsigned)(v * 1073741824.0);
    const int* tab = reinterpret_cast<const int*>(map + SPT_MAP_HEADER);
    constexpr int B = SPT_MAP_BITS, R = SPT_MAP_ROOT_BITS;
    int sh = 30 - R;
    int e = __ldg(tab + ((iv >> sh) << R) + (iu >> sh));
    tab += 1 << (2 * R);
    while (e < -1 && sh >= B) {
        sh -= B;
        e = __ldg(tab + ((size_t)(-2 - e) << (2 * B)) + (((iv >> sh) & ((1 << B) - 1)) << B) + ((iu >> sh) & ((1 << B) - 1)));
    }
    return e < -1 ? -1 : e;
}

// (E_rho, E_z) at (rho, z) of cell `leaf`, by one warp; every lane returns
// both.  Lane i of each half takes row i (power i of the rho coordinate, lower
// half E_rho, upper half E_z) as a polynomial in z: the row's coefficients
// are one coalesced line per power, the Horner chains of all rows run side by
// side, and four shuffles add the rows.  Bound by the record's 2.3 KB through
// L1/L2: a million points off the benchmark tip take 0.33 ms, their direct
// sums (the closest-segment, near and far phases, ~6300 warp instructions a
// point) 20 ms.  Twelve orders: eight need cells a third as wide for 1e-14,
// sixteen twice the bytes a point.
__device__ __forceinline__ void map_field(const double* map, int leaf, double rho, double z, double& er, double& ez) {
    const double* rec = map + (size_t)__ldg(map + 2) + (size_t)leaf * SPT_MAP_REC;
    const int lane = threadIdx.x & 31, i = lane & 15;
    const bool on = i < SPT_MAP_N;
    const double* a = rec + 8 + (lane >> 4) * SPT_MAP_N + (on ? i : 0);
    double c[SPT_MAP_N];
#pragma unroll
    for (int j = 0; j < SPT_MAP_N; ++j) c[j] = __ldg(a + j * 2 * SPT_MAP_N);
    // a cell on the axis (its centre one half-width off): E_rho = u A, u = rho / half-width, and A, E_z even in rho
    const double rc = __ldg(rec), iw = __ldg(rec + 2), u = rho * iw;
    const bool axis = rc * iw < 1.5;
    const double x = axis ? fma(0.5 * u, u, -1.0) : (rho - rc) * iw, y = (z - __ldg(rec + 1)) * iw;
    const double x2 = x * x, x4 = x2 * x2, y2 = y * y;
    double p = (i & 1) ? x : 1.0;
    if (i & 2) p *= x2;
    if (i & 4) p *= x4;
    if (i & 8) p *= x4 * x4;
    double e = c[SPT_MAP_N - 2], o = c[SPT_MAP_N - 1];
#pragma unroll
    for (int j = SPT_MAP_N - 4; j >= 0; j -= 2) {
        e = fma(e, y2, c[j]);
        o = fma(o, y2, c[j + 1]);
    }
    double r = on ? fma(o, y, e) * p : 0.0;
#pragma unroll
    for (int s = 8; s > 0; s >>= 1) r += __shfl_xor_sync(0xffffffffu, r, s);
    er = __shfl_sync(0xffffffffu, r, 0);
    ez = __shfl_sync(0xffffffffu, r, 16);
    if (axis) er *= u;
}

// Perturbation field of this lane's point (rho, z) where leaf >= 0, the warp
// taking its lanes' points one after another.
__device__ __forceinline__ void map_field_lanes(const double* map, int leaf, double rho, double z, double& er,
                                                double& ez) {
    const int lane = threadIdx.x & 31;
    for (unsigned m = __ballot_sync(0xffffffffu, leaf >= 0); m; m &= m - 1) {
        const int j = __ffs(m) - 1;
        double fr, fz;
        map_field(map, __shfl_sync(0xffffffffu, leaf, j), __shfl_sync(0xffffffffu, rho, j),
                  __shfl_sync(0xffffffffu, z, j), fr, fz);
        if (lane == j) {
            er = fr;
            ez = fz;
        }
    }
}

// E_rho at (x, y) turned into (E_x, E_y)
__device__ __forceinline__ void rotate_rho(double x, double y, double rho, double e_rho, double& ex, double& ey) {
    ex = ey = 0.0;
    if (rho != 0.0) {
        ex = e_rho * (x / rho);
        ey = e_rho * (y / rho);
    }
}

// Gauss-8 nodes of each whole panel (rho, z, w rows), kept with the field map:
// panels PANEL8_FROM to PANEL8_TO x ratio4 lengths away.  At two lengths its
// error (8.1^-16) is that of the reference's 32 sub-panel nodes, at a quarter
// of the ring evaluations; up to twice ratio4 it replaces the whole-panel
// Gauss-4, whose error at ratio4 = 8 is 32^-8 = 1e-12, and Gauss-4 serves to
// twice ratio2 (Gauss-2 at 300 lengths was the rule's largest error, 2e-12 near
// the corner of the 3000-panel well; 2e-13 at 600).
constexpr double kPanel8From = 2.0, kPanel8To = 2.0;
__device__ __forceinline__ const double* panel8(const SptBem& b) {
    const double* map = field_map(b);
    return map ? map + (size_t)__ldg(map + 3) : nullptr;
}

// Sums of one point's direct evaluation.  Its ring evaluations come in rounds
// of one per lane, and each round adds to one of four slots of its lane: near
// quadrature and cluster expansions by their number, round % 4, the far nodes
// of a chunk by quarters.  So one warp can take all rounds, or 2 or 4 warps a
// share of the slots each, and the result -- the slots added per lane, then the
// lanes -- is the same to the bit.
struct PointSums {
    double r[4], z[4];
    int round, share, shares;  // next round's number; this warp's share of 1, 2 or 4
    __device__ PointSums(int share_, int shares_) : round(0), share(share_), shares(shares_) {
#pragma unroll
        for (int k = 0; k < 4; ++k) r[k] = z[k] = 0.0;
    }
    // whether the next round is this warp's (alike in every lane)
    __device__ __forceinline__ bool mine() const { return (round & (shares - 1)) == share; }
    __device__ __forceinline__ void add(double er, double ez) {
        const int k = round & 3;  // a branch the whole warp takes
        if (k == 0) { r[0] += er; z[0] += ez; }
        else if (k == 1) { r[1] += er; z[1] += ez; }
        else if (k == 2) { r[2] += er; z[2] += ez; }
        else { r[3] += er; z[3] += ez; }
    }
    // the far rounds' quarters: slot 0 is the current quarter's, and four turns bring every slot home
    __device__ __forceinline__ void turn(double er, double ez) {
        const double r0 = r[0] + er, z0 = z[0] + ez;
        r[0] = r[1]; r[1] = r[2]; r[2] = r[3]; r[3] = r0;
        z[0] = z[1]; z[1] = z[2]; z[2] = z[3]; z[3] = z0;
    }
    // the whole sums, in lane 0
    __device__ __forceinline__ void total(double& er, double& ez) const {
        er = warp_sum((r[0] + r[1]) + (r[2] + r[3]));
        ez = warp_sum((z[0] + z[1]) + (z[2] + z[3]));
    }
};

// Counters of a warp's direct evaluations, and their sum into the CTA's.
struct PointCounts {
    unsigned long long n_near = 0, n_ring_near = 0, far_evals = 0, cl_evals = 0;
};
__device__ __forceinline__ void count_points(Ctx& c, const PointCounts& n) {
    count_add(c, SPT_CNT_NEAR_PAIRS, n.n_near);
    count_add(c, SPT_CNT_RING_NEAR, n.n_ring_near);
    count_add(c, SPT_CNT_RING_FAR, n.far_evals);
    count_add(c, SPT_CNT_CLUSTER_EVALS, n.cl_evals);
}

// Adaptive far sum (SPT_FAR_ADAPTIVE) at (re, ze), by one warp (nothing here
// waits on another warp).  Cluster expansions cover the runs of their clusters.
// The other runs are classified 32 at a time by their lower-bound distance:
// flagged runs at least ratio_run arclengths away take the 8-point rule over
// the whole run (list R3), runs whose every segment is at least ratio2 lengths
// away Gauss-2 on each segment (R2), the rest (M) are classified segment by
// segment -- the reference nodes (near segments masked), Gauss-8 where the
// panel nodes are given, Gauss-4, or Gauss-2 (lists L0, L8, L1, L2 in the
// warp's own shared scratch).  The flattened node list is then evaluated by the
// lanes, nodes read through L1/L2.  Without run bounds every run is in M.
//
// MIX false: float64, one ring evaluation in flight per lane (every copy in
// flight is an inlined copy of the ring kernel, and the trace kernels are bound
// by instruction fetch), into S.  MIX true: float32 Kahan sums, four in flight;
// mr, mz, mabs return them and the sum of |terms| in lane 0.
template <bool MIX>
__device__ void far_adaptive_warp(Ctx& c, double re, double ze, PointSums& S, PointCounts& cnt, double& mr, double& mz,
                                  double& mabs) {
    constexpr int NQ = MIX ? 4 : 1;
    const SptBem& b = c.bem;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nseg = b.n_seg, nps = b.nodes_per_seg;
    int* scratch = reinterpret_cast<int*>(c.tiles) + warp * kWarpScratchInts;
    unsigned char* lists = reinterpret_cast<unsigned char*>(scratch);  // L0 | L1 | L2 | L8, kWarpChunk each
    unsigned char* mask = lists + 4 * kWarpChunk;                      // near flags of L0
    int* R2 = scratch + 5 * kWarpChunk / 4;
    int* R3 = R2 + kWarpRuns;
    int* M = R3 + kWarpRuns;
    int* Mcls = M + kWarpRuns;
    unsigned* covered = reinterpret_cast<unsigned*>(Mcls + kWarpRuns);  // runs summed by cluster expansions
    const double inv = re > 0.0 ? 1.0 / re : 0.0;
    double cr_ = 0.0, cz_ = 0.0;                                // mixed form: the float64 expansions
    float fr = 0.f, fz = 0.f, kr = 0.f, kz = 0.f, sa = 0.f;     // mixed form: Kahan sums, sum of |float32 terms|
    const float ref = (float)re, invf = (float)inv;
    const double* cr = b.coarse;
    const double* cz = b.coarse + b.coarse_stride;
    const double* cw = b.coarse + 2 * b.coarse_stride;
    const bool run_rule = b.blk && b.run_nodes && b.ratio_run > 0.0;
    const unsigned lt = (1u << lane) - 1u;
    // Cluster expansions: lane = run; the run is covered by its highest
    // ancestor cluster that is at least kappa radii away, and the lane of the
    // cluster's first run lists that cluster.
    const int n_run = (nseg + SPT_BLOCK_SEGS - 1) / SPT_BLOCK_SEGS;
    const bool use_cl = b.blk && b.clusters && b.cluster_kappa > 0.0 && n_run <= SPT_MAX_CLUSTER_RUNS;
    if (use_cl) {
        const int nt = b.cluster_terms, rec_len = nt + 2;
        // the covering clusters' heads, listed first (the segment lists are free
        // until the chunk loop) and then expanded in one lane-parallel pass
        int* const heads = scratch;
        static_assert(SPT_MAX_CLUSTER_RUNS <= kWarpChunk, "the heads fit the segment lists");
        int n_heads = 0;
        for (int qb = 0; qb < n_run; qb += 32) {
            const int q = qb + lane;
            int lv = -1, idx = 0;
            if (q < n_run) {
                int off = 0;
                for (int l = 0; l < b.cluster_levels; ++l) {
                    const int i = off + (q >> l);
                    const double* rec = b.clusters + (size_t)i * rec_len;
                    const double dz = ze - __ldg(rec);
                    if (re * re + dz * dz >= b.cluster_kappa * b.cluster_kappa * __ldg(rec + 1) * __ldg(rec + 1)) {
                        lv = l;
                        idx = i;
                    }
                    off += (n_run + (1 << l) - 1) >> l;
                }
            }
            const unsigned cov = __ballot_sync(0xffffffffu, lv >= 0);
            if (lane == 0) covered[qb >> 5] = cov;
            const bool head = lv >= 0 && (q & ((1 << lv) - 1)) == 0;
            const unsigned hm = __ballot_sync(0xffffffffu, head);
            if (head) heads[n_heads + __popc(hm & lt)] = idx;
            n_heads += __popc(hm);
        }
        __syncwarp();
        for (int h0 = 0; h0 < n_heads; h0 += 32, ++S.round) {
            if (!S.mine()) continue;
            double er = 0.0, ez = 0.0;
            if (h0 + lane < n_heads) {
                cluster_field(b.clusters + (size_t)heads[h0 + lane] * rec_len, nt, re, ze, er, ez);
                ++cnt.cl_evals;
            }
            if (MIX) {
                cr_ += er;
                cz_ += ez;
            } else {
                S.add(er, ez);
            }
        }
        __syncwarp();
    }
    // floor(q / nps) = umulhi(q, nps_inv) for q below kWarpChunk nps <= 65536
    const unsigned nps_inv = 0xffffffffu / (unsigned)nps + 1u;
    const double* p8 = panel8(b);
    const double* p8r = p8;
    const double* p8z = p8 + 8 * (size_t)nseg;
    const double* p8w = p8 + 16 * (size_t)nseg;
    // the segment tests read ratio4 as the distance from which whole-panel Gauss-4 serves
    const double r4 = b.ratio4, r4s = p8 ? kPanel8To * r4 : r4, r2 = p8 ? kPanel8To * b.ratio2 : b.ratio2;
    for (int q0 = 0; q0 < n_run; q0 += kWarpRuns) {
        const int q = q0 + lane;
        int cls = -1;  // 3 run rule, 2 Gauss-2 on every segment, 1 no segment below ratio4, 0 full test
        if (q < n_run && !(use_cl && ((covered[q >> 5] >> (q & 31)) & 1u))) {
            cls = 0;
            if (b.blk) {
                const double lb = blk_lower(b, q, re, ze);
                const double lm = blk_lmax(b, q);
                if (run_rule && __ldg(b.blk + 5 * b.blk_stride + q) != 0.0 &&
                    lb >= b.ratio_run * __ldg(b.blk + 4 * b.blk_stride + q))
                    cls = 3;
                else if (lb >= r2 * lm) cls = 2;
                else if (lb >= r4s * lm) cls = 1;
            }
        }
        const unsigned b3 = __ballot_sync(0xffffffffu, cls == 3);
        const unsigned b2 = __ballot_sync(0xffffffffu, cls == 2);
        const unsigned bm = __ballot_sync(0xffffffffu, cls == 0 || cls == 1);
        if (cls == 3) R3[__popc(b3 & lt)] = q;
        if (cls == 2) R2[__popc(b2 & lt)] = q;
        if (cls == 0 || cls == 1) { M[__popc(bm & lt)] = q; Mcls[__popc(bm & lt)] = cls; }
        int nR2 = __popc(b2), nR3 = __popc(b3);
        const int nm = __popc(bm);
        __syncwarp();
        // the M runs, as many at a time as the lists hold; the R2 and R3 runs with the first
        for (int m0 = 0; m0 < nm || m0 == 0; m0 += kWarpChunk / SPT_BLOCK_SEGS, nR2 = nR3 = 0) {
        // segment classification of the M runs, one run at a time (lane = segment)
        int n0 = 0, n1 = 0, n2 = 0, n8 = 0;
        for (int mi = m0; mi < min(nm, m0 + kWarpChunk / SPT_BLOCK_SEGS); ++mi) {
            const int sg = M[mi] * SPT_BLOCK_SEGS + lane;
            const unsigned char at = (unsigned char)((mi - m0) * SPT_BLOCK_SEGS + lane);
            int lvl = 3;
            bool m = false;
            if (sg < nseg) {
                const int mc = Mcls[mi];
                const double L = segf(b, 4, sg);
                double proj, dmin;
                m = seg_near<true>(b, sg, re, ze, proj, dmin) && mc == 0;
                if (mc == 1) lvl = dmin < r2 * L ? 1 : 2;
                else if (p8 && dmin >= kPanel8From * L) lvl = dmin < r4s * L ? 4 : (dmin < r2 * L ? 1 : 2);
                else lvl = dmin < r4 * L ? 0 : (dmin < r2 * L ? 1 : 2);
            }
            const unsigned v0 = __ballot_sync(0xffffffffu, lvl == 0);
            const unsigned v1 = __ballot_sync(0xffffffffu, lvl == 1);
            const unsigned v2 = __ballot_sync(0xffffffffu, lvl == 2);
            const unsigned v8 = __ballot_sync(0xffffffffu, lvl == 4);
            if (lvl == 0) {
                const int pos = n0 + __popc(v0 & lt);
                lists[pos] = at;
                mask[pos] = (unsigned char)m;
            } else if (lvl == 1) {
                lists[kWarpChunk + n1 + __popc(v1 & lt)] = at;
            } else if (lvl == 2) {
                lists[2 * kWarpChunk + n2 + __popc(v2 & lt)] = at;
            } else if (lvl == 4) {
                lists[3 * kWarpChunk + n8 + __popc(v8 & lt)] = at;
            }
            n0 += __popc(v0);
            n1 += __popc(v1);
            n2 += __popc(v2);
            n8 += __popc(v8);
        }
        __syncwarp();
        auto listed = [&](int list, int k) {  // segment k of a list
            const int v = lists[list * kWarpChunk + k];
            return M[m0 + v / SPT_BLOCK_SEGS] * SPT_BLOCK_SEGS + v % SPT_BLOCK_SEGS;
        };
        const int e0 = n0 * nps, e8 = e0 + 8 * n8, e1 = e8 + 4 * n1, e2 = e1 + 2 * n2;
        const int e3 = e2 + 2 * SPT_BLOCK_SEGS * nR2, e4 = e3 + SPT_RUN_NODES * nR3;
        const int rounds = (e4 + 32 * NQ - 1) / (32 * NQ);
#pragma unroll 1
        for (int quarter = 0; quarter < (MIX ? 1 : 4); ++quarter) {
        double tr_ = 0.0, tz_ = 0.0;
        const bool own = MIX || (quarter & (S.shares - 1)) == S.share;
        const int first = MIX ? 0 : rounds * quarter / 4, last = MIX ? rounds : (own ? rounds * (quarter + 1) / 4 : first);
#pragma unroll 1
        for (int rd = first; rd < last; ++rd) {
            const int q0i = rd * 32 * NQ + lane;
            double rq[NQ], zq[NQ], wq[NQ];
            bool in[NQ];
#pragma unroll
            for (int j = 0; j < NQ; ++j) {
                const int qq = q0i + j * 32;
                in[j] = qq < e4;
                size_t src = 0;
                const double *tr = cr, *tz = cz, *tw = cw;
                if (!in[j]) {
                    // padding lane: any valid node, not accumulated
                } else if (qq < e0) {
                    const int li = (int)__umulhi((unsigned)qq, nps_inv);
                    src = (size_t)listed(0, li) * nps + (qq - li * nps);
                    tr = b.node;
                    tz = b.node + b.node_stride;
                    tw = b.node + 2 * b.node_stride;
                    in[j] = !mask[li];  // near segments are the near quadrature's
                } else if (qq < e8) {
                    const int i = qq - e0;
                    src = (size_t)listed(3, i >> 3) * 8 + (i & 7);
                    tr = p8r;
                    tz = p8z;
                    tw = p8w;
                } else if (qq < e1) {
                    const int i = qq - e8;
                    src = (size_t)listed(1, i >> 2) * 6 + (i & 3);
                } else if (qq < e2) {
                    const int i = qq - e1;
                    src = (size_t)listed(2, i >> 1) * 6 + 4 + (i & 1);
                } else if (qq < e3) {
                    const int i = qq - e2;
                    const int sgi = R2[i / (2 * SPT_BLOCK_SEGS)] * SPT_BLOCK_SEGS + ((i & (2 * SPT_BLOCK_SEGS - 1)) >> 1);
                    if (sgi < nseg) src = (size_t)sgi * 6 + 4 + (i & 1);
                    else in[j] = false;  // past the last segment of a short final run
                } else {
                    const int i = qq - e3;
                    src = (size_t)R3[i / SPT_RUN_NODES] * SPT_RUN_NODES + (i % SPT_RUN_NODES);
                    tr = b.run_nodes;
                    tz = b.run_nodes + b.run_stride;
                    tw = b.run_nodes + 2 * b.run_stride;
                }
                rq[j] = __ldg(tr + src);
                zq[j] = __ldg(tz + src);
                wq[j] = __ldg(tw + src);
            }
            if constexpr (MIX) {
#pragma unroll
                for (int j = 0; j < NQ; ++j) {
                    if (!in[j]) continue;
                    const double dz = ze - zq[j];
                    float er, ez;
                    if (ring_far_f(ref, invf, (float)(re - rq[j]), (float)(re + rq[j]), (float)dz, (float)rq[j], er, ez)) {
                        const float w = (float)wq[j];
                        kahan_add(fr, kr, w * er);
                        kahan_add(fz, kz, w * ez);
                        sa += fabsf(w * er) + fabsf(w * ez);
                    } else {
                        // close to the ring: the term in float64, summed like the others
                        double e64r, e64z;
                        ring_field_far_cold(re, inv, dz, rq[j], e64r, e64z);
                        const float ter = (float)(wq[j] * e64r), tez = (float)(wq[j] * e64z);
                        kahan_add(fr, kr, ter);
                        kahan_add(fz, kz, tez);
                        sa += fabsf(ter) + fabsf(tez);
                    }
                    ++cnt.far_evals;
                }
            } else {
                double er = 0.0, ez = 0.0;
                if (in[0]) {
                    ring_field_far<false, true>(re, inv, ze - zq[0], rq[0], er, ez);
                    ++cnt.far_evals;
                }
                tr_ = fma(wq[0], er, tr_);
                tz_ = fma(wq[0], ez, tz_);
            }
        }
        if (!MIX) S.turn(tr_, tz_);
        }
        __syncwarp();  // the lists are rewritten by the next chunk
        }
    }
    if (MIX) {
        mr = warp_sum(cr_ + ((double)fr - (double)kr));
        mz = warp_sum(cz_ + ((double)fz - (double)kz));
        mabs = warp_sum((double)sa);
    }
}

// ---------------------------------------------------------------------------
// BEM field of a list of points, in phases.  Records live in c.bpt (8 doubles
// each: x, y, z, rho_e, z_e, then results); every phase is called by all
// threads of the CTA.

// A: closest segment and on-surface offset of records [0, n).  With `frame`,
// also the closest segment, its parameter t and the distance, for the
// surrogate's inputs.
// One warp, record k.
__device__ __forceinline__ void closest_point(Ctx& c, double* P, int k, bool frame) {
    const SptBem& b = c.bem;
    const int lane = threadIdx.x & 31;
    // record k: [0]x [1]y [2]z [3]rho_e [4]z_e [5]ax [6]ay [7]near_r ; near_z in ntmp
    const int nseg = b.n_seg;
    {
        const double x = P[8 * k + 0], y = P[8 * k + 1], z = P[8 * k + 2];
        const double rho = hypot(x, y);
        double best = INFINITY;
        int bs = 0x7fffffff;
        if (b.blk) {
            const int nblk = (nseg + SPT_BLOCK_SEGS - 1) / SPT_BLOCK_SEGS;
            // The on-surface offset below needs a distance under 1e-9 of the
            // closest segment's length.  Where no segment is within 1e-8 of its
            // length (runs out of reach by their rigorous bounds, the others'
            // segments one by one), the closest segment plays no further part,
            // and the evaluation point is the point itself -- the offset path's
            // rho + 0 and z + 0 bit for bit (z = 0 excepted: there the sign of
            // the zero would follow the normal).
            if (!frame && z != 0.0) {
                bool hit = false;
                for (int q0 = 0; q0 < nblk; q0 += 32) {
                    const bool cand = q0 + lane < nblk &&
                                      !(blk_lower(b, q0 + lane, rho, z) > 1e-8 * blk_lmax(b, q0 + lane));
                    for (unsigned cm = __ballot_sync(0xffffffffu, cand); cm; cm &= cm - 1) {
                        const int s = (q0 + __ffs(cm) - 1) * SPT_BLOCK_SEGS + lane;
                        double proj, dist;
                        if (s < nseg) {
                            seg_near<true>(b, s, rho, z, proj, dist);
                            hit |= !(dist > 1e-8 * segf(b, 4, s));
                        }
                    }
                }
                if (!__any_sync(0xffffffffu, hit)) {
                    if (lane == 0) {
                        P[8 * k + 3] = rho;
                        P[8 * k + 4] = z;
                    }
                    return;
                }
            }
            // the run with the smallest lower bound gives an upper bound of the
            // minimum; only runs whose lower bound does not exceed it are scanned
            // (each lane still takes its segments in increasing order)
            double lbm = INFINITY;
            int qm = 0;
            for (int q = lane; q < nblk; q += 32) {
                const double lb = blk_lower(b, q, rho, z);
                if (lb < lbm) { lbm = lb; qm = q; }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const double ol = __shfl_xor_sync(0xffffffffu, lbm, o);
                const int oq = __shfl_xor_sync(0xffffffffu, qm, o);
                if (ol < lbm || (ol == lbm && oq < qm)) { lbm = ol; qm = oq; }
            }
            double ub = INFINITY;
            if (qm * SPT_BLOCK_SEGS + lane < nseg) ub = seg_dist2(b, qm * SPT_BLOCK_SEGS + lane, rho, z);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) ub = fmin(ub, __shfl_xor_sync(0xffffffffu, ub, o));
            const double ubd = sqrt(ub);
            for (int q0 = 0; q0 < nblk; q0 += 32) {
                const bool cand = q0 + lane < nblk && !(blk_lower(b, q0 + lane, rho, z) > ubd);
                unsigned cm = __ballot_sync(0xffffffffu, cand);
                while (cm) {
                    const int j = __ffs(cm) - 1;
                    cm &= cm - 1;
                    const int s = (q0 + j) * SPT_BLOCK_SEGS + lane;
                    if (s < nseg) {
                        const double d2 = seg_dist2(b, s, rho, z);
                        if (d2 < best) { best = d2; bs = s; }
                    }
                }
            }
        } else {
            for (int s = lane; s < nseg; s += 32) {
                const double d2 = seg_dist2(b, s, rho, z);
                if (d2 < best) { best = d2; bs = s; }
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int os = __shfl_xor_sync(0xffffffffu, bs, o);
            if (ob < best || (ob == best && os < bs)) { best = ob; bs = os; }
        }
        if (lane == 0) {
            if (bs >= nseg) bs = 0;  // every distance was NaN: the reference keeps index 0
            const double Ls = segf(b, 4, bs);
            const double thr = __dmul_rn(1e-9, Ls);
            const double off = (best < __dmul_rn(thr, thr)) ? __dmul_rn(1e-4, Ls) : 0.0;
            double re = __dadd_rn(rho, __dmul_rn(off, segf(b, 7, bs)));
            if (rho == 0.0) re = 0.0;
            P[8 * k + 3] = re;
            P[8 * k + 4] = __dadd_rn(z, __dmul_rn(off, segf(b, 8, bs)));
            if (frame) {
                const double p0x = segf(b, 0, bs), p0y = segf(b, 1, bs), ax = segf(b, 2, bs), ay = segf(b, 3, bs);
                double tt = ((rho - p0x) * ax + (z - p0y) * ay) / (ax * ax + ay * ay);
                c.sseg[k] = bs;
                c.st[k] = fmin(fmax(tt, 0.0), 1.0);
                c.sd[k] = sqrt(best);
            }
        }
    }
}

static __device__ void bem_closest(Ctx& c, int n, bool frame) {
    // one warp per point
    for (int k = threadIdx.x >> 5; k < n; k += c.nw) closest_point(c, c.bpt, k, frame);
    __syncthreads();
}


// B at (re, ze), by one warp: the near-segment sinh quadrature
// (bem/axisymmetric.py:566-600) into S.  FAST (the adaptive rule): in rounds;
// else every node into slot 0, in the reference rule's order.
template <bool FAST>
__device__ __forceinline__ void near_sums(Ctx& c, double re, double ze, PointSums& S, PointCounts& n) {
    const SptBem& b = c.bem;
    const int lane = threadIdx.x & 31;
    const int nseg = b.n_seg;
    {
        const double inv = re > 0.0 ? 1.0 / re : 0.0;
        const int nblk = (nseg + SPT_BLOCK_SEGS - 1) / SPT_BLOCK_SEGS;
        for (int q0 = 0; q0 < nblk; q0 += 32) {
          // runs that may hold a near segment (every run without the bounds table)
          const bool cand = q0 + lane < nblk && !(b.blk && blk_lower(b, q0 + lane, re, ze) >= blk_lmax(b, q0 + lane));
          unsigned cm = __ballot_sync(0xffffffffu, cand);
          while (cm) {
            const int jq = __ffs(cm) - 1;
            cm &= cm - 1;
            const int s0 = (q0 + jq) * SPT_BLOCK_SEGS;
            const int s = s0 + lane;
            double proj = 0.0, dist = 0.0;
            const bool nr = (s < nseg) && seg_near<FAST>(b, s, re, ze, proj, dist);
            unsigned mask = __ballot_sync(0xffffffffu, nr);
            // the sinh map's limits and intervals, by every near segment's lane at once
            double lo = 0.0, hi = 0.0;
            if (nr) {
                const double Ls = segf(b, 4, s);
                dist = fmax(dist, 1e-15 * Ls);
                if constexpr (FAST) {  // the limits to 1e-16 absolute, as v is used
                    const double id = rcp_pos(dist), a = proj * id, e = (Ls - proj) * id;
                    lo = -log(a + sqrt_pos(fma(a, a, 1.0)));
                    hi = log(e + sqrt_pos(fma(e, e, 1.0)));
                } else {
                    lo = asinh(-proj / dist);
                    hi = asinh((Ls - proj) / dist);
                }
            }
            while (mask) {
                const int j = __ffs(mask) - 1;
                mask &= mask - 1;
                const int sg = s0 + j;
                const double sp = __shfl_sync(0xffffffffu, proj, j), d = __shfl_sync(0xffffffffu, dist, j);
                const double v0 = __shfl_sync(0xffffffffu, lo, j), span = __shfl_sync(0xffffffffu, hi, j) - v0;
                const int cnt = max(1, (int)ceil(span / 0.5));
                const double width = FAST ? span * rcp_pos((double)cnt) : span / cnt, half = 0.5 * width;
                
                const double p0r = segf(b, 0, sg), p0z = segf(b, 1, sg), ur = segf(b, 5, sg), uz = segf(b, 6, sg);
                const double sg0 = segf(b, 9, sg), dsg = FAST ? (segf(b, 10, sg) - sg0) * rcp_pos(segf(b, 4, sg)) : 0.0;
                for (int q0 = 0; q0 < cnt * 8; q0 += 32, ++S.round) {
                    const int qn = q0 + lane;
                    if ((FAST && !S.mine()) || qn >= cnt * 8) continue;
                    const int iv = qn >> 3, gi = qn & 7;
                    const double v = fma(iv + 0.5 * (b.gauss8_x[gi] + 1.0), width, v0);
                    double er, ez;
                    if constexpr (FAST) {
                        // sinh and cosh from one exponential (sinh to 1e-16 of d, and the node is at least d from
                        // the point)
                        const double ev = exp(v), em = rcp_pos(ev);
                        const double sl = fma(0.5 * d, ev - em, sp);
                        const double sr = fma(sl, ur, p0r), sz = fma(sl, uz, p0z);
                        const double w = fma(sl, dsg, sg0) * (2.0 * kPi * sr) * (0.5 * d * (ev + em)) * half * b.gauss8_w[gi];
                        ring_field_far<true, true>(re, inv, ze - sz, sr, er, ez);
                        S.add(w * er, w * ez);
                    } else {
                        // the reference's own operations: a node's place is rounded at ulp(rho), 1e-10 of its
                        // distance at a picometre, and a^2 - rho^2 + z^2 cancels (1e-12 of the field at 0.1 nm
                        // from a 2 um wall), so traces of ill-conditioned particles follow this rounding
                        const double sl = sp + d * sinh(v);
                        const double sr = p0r + sl * ur, sz = p0z + sl * uz;
                        const double dens = sg0 + (sl / segf(b, 4, sg)) * (segf(b, 10, sg) - sg0);
                        const double w = dens * (2.0 * kPi * sr) * d * cosh(v) * half * b.gauss8_w[gi];
                        ring_field(re, ze - sz, sr, er, ez);
                        S.r[0] += w * er;
                        S.z[0] += w * ez;
                    }
                }
                if (lane == 0 && S.share == 0) { n.n_near += 1; n.n_ring_near += (unsigned long long)cnt * 8; }
            }
          }
        }
    }
}

// The same for record k of the reference rule: lane 0 ends with near_r in slot
// 7 and near_z in ntmp[3k + 2].
__device__ __forceinline__ void near_point(Ctx& c, double* P, int k, PointCounts& n) {
    PointSums S(0, 1);
    near_sums<false>(c, P[8 * k + 3], P[8 * k + 4], S, n);
    const double r = warp_sum(S.r[0]), z = warp_sum(S.z[0]);
    if ((threadIdx.x & 31) == 0) {
        P[8 * k + 7] = r;
        c.ntmp[3 * k + 2] = z;
    }
}

// The adaptive rule's near and far sums at (re, ze) into S.  The mixed form
// sums in float32 first, and in float64 again when that sum is ill-conditioned
// (its sum of |terms| above kappa times the whole field); it takes all rounds,
// and its float64 sums are the float64 form's.
template <int FORM>
__device__ __forceinline__ void adaptive_sums(Ctx& c, double re, double ze, PointSums& S, PointCounts& n) {
    double mr, mz, mabs;
    near_sums<true>(c, re, ze, S, n);
    if constexpr (FORM == SPT_FORM_FP64) {
        far_adaptive_warp<false>(c, re, ze, S, n, mr, mz, mabs);
    } else {
        const int round = S.round;
        double nr, nz;
        S.total(nr, nz);
        far_adaptive_warp<true>(c, re, ze, S, n, mr, mz, mabs);
        const double er = nr + mr, tz = (nz + mz) + c.g.E_gun;
        bool redo = !(mabs <= c.kappa * sqrt(er * er + tz * tz));
        redo = __shfl_sync(0xffffffffu, redo, 0);
        if (redo) {
            if ((threadIdx.x & 31) == 0) atomicAdd(c.cnt + SPT_CNT_FP64_ROUNDS, 1ull);
            S.round = round;
            far_adaptive_warp<false>(c, re, ze, S, n, mr, mz, mabs);
        } else if ((threadIdx.x & 31) == 0) {
            S.r[0] += mr;
            S.z[0] += mz;
        }
    }
}

// Next record for this warp from the CTA's task counter (dynamic assignment:
// points near the surface cost many times more than distant ones).
__device__ __forceinline__ int next_task(int* counter) {
    int k = 0;
    if ((threadIdx.x & 31) == 0) k = atomicAdd(counter, 1);
    return __shfl_sync(0xffffffffu, k, 0);
}

// B + C: exact BEM field (E_rho, E_z into record slots 5, 6) of records [0, n)
// whose slots 3, 4 hold the evaluation point.  FORM: SPT_FORM_FP64 sums in
// float64; the other forms sum in float32 first and redo an ill-conditioned
// sum in float64.
template <int FORM, int FAR>
__device__ __forceinline__ void bem_sums(Ctx& c, int n, int* status_flag) {
    const SptBem& b = c.bem;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double* P = c.bpt;
    const int nseg = b.n_seg;
    const int nps = b.nodes_per_seg;
    if (n <= 0) return;
    // adaptive rule with a field map: the map gives the points its cells hold
    const double* const map = FAR == SPT_FAR_ADAPTIVE ? field_map(b) : nullptr;
    PointCounts cnt;
    bool ok = true;
    if constexpr (FAR == SPT_FAR_ADAPTIVE) {
        // B + C: one point per warp task, taken dynamically
        __shared__ int s_far_task;
        __syncthreads();
        if (tid == 0) s_far_task = c.nw;
        __syncthreads();
        for (int k = warp; k < n; k = next_task(&s_far_task)) {
            const double re = P[8 * k + 3], ze = P[8 * k + 4];
            const int leaf = map ? map_find(map, re, ze) : -1;
            double er, ez;
            if (leaf >= 0) {
                map_field(map, leaf, re, ze, er, ez);
                if (lane == 0) ++cnt.cl_evals;
            } else {
                PointSums S(0, 1);
                adaptive_sums<FORM>(c, re, ze, S, cnt);
                S.total(er, ez);
            }
            if (lane == 0) {
                P[8 * k + 5] = er;
                P[8 * k + 6] = ez;
            }
            __syncwarp();
        }
        __syncthreads();
        count_points(c, cnt);
    } else {
        // B: near-segment sinh quadrature (one warp per point)
        for (int k = warp; k < n; k += c.nw) near_point(c, P, k, cnt);
        count_points(c, cnt);
        __syncthreads();
        // C: far sum, rounds over TMA-staged node tiles shared by the whole CTA;
        // the round's point count selects how many nodes each thread keeps in flight
        unsigned long long far_evals = 0;
        const int tile_cap = c.L.tile_cap;
        const int segs_per_tile = min(tile_cap / nps, 256);
        const int n_tiles = (nseg + segs_per_tile - 1) / segs_per_tile;
        for (int r0 = 0; r0 < n; r0 += c.round_pts) {
            const int np_ = min(c.round_pts, n - r0);
            if constexpr (FORM == SPT_FORM_FP64) {
                if (np_ == 1) far_round<1, 8, false>(c, r0, np_, n_tiles, segs_per_tile, ok, far_evals);
                else if (np_ == 2) far_round<2, 4, false>(c, r0, np_, n_tiles, segs_per_tile, ok, far_evals);
                else far_round<4, 2, false>(c, r0, np_, n_tiles, segs_per_tile, ok, far_evals);
            } else {
                // mixed form (and the exact sums of the learned form): float32 first,
                // float64 again for a round whose float32 sums are ill-conditioned
                if (np_ == 1) far_round<1, 4, true>(c, r0, np_, n_tiles, segs_per_tile, ok, far_evals);
                else if (np_ == 2) far_round<2, 2, true>(c, r0, np_, n_tiles, segs_per_tile, ok, far_evals);
                else far_round<4, 1, true>(c, r0, np_, n_tiles, segs_per_tile, ok, far_evals);
                const bool redo = *c.redo != 0;
                // every thread has read the flag before the next round's float32 pass resets it
                __syncthreads();
                if (redo) {
                    if (tid == 0) atomicAdd(c.cnt + SPT_CNT_FP64_ROUNDS, 1ull);
                    // the tile shape the float64 form takes for this round size (same sums, bit for bit)
                    if (np_ == 1) far_round<1, 8, false>(c, r0, np_, n_tiles, segs_per_tile, ok, far_evals);
                    else if (np_ == 2) far_round<2, 4, false>(c, r0, np_, n_tiles, segs_per_tile, ok, far_evals);
                    else far_round<4, 2, false>(c, r0, np_, n_tiles, segs_per_tile, ok, far_evals);
                }
            }
        }
        count_add(c, SPT_CNT_RING_FAR, far_evals);
    }
    if (!ok && tid == 0) *status_flag = SPT_GROUP_TIMEOUT;
}

// D: rotate E_rho of records [0, n) into (x, y) (record slots 5, 6, 7 = ex, ey, ez)
static __device__ void bem_rotate(Ctx& c, int n) {
    const int tid = threadIdx.x;
    double* P = c.bpt;
    for (int k = tid; k < n; k += c.nt) {
        const double x = P[8 * k + 0], y = P[8 * k + 1];
        const double rho = hypot(x, y);
        const double e_rho = P[8 * k + 5], e_z = P[8 * k + 6];
        double ex = 0.0, ey = 0.0;
        if (rho != 0.0) {
            ex = e_rho * (x / rho);
            ey = e_rho * (y / rho);
        }
        P[8 * k + 5] = ex;
        P[8 * k + 6] = ey;
        P[8 * k + 7] = e_z;
    }
    __syncthreads();
}


// ---------------------------------------------------------------------------
// learned form: the MLP surrogate evaluated on the tensor cores inside the
// stage (parameter offsets in the flat parameter array)
constexpr int kOW1 = 0, kOB1 = 256, kOW2 = 384, kOB2 = 16768, kOW3 = 16896, kOB3 = 33280, kOW4 = 33408, kOB4 = 49792,
              kOW5 = 49920, kOB5 = 50176;

// Surrogate field (E_rho, E_z) of records [0, n) into c.sout, from the
// closest-point frame bem_closest(c, n, true) left in sseg/st/sd.  Rows are
// processed 128 at a time: features and the first layer on the CUDA cores
// into a BF16 activation tile, three 128 x 128 layers as tcgen05.mma (K = 16
// steps) into the CTA's TMEM accumulator with the weights streamed into a
// BF16 tile, bias + SiLU applied while reading TMEM back, the last layer on
// the CUDA cores, then rescaling and rotation from the (normal, tangent)
// frame of the closest segment.
static __device__ void mlp_points(Ctx& c, int n, int* status_flag) {
    const SptBem& b = c.bem;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float* W = c.sw;
    const double lmin = log(c.dmin), lspan = log(c.dmax) - lmin;
    for (int cs = 0; cs < n; cs += 128) {
        const int m = min(128, n - cs);
        if (tid < 128) {
            float u1 = 0.f, u2 = 0.f;
            if (tid < m) {
                const int k = cs + tid;
                const int sg = c.sseg[k];
                const double sarc = (c.s_start[sg] + c.st[k] * segf(b, 4, sg)) / c.s_end;
                const double ld = log(fmin(fmax(c.sd[k], c.dmin), c.dmax));
                u1 = (float)(2.0 * (ld - lmin) / lspan - 1.0);
                u2 = (float)(2.0 * sarc - 1.0);
            }
            c.feat[2 * tid] = u1;
            c.feat[2 * tid + 1] = u2;
        }
        __syncthreads();
        for (int idx = tid; idx < 128 * 128; idx += c.nt) {
            const int r = idx >> 7, j = idx & 127;
            float h = 0.f;
            if (r < m) {
                const float v = fmaf(W[kOW1 + 2 * j], c.feat[2 * r], fmaf(W[kOW1 + 2 * j + 1], c.feat[2 * r + 1], W[kOB1 + j]));
                h = spt_umma::silu(v);
            }
            *reinterpret_cast<__nv_bfloat16*>(c.act + spt_umma::kmajor128(r, j)) = __float2bfloat16_rn(h);
        }
        for (int l = 0; l < 3; ++l) {
            const int ow = l == 0 ? kOW2 : (l == 1 ? kOW3 : kOW4);
            const int ob = l == 0 ? kOB2 : (l == 1 ? kOB3 : kOB4);
            // weights as the B operand: element (n = out, k = in) at W16[ow + n*128 + k], K-major
            for (int v = tid; v < 2048; v += c.nt) {
                const int nrow = v >> 4, kg = v & 15;
                const uint4 val = *reinterpret_cast<const uint4*>(c.sw16 + ow + nrow * 128 + kg * 8);
                *reinterpret_cast<uint4*>(c.wt + ((nrow >> 3) * 16 + kg) * 128 + (nrow & 7) * 16) = val;
            }
            spt_umma::fence_proxy();
            __syncthreads();
            if (tid == 0) {
                spt_umma::fence_after();
                const uint32_t idesc = spt_umma::idesc_bf16_128(0, 0);
#pragma unroll
                for (int kk = 0; kk < 8; ++kk)
                    spt_umma::mma(c.tmem, spt_umma::desc(c.act + kk * 256, 128, 2048),
                                  spt_umma::desc(c.wt + kk * 256, 128, 2048), idesc, kk > 0 ? 1u : 0u);
                spt_umma::commit(&c.bars[2]);
            }
            const bool ok = mbar_wait(&c.bars[2], c.phase[2]);
            c.phase[2] ^= 1u;
            if (!ok && tid == 0) *status_flag = SPT_GROUP_TIMEOUT;
            spt_umma::fence_after();
            // epilogue: warp w reads TMEM lanes 32 (w % 4) .. +31 (rows); with 8 warps
            // columns 64 (w / 4) .. +63, with 4 warps all 128 columns
            const int row = 32 * (warp & 3) + lane;
            for (int cb = 64 * (warp >> 2); cb < 128; cb += 64 * (c.nw >> 2))
#pragma unroll
            for (int c0 = 0; c0 < 64; c0 += 16) {
                float v[16];
                spt_umma::ld16(c.tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(cb + c0), v);
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const int col = cb + c0 + i;
                    const float h = spt_umma::silu(v[i] + W[ob + col]);
                    *reinterpret_cast<__nv_bfloat16*>(c.act + spt_umma::kmajor128(row, col)) = __float2bfloat16_rn(h);
                }
            }
            spt_umma::fence_before();
            spt_umma::fence_proxy();
            __syncthreads();
        }
        // last layer, rescaling and rotation: one warp per row
        for (int r = warp; r < m; r += c.nw) {
            float a0 = 0.f, a1 = 0.f;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int j = lane + 32 * q;
                const float h = __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(c.act + spt_umma::kmajor128(r, j)));
                a0 = fmaf(W[kOW5 + j], h, a0);
                a1 = fmaf(W[kOW5 + 128 + j], h, a1);
            }
            a0 = warp_sum(a0);
            a1 = warp_sum(a1);
            if (lane == 0) {
                const int k = cs + r;
                const int sg = c.sseg[k];
                const double t = c.st[k];
                const double sig = fabs(segf(b, 9, sg) + t * (segf(b, 10, sg) - segf(b, 9, sg))) + c.sig_floor;
                const double pos = (log(fmin(fmax(c.sd[k], c.dmin), c.dmax)) - lmin) / lspan * 63.0;
                const int i0 = min(62, max(0, (int)floor(pos)));
                const double fr = fmin(fmax(pos - i0, 0.0), 1.0);
                const double g = exp(c.log_scale[i0] + fr * (c.log_scale[i0 + 1] - c.log_scale[i0]));
                const double en = ((double)a0 + (double)W[kOB5]) * sig * g;
                const double et = ((double)a1 + (double)W[kOB5 + 1]) * sig * g;
                c.sout[2 * k] = en * segf(b, 7, sg) + et * segf(b, 5, sg);
                c.sout[2 * k + 1] = en * segf(b, 8, sg) + et * segf(b, 6, sg);
            }
        }
        __syncthreads();
    }
}

__device__ __forceinline__ bool spot_pick(uint32_t key, int particle, double frac) {
    uint32_t h = key * 0x9E3779B1u ^ (uint32_t)particle * 0x85EBCA77u;
    h ^= h >> 15;
    h *= 0x2C1B3C6Du;
    h ^= h >> 12;
    return (double)(h & 0xFFFFu) < frac * 65536.0;
}

// BEM field of the listed points in the learned form: the surrogate for
// every point, the exact sum for points within the band and for the spot
// checks (stable partition: exact records first), surrogate error of the
// spot checks recorded, then the rotation of phase D.
template <int FAR>
__device__ void surrogate_points(Ctx& c, int n, int* status_flag) {
    const int tid = threadIdx.x;
    double* P = c.bpt;
    __shared__ int s_cnt[kMaxWarps + 1];
    __shared__ int s_tot[2];
    bem_closest(c, n, true);
    mlp_points(c, n, status_flag);
    // stable partition of records [0, n): exact (band or spot) first.  The
    // destination of every record is found first (kept in sseg, which the
    // MLP no longer needs), then the records move through the act/wt scratch
    // (8 doubles each: slots 0-4 of the record, the surrogate E_rho, E_z, and
    // the list entry, negated minus one when the point lies in the band).
    if (tid == 0) s_tot[0] = 0;
    __syncthreads();
    for (int base = 0; base < n; base += c.nt) {
        const int k = base + tid;
        const bool ex = k < n && (c.sd[k] < c.band || spot_pick(c.key, c.list[k], c.spot));
        const unsigned bal = __ballot_sync(0xffffffffu, ex);
        if ((tid & 31) == 0 && bal) atomicAdd(&s_tot[0], __popc(bal));
    }
    __syncthreads();
    const int ne = s_tot[0];
    int run_ex = 0, run_su = 0;
    for (int base = 0; base < n; base += c.nt) {
        const int k = base + tid;
        const bool valid = k < n;
        const bool band = valid && c.sd[k] < c.band;
        const bool ex = valid && (band || spot_pick(c.key, c.list[k], c.spot));
        const unsigned be = __ballot_sync(0xffffffffu, ex);
        if ((tid & 31) == 0) s_cnt[tid >> 5] = __popc(be);
        __syncthreads();
        int pre_e = 0, tot_e = 0;
        for (int w = 0; w < c.nw; ++w) {
            if (w < (tid >> 5)) pre_e += s_cnt[w];
            tot_e += s_cnt[w];
        }
        const int chunk = min(c.nt, n - base);
        const int before = min((tid >> 5) * 32, chunk);  // records of this chunk before this warp
        const unsigned lt = (1u << (tid & 31)) - 1u;
        if (valid) {
            const int lane_e = __popc(be & lt);
            const int dst = ex ? run_ex + pre_e + lane_e : ne + run_su + (before - pre_e) + ((tid & 31) - lane_e);
            c.sseg[k] = 2 * dst + (band ? 1 : 0);
        }
        run_ex += tot_e;
        run_su += chunk - tot_e;
        __syncthreads();
    }
    double* tmp = reinterpret_cast<double*>(c.act);  // act + wt: 8192 doubles >= 8 n
    for (int k = tid; k < n; k += c.nt) {
        const int code = c.sseg[k];
        const int d = code >> 1;
        for (int f = 0; f < 5; ++f) tmp[8 * d + f] = P[8 * k + f];
        tmp[8 * d + 5] = c.sout[2 * k];
        tmp[8 * d + 6] = c.sout[2 * k + 1];
        tmp[8 * d + 7] = (code & 1) ? -(double)c.list[k] - 1.0 : (double)c.list[k];
    }
    __syncthreads();
    for (int k = tid; k < n; k += c.nt) {
        for (int f = 0; f < 5; ++f) P[8 * k + f] = tmp[8 * k + f];
        c.sout[2 * k] = tmp[8 * k + 5];
        c.sout[2 * k + 1] = tmp[8 * k + 6];
        const double v = tmp[8 * k + 7];
        c.list[k] = v < 0.0 ? (int)(-v - 1.0) : (int)v;
        c.fld[3 * k] = v < 0.0 ? 1.0 : 0.0;  // band flag, kept where the sums do not write
    }
    __syncthreads();
    bem_sums<SPT_FORM_SURROGATE, FAR>(c, ne, status_flag);
    unsigned long long n_spot = 0, n_band = 0;
    for (int k = tid; k < n; k += c.nt) {
        if (k >= ne) {
            P[8 * k + 5] = c.sout[2 * k];
            P[8 * k + 6] = c.sout[2 * k + 1];
        } else if (c.fld[3 * k] == 0.0) {  // a spot check: exact and surrogate both known
            // error relative to the whole external field there (uniform + perturbation)
            const double er = P[8 * k + 5], ez = P[8 * k + 6];
            const double dr = c.sout[2 * k] - er, dz = c.sout[2 * k + 1] - ez;
            const double tz = ez + c.g.E_gun;
            const float rel = (float)(sqrt(dr * dr + dz * dz) / fmax(sqrt(er * er + tz * tz), 1e-300));
            if (c.sstats) atomicMax(reinterpret_cast<unsigned int*>(c.sstats) + 6, __float_as_uint(rel));
            ++n_spot;
        } else {
            ++n_band;
        }
    }
    if (c.sstats) {
        const unsigned long long nsur = (unsigned long long)(n - ne);
        if (tid == 0 && nsur) atomicAdd(c.sstats + 0, nsur);
        n_band = warp_sum(n_band);
        n_spot = warp_sum(n_spot);
        if ((tid & 31) == 0) {
            if (n_band) atomicAdd(c.sstats + 1, n_band);
            if (n_spot) atomicAdd(c.sstats + 2, n_spot);
        }
    }
    __syncthreads();
    bem_rotate(c, n);
}

// Direct field of the point (x, y, z) by this warp, or its share of it: on-surface
// offset, near quadrature and adaptive far sum into S.  Uses the warp's own
// record c.wrec.
template <int FORM>
__device__ __forceinline__ void direct_sums(Ctx& c, double x, double y, double z, PointSums& S, PointCounts& n) {
    double* const P = c.wrec;
    if ((threadIdx.x & 31) == 0) {
        P[0] = x;
        P[1] = y;
        P[2] = z;
    }
    __syncwarp();
    closest_point(c, P, 0, false);
    __syncwarp();
    adaptive_sums<FORM>(c, P[3], P[4], S, n);
    __syncwarp();
}

// The same for the whole point, rotated; lane 0 returns it.
template <int FORM>
__device__ __forceinline__ void direct_point(Ctx& c, double x, double y, double z, PointCounts& n, double& ex,
                                             double& ey, double& ez) {
    PointSums S(0, 1);
    direct_sums<FORM>(c, x, y, z, S, n);
    double er;
    S.total(er, ez);
    rotate_rho(x, y, hypot(x, y), er, ex, ey);
}

// Direct points of a CTA with fewer points than half its warps: each point's
// rounds are shared by 2 or 4 warps (a point is a chain of ~15 rounds of one
// ring evaluation per lane, 20 us on one warp, and the CTA waits for it).  A
// warp leaves its slots, lane by lane, in `part`; after a barrier the point's
// warp adds them as PointSums::total does.
__device__ __forceinline__ int split_shares(int n, int warps) {
    return 4 * n <= warps ? 4 : (2 * n <= warps ? 2 : 1);
}
__device__ __forceinline__ void split_store(const PointSums& S, double* part) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if ((k & (S.shares - 1)) == S.share) {
            part[64 * k + lane] = S.r[k];
            part[64 * k + 32 + lane] = S.z[k];
        }
}
__device__ __forceinline__ void split_total(const double* part, double& er, double& ez) {
    const int lane = threadIdx.x & 31;
    const double* p = part + lane;
    er = warp_sum((p[0] + p[64]) + (p[128] + p[192]));
    ez = warp_sum((p[32] + p[96]) + (p[160] + p[224]));
}

// BEM field of the particles c.list[0..n) into c.fld, float64 adaptive form:
// one point a warp task, or its shares while there are few points.
__device__ __forceinline__ void bem_points_direct(Ctx& c, int n) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, E = c.E;
    const double* sp = c.sp;
    double* const part = c.tiles + (size_t)c.nw * (kWarpScratchInts / 2);
    __shared__ int s_task;
    const int shares = split_shares(n, c.nw);
    if (threadIdx.x == 0) s_task = c.nw;
    __syncthreads();
    PointCounts cnt;
    auto store = [&](int i, double er, double ez) {  // lane 0
        double ex, ey;
        rotate_rho(sp[i], sp[E + i], hypot(sp[i], sp[E + i]), er, ex, ey);
        c.fld[3 * i + 0] = ex;
        c.fld[3 * i + 1] = ey;
        c.fld[3 * i + 2] = ez;
    };
    for (int t = warp; t < n * shares; t = next_task(&s_task)) {
        const int k = t / shares, i = c.list[k];
        PointSums S(t - k * shares, shares);
        direct_sums<SPT_FORM_FP64>(c, sp[i], sp[E + i], sp[2 * E + i], S, cnt);
        if (shares == 1) {
            double er, ez;
            S.total(er, ez);
            if (lane == 0) store(i, er, ez);
        } else {
            split_store(S, part + 256 * k);
        }
    }
    if (shares > 1) {
        __syncthreads();
        for (int k = warp; k < n; k += c.nw) {
            double er, ez;
            split_total(part + 256 * k, er, ez);
            if (lane == 0) store(c.list[k], er, ez);
        }
    }
    count_points(c, cnt);
    __syncthreads();
}

// BEM field of the records [0, n) with the adaptive far rule, each point one
// warp task from start to end -- closest segment and on-surface offset, near
// quadrature, far sum, rotation -- taken dynamically from a CTA counter, so
// the only barrier is the one at the end.
template <int FORM>
__device__ void bem_points_fused(Ctx& c, int n) {
    const int lane = threadIdx.x & 31;
    double* P = c.bpt;
    __shared__ int s_task;
    if (threadIdx.x == 0) s_task = c.nw;
    __syncthreads();
    PointCounts cnt;
    for (int k = threadIdx.x >> 5; k < n; k = next_task(&s_task)) {
        double ex, ey, ez;
        direct_point<FORM>(c, P[8 * k + 0], P[8 * k + 1], P[8 * k + 2], cnt, ex, ey, ez);
        if (lane == 0) {
            P[8 * k + 5] = ex;
            P[8 * k + 6] = ey;
            P[8 * k + 7] = ez;
        }
        __syncwarp();
    }
    count_points(c, cnt);
    __syncthreads();
}

// BEM field of the n points listed in c.bpt (x, y, z at slots 0..2 of each
// 8-double record): the reference's evaluation, phases A-D, or the adaptive
// rule's one task per point.
template <int FORM, int FAR>
__device__ void bem_points(Ctx& c, int n, int* status_flag) {
    if constexpr (FAR == SPT_FAR_ADAPTIVE) {
        bem_points_fused<FORM>(c, n);
    } else {
        bem_closest(c, n, false);
        bem_sums<FORM, FAR>(c, n, status_flag);
        bem_rotate(c, n);
    }
}

// Softened pair sum over the live sources of the group (forces.py:16-29), mixed
// form: sum_j k q_i q_j (r_i - r_j) / (|r_i - r_j|^2 + a^2)^1.5, sources given
// by src(j, x, y, z, q).  Separations are taken in float64 (nearby particles
// far from the origin), then the rest in float32 with Kahan-compensated sums.
template <typename SRC>
__device__ __forceinline__ void pair_sum(const Ctx& c, int nl, int j0, int jstep, double xi, double yi, double zi,
                                         double qk, SRC src, double& fx, double& fy, double& fz, double& sabs) {
    // live sources j0, j0 + jstep, ... (the callers split one target's sources
    // over the lanes of a warp and add the partial sums)
    float ax = 0.f, ay = 0.f, az = 0.f, cx = 0.f, cy = 0.f, cz = 0.f, sa = 0.f;
    const float soft2 = (float)c.soft2;
    for (int jj = j0; jj < nl; jj += jstep) {
        double x, y, z, q;
        src(c.lidx[jj], x, y, z, q);
        const float dx = (float)(xi - x), dy = (float)(yi - y), dz = (float)(zi - z);
        const float r2 = fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, soft2)));
        const float rs = rsqrtf(r2);
        const float cf = (float)(qk * q) * (rs * rs * rs);
        kahan_add(ax, cx, cf * dx);
        kahan_add(ay, cy, cf * dy);
        kahan_add(az, cz, cf * dz);
        sa += fabsf(cf * dx) + fabsf(cf * dy) + fabsf(cf * dz);
    }
    sabs += sa;
    fx = (double)ax - (double)cx;
    fy = (double)ay - (double)cy;
    fz = (double)az - (double)cz;
}

// The indices of the live particles, in order, and their number, into c.lidx
// and c.nl: by the first warp; a barrier follows before they are read.
__device__ __forceinline__ void list_live(Ctx& c) {
    if (threadIdx.x >= 32) return;
    const int lane = threadIdx.x;
    int n = 0;
    for (int base = 0; base < c.E; base += 32) {
        const bool on = base + lane < c.E && c.live[base + lane];
        const unsigned m = __ballot_sync(0xffffffffu, on);
        if (on) c.lidx[n + __popc(m & ((1u << lane) - 1u))] = (uint16_t)(base + lane);
        n += __popc(m);
    }
    if (lane == 0) {
        c.nl[0] = n;
        if (n == 0) c.lidx[0] = 0;
    }
}

// 1 / sqrt(x)^3 times q, for positive normal x: the hardware's 20-bit estimate
// and one third-order Newton step (the next term is 5 e^3 / 16 < 1e-17).  The
// step takes x no larger than 2^997 (by its high word: a comparison of doubles
// made stage_flat 4 % slower), so that the result is 0, as the quotient's is, up
// to infinity (a softening that turns the pair force off, a runaway particle's
// square); a NaN stays one through y.
__device__ __forceinline__ double pair_coef(double x, double q) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double xs = __hiloint2double(min(__double2hiint(x), (1023 + 997) << 20), __double2loint(x));
    const double e = fma(-(xs * y), y, 1.0);
    y = fma(y * e, fma(0.375, e, 0.5), y);
    return (q * y) * (y * y);
}

// Float64 pair sums of one target (forces.py:16-191): the softened Coulomb
// force of the live sources and of their images, in one loop over the live
// list (the sources share dx, dy and their loads, and nothing in the loop
// branches, so that iterations overlap; the sums apart took a square root and
// a division with their special cases for each of up to four sets, one
// iteration after the other).  SETS: 1 Coulomb only; 2 and the plane image
// (z -> plane - z, -q); 4 and, in the apex frame, the sphere image and its
// plane image (forces.py:101-191), from img.  `zc` is subtracted from z for
// the images, `plane` the mirror sum of z + z'.
struct PairForces {
    double cx = 0.0, cy = 0.0, cz = 0.0;      // Coulomb
    double ax = 0.0, ay = 0.0, az = 0.0;      // sphere images
    double bx = 0.0, by = 0.0, bz = 0.0;      // plane images
    double dx = 0.0, dy = 0.0, dz = 0.0;      // plane images of the sphere images
};
template <int SETS, typename SRC, typename IMG>
__device__ __forceinline__ void pair_forces(int n, int j0, int jstep, double xi, double yi, double zi, double qk,
                                            double soft2, double zc, double plane, SRC src, IMG img, PairForces& f) {
    const double zl = zi - zc;
#pragma unroll 2
    for (int jj = j0; jj < n; jj += jstep) {
        double x, y, z, q;
        const int j = src(jj, x, y, z, q);
        const double dx = xi - x, dy = yi - y, dz = zi - z, qq = qk * q;
        const double r = fma(dx, dx, dy * dy);
        const double c = pair_coef(fma(dz, dz, r) + soft2, qq);
        f.cx = fma(c, dx, f.cx);
        f.cy = fma(c, dy, f.cy);
        f.cz = fma(c, dz, f.cz);
        if constexpr (SETS >= 2) {
            const double ez = zl - (plane - (z - zc));
            const double b = pair_coef(fma(ez, ez, r) + soft2, -qq);
            f.bx = fma(b, dx, f.bx);
            f.by = fma(b, dy, f.by);
            f.bz = fma(b, ez, f.bz);
        }
        if constexpr (SETS >= 4) {
            double ix, iy, iz, iq;
            img(j, ix, iy, iz, iq);
            const double ux = xi - ix, uy = yi - iy, uz = zl - iz, vz = zl - (plane - iz), uq = qk * iq;
            const double ur = fma(ux, ux, uy * uy);
            const double a = pair_coef(fma(uz, uz, ur) + soft2, uq);
            f.ax = fma(a, ux, f.ax);
            f.ay = fma(a, uy, f.ay);
            f.az = fma(a, uz, f.az);
            const double d = pair_coef(fma(vz, vz, ur) + soft2, -uq);
            f.dx = fma(d, ux, f.dx);
            f.dy = fma(d, uy, f.dy);
            f.dz = fma(d, vz, f.dz);
        }
    }
}

// sum of v over the T consecutive lanes of a lane group (T a power of two <= 32)
__device__ __forceinline__ double group_sum(double v, int T) {
    for (int o = T >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// ---------------------------------------------------------------------------
// one stage evaluation for the CTA's group: acc = cm*E + Fc/m + Fimg/m on
// live particles (geometry.py:289-299).  Positions in c.sp (3E), result in
// out (3 arrays of stride E... stored as out[0*E+i], out[E+i], out[2E+i]).

// BEM image-charge force on the stage positions c.sp of the group, into
// c.img (fx, fy, fz: 3E), from the image tables in c.bem.image.  Out of line:
// its per-mode register arrays stay out of the stage code's allocation.
static __device__ __noinline__ void stage_image_force(Ctx& c) {
    __shared__ int s_imgflag;
    const int E = c.E;
    const double* sx = c.sp;
    spt_img::ImgParams ip = spt_img::image_params(c.bem.image, &c.g, c.kc, 0.0);
    ip.soft2 = c.soft2;
    ip.chunks = image_chunks(c.bem.image.n_nodes, c.nt);
    auto load = [&](int i, double& x, double& y, double& z, double& q) {
        x = sx[i];
        y = sx[E + i];
        z = sx[2 * E + i];
        q = c.live[i] ? c.q[i] : 0.0;
    };
    spt_img::group_force<SPT_TRACE_IMAGE_MODES, false>(c.bem.image, ip, E, load, c.imgs, c.img, c.img + E, c.img + 2 * E,
                                                 &s_imgflag);
}

// GIVEN: the BEM perturbation field of every particle that takes one is in
// c.fld already (spt_accel's first pass).
template <int KIND, int FORM, int FAR, bool GIVEN = false>
__device__ void stage_accel(Ctx& c, double* out, int* status_flag) {
    const int E = c.E, tid = threadIdx.x;
    const double* sx = c.sp;
    const double* sy = c.sp + E;
    const double* sz = c.sp + 2 * E;
    const SptGeometry& g = c.g;

    // 1. external field
    if constexpr (!GIVEN && (KIND == SPT_GEOM_TIP_BEM || KIND == SPT_GEOM_WELL_BEM || KIND == SPT_GEOM_POST_BEM)) {
        // Field map (float64 and mixed forms): warp w takes particles w, w + nw,
        // ... (one per lane, spread over all warps of a small group), the
        // mapped ones are evaluated here and the rest compacted into c.list;
        // without a map every particle that needs the field is listed.
        const double* map = nullptr;
        if constexpr (FORM != SPT_FORM_SURROGATE && FAR == SPT_FAR_ADAPTIVE) map = field_map(c.bem);
        for (int i = tid; i < 3 * E; i += c.nt) c.fld[i] = 0.0;
        __shared__ int s_wcount[kMaxWarps + 1];
        int n_list = 0;
        for (int base = 0; base < E; base += c.nt) {
            const int i = map ? base + (tid >> 5) + c.nw * (tid & 31) : base + tid;
            bool need = false;
            double rho = 0.0, zi = 0.0;
            if (i < E && c.live[i]) {
                const double x = sx[i], y = sy[i], z = sz[i];
                need = bem_valid<KIND>(x, y, z, g) && blend_weight(z, g.z_handoff) > 0.0;
                if (map && need) {
                    rho = hypot(x, y);
                    zi = z;
                }
            }
            bool mapped = false;
            double mx = 0.0, my = 0.0, mz = 0.0;
            if (map) {
                const int leaf = need ? map_find(map, rho, zi) : -1;
                mapped = leaf >= 0;
                double er = 0.0;
                map_field_lanes(map, leaf, rho, zi, er, mz);
                if (mapped) rotate_rho(sx[i], sy[i], rho, er, mx, my);
                need = need && !mapped;
                count_add(c, SPT_CNT_CLUSTER_EVALS, mapped ? 1ull : 0ull);
            }
            const unsigned bal = __ballot_sync(0xffffffffu, need);
            if ((tid & 31) == 0) s_wcount[tid >> 5] = __popc(bal);
            __syncthreads();  // also: every zero of c.fld is written before a field
            if (tid == 0) {
                int acc = 0;
                for (int w = 0; w < c.nw; ++w) { const int t = s_wcount[w]; s_wcount[w] = acc; acc += t; }
                s_wcount[c.nw] = acc;
            }
            if (mapped) {
                c.fld[3 * i + 0] = mx;
                c.fld[3 * i + 1] = my;
                c.fld[3 * i + 2] = mz;
            }
            __syncthreads();
            if (need) {
                const int pos = n_list + s_wcount[tid >> 5] + __popc(bal & ((1u << (tid & 31)) - 1u));
                c.list[pos] = i;
                if constexpr (!(FORM == SPT_FORM_FP64 && FAR == SPT_FAR_ADAPTIVE)) {
                    c.bpt[8 * pos + 0] = sx[i];
                    c.bpt[8 * pos + 1] = sy[i];
                    c.bpt[8 * pos + 2] = sz[i];
                }
            }
            n_list += s_wcount[c.nw];
            __syncthreads();
        }
        if (n_list > 0) {
            if constexpr (FORM == SPT_FORM_FP64 && FAR == SPT_FAR_ADAPTIVE) {
                bem_points_direct(c, n_list);
            } else {
            if constexpr (FORM == SPT_FORM_SURROGATE)
                surrogate_points<FAR>(c, n_list, status_flag);
            else
                bem_points<FORM, FAR>(c, n_list, status_flag);
            // scatter: fld[i] = blended field
            for (int k = tid; k < n_list; k += c.nt) {
                const int i = c.list[k];
                c.fld[3 * i + 0] = c.bpt[8 * k + 5];
                c.fld[3 * i + 1] = c.bpt[8 * k + 6];
                c.fld[3 * i + 2] = c.bpt[8 * k + 7];
            }
            }
        }
        __syncthreads();
    }

    // 1b. BEM image-charge force of a tip or well built with z0
    // (bem/geometry.py:326-344, 780-797; bem/image_charge.py:816-1056):
    // the group's joint mode solve, into c.img (fx, fy, fz: 3E)
    bool bem_img = false;
    if constexpr (KIND == SPT_GEOM_TIP_BEM || KIND == SPT_GEOM_WELL_BEM) {
        bem_img = g.has_image && c.bem.image.n_nodes >= 2;
        if (bem_img) stage_image_force(c);
    }

    // 2. image sources for the sphere-on-plane construction (forces.py:170-183)
    const bool three_img = (KIND == SPT_GEOM_TIP || KIND == SPT_GEOM_POST_BEM) && g.has_image;
    if (three_img) {
        const double a = g.R - g.z0;
        const double zc = (KIND == SPT_GEOM_POST_BEM) ? g.L : 0.0;
        for (int j = tid; j < E; j += c.nt) {
            const double x = sx[j], y = sy[j], z = sz[j] - zc;
            const double d = sqrt(x * x + y * y + z * z);
            const double ds = d > 0.0 ? d : a;
            const double sh = (a * a) / (ds * ds);
            c.img[j] = x * sh;
            c.img[E + j] = y * sh;
            c.img[2 * E + j] = z * sh;
            c.img[3 * E + j] = -c.q[j] * (a / ds);
        }
        __syncthreads();
    }

    // 3. per live particle: field + pair sums over the live sources.  Each
    // target's sources are split over T lanes of a warp (as many as the CTA has
    // threads per live particle and no more than their number asks for, a power
    // of two, at most 32), whose partial sums are added with shuffles.  Mixed form: the sums run in float32 first; a
    // target whose sum of |float32 terms| / m exceeds kappa times its whole
    // acceleration is summed again in float64.
    const int nl = c.nl[0];
    for (int i = tid; i < E; i += c.nt)
        if (!c.live[i]) out[i] = out[E + i] = out[2 * E + i] = 0.0;
    int T = 1;
    while (T < 32 && T < nl && T * 2 * nl <= c.nt) T *= 2;
    const int per_pass = c.nt / T;
    const int sub = tid & (T - 1);
    const int lead = (tid & 31) & ~(T - 1);  // lane of the target's first sub-lane
    unsigned long long pairs = 0, redone = 0;
    const bool flat_img = KIND == SPT_GEOM_FLAT && g.has_image;
    const double zc = (KIND == SPT_GEOM_POST_BEM) ? g.L : 0.0;
    const double plane = flat_img ? -2.0 * g.z0 : -2.0 * (zc + g.z0);
    for (int base = 0; base < nl; base += per_pass) {
        const int at = base + tid / T;
        const bool act = at < nl;
        constexpr bool mix = FORM != SPT_FORM_FP64;
        const int i = c.lidx[act ? at : 0];
        const double xi = sx[i], yi = sy[i], zi = sz[i];
        const double qk = c.kc * c.q[i];
        double fcx, fcy, fcz, fix, fiy, fiz;
        auto reduce = [&]() {
            fcx = group_sum(fcx, T); fcy = group_sum(fcy, T); fcz = group_sum(fcz, T);
            fix = group_sum(fix, T); fiy = group_sum(fiy, T); fiz = group_sum(fiz, T);
        };
        // this lane's share of the target's Coulomb (fc) and image (fi) sums (lanes without work add zeros)
        auto pass64 = [&](bool on) {
            PairForces f;
            auto real = [&](int jj, double& x, double& y, double& z, double& q) {
                const int j = c.lidx[jj];
                x = sx[j]; y = sy[j]; z = sz[j]; q = c.q[j];
                return j;
            };
            auto sphere = [&](int j, double& x, double& y, double& z, double& q) {
                x = c.img[j]; y = c.img[E + j]; z = c.img[2 * E + j]; q = c.img[3 * E + j];
            };
            const int n = on ? nl : 0;
            if constexpr (KIND == SPT_GEOM_TIP || KIND == SPT_GEOM_POST_BEM) {
                if (three_img) pair_forces<4>(n, sub, T, xi, yi, zi, qk, c.soft2, zc, plane, real, sphere, f);
                else pair_forces<1>(n, sub, T, xi, yi, zi, qk, c.soft2, zc, plane, real, sphere, f);
            } else if constexpr (KIND == SPT_GEOM_FLAT) {
                if (flat_img) pair_forces<2>(n, sub, T, xi, yi, zi, qk, c.soft2, 0.0, plane, real, sphere, f);
                else pair_forces<1>(n, sub, T, xi, yi, zi, qk, c.soft2, 0.0, plane, real, sphere, f);
            } else {
                pair_forces<1>(n, sub, T, xi, yi, zi, qk, c.soft2, 0.0, plane, real, sphere, f);
            }
            // a lone particle has no Coulomb force, whatever the softening makes of its own term
            fcx = E > 1 ? f.cx : 0.0; fcy = E > 1 ? f.cy : 0.0; fcz = E > 1 ? f.cz : 0.0;
            fix = (f.ax + f.bx) + f.dx; fiy = (f.ay + f.by) + f.dy; fiz = (f.az + f.bz) + f.dz;
        };
        double sabs = 0.0;
        auto pass32 = [&](bool on) {
            fcx = fcy = fcz = fix = fiy = fiz = sabs = 0.0;
            if (!on) return;
            auto real = [&](int j, double& x, double& y, double& z, double& q) {
                x = sx[j]; y = sy[j]; z = sz[j]; q = c.q[j];
            };
            if (E > 1) pair_sum(c, nl, sub, T, xi, yi, zi, qk, real, fcx, fcy, fcz, sabs);
            if (flat_img) {
                auto mirror = [&](int j, double& x, double& y, double& z, double& q) {
                    x = sx[j]; y = sy[j]; z = plane - sz[j]; q = -c.q[j];
                };
                pair_sum(c, nl, sub, T, xi, yi, zi, qk, mirror, fix, fiy, fiz, sabs);
            } else if (three_img) {
                const double zl = zi - zc;
                double s1x, s1y, s1z, s2x, s2y, s2z, s3x, s3y, s3z;
                auto sphere = [&](int j, double& x, double& y, double& z, double& q) {
                    x = c.img[j]; y = c.img[E + j]; z = c.img[2 * E + j]; q = c.img[3 * E + j];
                };
                auto mirror = [&](int j, double& x, double& y, double& z, double& q) {
                    x = sx[j]; y = sy[j]; z = plane - (sz[j] - zc); q = -c.q[j];
                };
                auto mirror_sphere = [&](int j, double& x, double& y, double& z, double& q) {
                    x = c.img[j]; y = c.img[E + j]; z = plane - c.img[2 * E + j]; q = -c.img[3 * E + j];
                };
                pair_sum(c, nl, sub, T, xi, yi, zl, qk, sphere, s1x, s1y, s1z, sabs);
                pair_sum(c, nl, sub, T, xi, yi, zl, qk, mirror, s2x, s2y, s2z, sabs);
                pair_sum(c, nl, sub, T, xi, yi, zl, qk, mirror_sphere, s3x, s3y, s3z, sabs);
                fix = (s1x + s2x) + s3x;
                fiy = (s1y + s2y) + s3y;
                fiz = (s1z + s2z) + s3z;
            }
        };
        if (act && sub == 0) {
            pairs += (E > 1 ? E : 0) + (flat_img ? E : 0) + (three_img ? 3 * E : 0);
        }
        if constexpr (mix) pass32(act);
        else pass64(act);
        reduce();
        sabs = group_sum(sabs, T);
        auto bem_image = [&]() {  // the BEM image force of 1b takes the place of a pair-sum image
            if (bem_img && act && sub == 0) {
                fix = c.img[i];
                fiy = c.img[E + i];
                fiz = c.img[2 * E + i];
            }
        };
        bem_image();
        double ex = 0.0, ey = 0.0, ez = 0.0;
        if (act && sub == 0) {
            if (KIND == SPT_GEOM_FLAT) {
                ex = 0.0; ey = 0.0; ez = (zi >= 0.0) ? g.E_gun : 0.0;
            } else if (KIND == SPT_GEOM_TIP) {
                tip_field(xi, yi, zi, g.E_gun, g.R, ex, ey, ez);
            } else {
                // blend(near, far) with near = where(valid, uniform + pert, 0) (bem/geometry.py:44-55, bem/fields.py:186-211)
                const double w = blend_weight(zi, g.z_handoff);
                const bool valid = bem_valid<KIND>(xi, yi, zi, g);
                const double fz = (zi >= 0.0) ? g.E_gun : 0.0;
                double nx = 0.0, ny = 0.0, nz = 0.0;
                if (valid && w > 0.0) {
                    nx = 0.0 + c.fld[3 * i + 0];
                    ny = 0.0 + c.fld[3 * i + 1];
                    nz = g.E_gun + c.fld[3 * i + 2];
                } else if (valid) {
                    nx = 0.0; ny = 0.0; nz = g.E_gun;  // pert finite; times w = 0
                }
                ex = w * nx + (1.0 - w) * 0.0;
                ey = w * ny + (1.0 - w) * 0.0;
                ez = w * nz + (1.0 - w) * fz;
            }
        }
        const double mi = act ? c.m[i] : 1.0;
        auto accel_of = [&](double& ax, double& ay, double& az) {
            ax = (c.cm * ex + fcx / mi) + fix / mi;
            ay = (c.cm * ey + fcy / mi) + fiy / mi;
            az = (c.cm * ez + fcz / mi) + fiz / mi;
        };
        double ax = 0.0, ay = 0.0, az = 0.0;
        bool redo = false;
        if (act && sub == 0) {
            accel_of(ax, ay, az);
            redo = mix && !(sabs / mi <= c.kappa * sqrt(ax * ax + ay * ay + az * az));
        }
        if constexpr (mix) {
            redo = __shfl_sync(0xffffffffu, redo, lead);
            if (__any_sync(0xffffffffu, redo)) {
                pass64(act && redo);
                reduce();
                bem_image();
                if (act && redo && sub == 0) {
                    accel_of(ax, ay, az);
                    ++redone;
                }
            }
        }
        if (act && sub == 0) {
            out[i] = ax;
            out[E + i] = ay;
            out[2 * E + i] = az;
        }
    }
    if constexpr (FORM != SPT_FORM_FP64) count_add(c, SPT_CNT_FP64_TARGETS, redone);
    c.pairs += pairs;  // counted once a group: a warp sum here would be in every stage's chain
    __syncthreads();
}

// ---------------------------------------------------------------------------
// add the CTA's shared-memory counters to the global ones and clear them;
// all threads call, after a barrier that orders every count_add before it
__device__ inline void flush_counters(Ctx& c, unsigned long long* counters) {
    for (int k = threadIdx.x; k < SPT_N_COUNTERS; k += blockDim.x) {
        const unsigned long long v = c.cnt[k];
        if (counters && v) atomicAdd(counters + k, v);
        c.cnt[k] = 0;
    }
}

__device__ inline void init_barriers(Ctx& c) {
    c.phase[0] = 0u;
    c.phase[1] = 0u;
    c.phase[2] = 0u;
    if (threadIdx.x == 0) {
        mbar_init(&c.bars[0], 1);
        mbar_init(&c.bars[1], 1);
        mbar_init(&c.bars[2], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
}

// ---------------------------------------------------------------------------
// the persistent integrator

struct GroupScalars {
    double t, h, hr, next_cp, err, h_next, next_out;
    int status, exhausted, accepted, out_ptr, out_exh, fire_out;
    long long n_acc, n_rej;
};

// number of entries of the ascending array v[0..n) that are <= x
__device__ __forceinline__ int count_le(const double* v, int n, double x) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (v[mid] <= x) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// Cubic Hermite pieces (screens.py:118-152), evaluated in the reference's order.
__device__ __forceinline__ double hermite_z(double p0, double v0, double p1, double v1, double dt, double s) {
    const double s2 = s * s, s3 = s2 * s;
    const double h00 = 2 * s3 - 3 * s2 + 1, h10 = s3 - 2 * s2 + s, h01 = -2 * s3 + 3 * s2, h11 = s3 - s2;
    return h00 * p0 + h10 * dt * v0 + h01 * p1 + h11 * dt * v1;
}

__device__ __forceinline__ double sgn(double x) { return x > 0.0 ? 1.0 : (x < 0.0 ? -1.0 : 0.0); }

// Screen crossings of one particle over one accepted step (screens.py:43-115,
// 155-168): the Hermite z(s) is split at its extrema so each bracket is
// monotone; a sign change over a bracket is located by 60 bisections and the
// crossing state (Hermite position and derivative) is appended to the record
// buffer.  Half-open (t_old, t_new]: a start exactly on the screen is not a crossing.
static __device__ __noinline__ void screen_crossings(const SptTraceParams& prm, const double* o, const double* n, double t_old,
                                 double dt, long long particle) {
    const double z0 = o[2], z1 = n[2];
    bool moving = false;
    for (int k = 0; k < 6; ++k) moving |= (o[k] != n[k]);
    if (!moving || !(dt > 0.0)) return;
    const double u0 = dt * o[5], u1 = dt * n[5];
    double A = 3 * (2 * (z0 - z1) + u0 + u1);
    double B = 2 * (3 * (z1 - z0) - 2 * u0 - u1);
    double C = u0;
    double sc = fmax(fmax(fabs(A), fabs(B)), fabs(C));
    sc = sc > 0.0 ? sc : 1.0;
    A /= sc; B /= sc; C /= sc;
    const double disc = B * B - 4 * A * C;
    const double q = -0.5 * (B + (B >= 0.0 ? 1.0 : -1.0) * sqrt(fmax(disc, 0.0)));
    double r0 = q / (A != 0.0 ? A : 1.0);
    const double r1 = C / (q != 0.0 ? q : 1.0);
    const double lin = -C / (B != 0.0 ? B : 1.0);
    if (A == 0.0) r0 = lin;
    const bool v0 = (disc >= 0.0) && (A != 0.0 || B != 0.0) && (r0 > 0.0) && (r0 < 1.0);
    const bool v1 = (disc >= 0.0) && (A != 0.0) && (q != 0.0) && (r1 > 0.0) && (r1 < 1.0);
    double cut[4] = {0.0, v0 ? r0 : 1.0, v1 ? r1 : 1.0, 1.0};
    if (cut[1] > cut[2]) { const double tmp = cut[1]; cut[1] = cut[2]; cut[2] = tmp; }
    for (int sidx = 0; sidx < prm.n_screens; ++sidx) {
        const double zs = prm.screens[sidx];
        for (int iv = 0; iv < 3; ++iv) {
            const double left = cut[iv], right = cut[iv + 1];
            const double f0 = hermite_z(z0, o[5], z1, n[5], dt, left) - zs;
            const double f1 = hermite_z(z0, o[5], z1, n[5], dt, right) - zs;
            if (!(right > left) || f0 == 0.0 || sgn(f0) == sgn(f1)) continue;
            double lo = left, hi = right, flo = f0;
            for (int it = 0; it < 60; ++it) {
                const double mid = 0.5 * (lo + hi);
                const double fm = hermite_z(z0, o[5], z1, n[5], dt, mid) - zs;
                const bool same = sgn(fm) == sgn(flo);
                if (same) { lo = mid; flo = fm; } else { hi = mid; }
            }
            const double sv = 0.5 * (lo + hi);
            const double s2 = sv * sv, s3 = s2 * sv;
            const double h00 = 2 * s3 - 3 * s2 + 1, h10 = s3 - 2 * s2 + sv, h01 = -2 * s3 + 3 * s2, h11 = s3 - s2;
            const double d00 = 6 * s2 - 6 * sv, d10 = 3 * s2 - 4 * sv + 1, d01 = -6 * s2 + 6 * sv, d11 = 3 * s2 - 2 * sv;
            const unsigned long long slot = atomicAdd(prm.screen_count, 1ull);
            if ((long long)slot >= prm.screen_capacity) continue;
            const long long cap = prm.screen_capacity;
            double* r = prm.screen_rec;
            r[0 * cap + slot] = t_old + sv * dt;
            for (int k = 0; k < 3; ++k) {
                r[(1 + k) * cap + slot] = h00 * o[k] + (h10 * dt) * o[3 + k] + h01 * n[k] + (h11 * dt) * n[3 + k];
                r[(4 + k) * cap + slot] = (d00 / dt) * o[k] + d10 * o[3 + k] + (d01 / dt) * n[k] + d11 * n[3 + k];
            }
            r[7 * cap + slot] = (double)sidx;
            r[8 * cap + slot] = (double)particle;
        }
    }
}

static __device__ __noinline__ void write_output(const SptTraceParams& prm, long long n_particles, int k, long long pidx,
                                             double t, const double* s) {
    double* r = prm.output_rec + (size_t)k * 7 * n_particles;
    r[pidx] = t;
    for (int c = 0; c < 6; ++c) r[(size_t)(1 + c) * n_particles + pidx] = s[c];
    prm.output_flag[(size_t)k * n_particles + pidx] = 1;
}

// learned-form parameters into the context, and the CTA's 128 TMEM columns
// (the 128 x 128 FP32 accumulator) for its whole lifetime; all threads call
static __device__ void bind_surrogate(Ctx& c, const SptTraceParams& prm, uint32_t* s_tmem) {
    c.sw = prm.sur_w;
    c.sw16 = static_cast<const __nv_bfloat16*>(prm.sur_w16);
    c.s_start = prm.sur_s_start;
    c.log_scale = prm.sur_log_scale;
    c.s_end = prm.sur_s_end;
    c.sig_floor = prm.sur_sig_floor;
    c.band = prm.sur_band;
    c.spot = prm.sur_spot;
    c.dmin = prm.sur_d_min;
    c.dmax = prm.sur_d_max;
    c.sstats = prm.sur_stats;
    if ((threadIdx.x >> 5) == 0) spt_umma::alloc(s_tmem, 128);
    spt_umma::fence_before();
    __syncthreads();
    spt_umma::fence_after();
    c.tmem = *s_tmem;
}

static __device__ void release_surrogate(Ctx& c) {
    spt_umma::fence_before();
    __syncthreads();
    if ((threadIdx.x >> 5) == 0) spt_umma::dealloc(c.tmem, 128);
}

// Persistent trace kernel for geometry kind KIND, arithmetic form FORM and far
// rule FAR.  Launched with blockDim.x in {32, 64, 128, 256} (at most 128
// registers a thread, so two 256-thread CTAs, four of 128 or eight of 64 fit
// an SM's register file); every CTA takes groups from the work queue until it
// is empty.
template <int KIND, int FORM, int FAR>
__global__ void __launch_bounds__(kMaxThreads, 2)
trace_kernel(const __grid_constant__ SptState st, const __grid_constant__ SptTraceParams prm,
             const __grid_constant__ SptGeometry geo, const __grid_constant__ SptBem bem, int* work,
             double* big_slots) {
    extern __shared__ __align__(16) double smem[];
    __shared__ GroupScalars gs;
    __shared__ int s_g;
    __shared__ double s_red[kMaxWarps];
    __shared__ int s_flag;
    __shared__ unsigned long long s_cnt[SPT_N_COUNTERS];
    const int tid = threadIdx.x;
    Ctx c(geo, bem);
    c.cm = prm.charge_to_mass;
    c.kc = prm.coulomb_constant;
    c.soft2 = prm.plummer_radius * prm.plummer_radius;
    const int Emax = st.max_group_size;
    constexpr bool sur = FORM == SPT_FORM_SURROGATE;
    bind(c, smem, Emax, FAR, big_slots ? big_slots + (size_t)blockIdx.x * big_slot_doubles(Emax) : nullptr, s_cnt, sur);
    // launch-configuration parameters (bind sets the defaults)
    c.round_pts = (prm.round_points >= 1 && prm.round_points <= kRound) ? prm.round_points : kRound;
    if (prm.kappa_max > 0.0) c.kappa = prm.kappa_max;
    __shared__ uint32_t s_tmem;
    if constexpr (sur) bind_surrogate(c, prm, &s_tmem);
    init_barriers(c);
    const int nt = c.nt;
    // y0 (state at the step start), nw (candidate state) and the seven stage
    // slopes kp (positions' = velocities) and kv (velocities' = accelerations):
    // component k of particle i at Y0[k * Emax + i], KP(s)[k * E + i]
    double* const Y0 = c.y0;
    double* const NW = c.nw_;
    auto KP = [&](int s_) { return c.kp + 3 * s_ * Emax; };
    auto KV = [&](int s_) { return c.kv + 3 * s_ * Emax; };

    // groups to process: all, or the compacted running ones (count written on the device)
    const int n_run = st.n_active ? *st.n_active : st.n_groups;
    for (;;) {
        if (tid == 0) s_g = atomicAdd(work, 1);
        __syncthreads();
        const int gi = s_g;
        __syncthreads();
        if (gi >= n_run) break;
        const int g = st.group_order ? st.group_order[gi] : gi;
        const long long base = st.group_offset[g];
        const int E = (int)(st.group_offset[g + 1] - base);
        if (tid == 0) {
            gs.status = st.status[g];
            gs.t = st.t[g];
            gs.h = st.h[g];
            gs.n_acc = st.n_accepted[g];
            gs.n_rej = st.n_rejected[g];
            s_flag = 0;
        }
        __syncthreads();
        if (E <= 0 || gs.status >= SPT_GROUP_DONE) continue;
        // the layout keeps the Emax offsets; the stage routines use this group's E
        c.E = E;
        for (int i = tid; i < E; i += nt) {
            Y0[0 * Emax + i] = st.x[base + i]; Y0[1 * Emax + i] = st.y[base + i]; Y0[2 * Emax + i] = st.z[base + i];
            Y0[3 * Emax + i] = st.vx[base + i]; Y0[4 * Emax + i] = st.vy[base + i]; Y0[5 * Emax + i] = st.vz[base + i];
            c.tb[i] = st.t_birth[base + i];
            c.td[i] = st.t_death[base + i];
            c.q[i] = st.charge[base + i];
            c.m[i] = st.mass[base + i];
        }
        __syncthreads();
        // sorted birth times (batched_rk45.py:164): rank sort, ties by index
        for (int i = tid; i < E; i += nt) {
            const double v = c.tb[i];
            int r = 0;
            for (int j = 0; j < E; ++j) { const double u = c.tb[j]; r += (u < v) || (u == v && j < i); }
            c.cps[r] = v;
        }
        __syncthreads();
        if (tid == 0) {
            gs.fire_out = -1;
            if (gs.status == SPT_GROUP_NEW) {
                gs.t = c.cps[0];
                gs.h = (prm.t_max - gs.t) * prm.initial_step_fraction;
                // a group born entirely at or after t_max has nothing to integrate: it is
                // done as it stands (the reference would take a backward step to t_max)
                gs.status = gs.t < prm.t_max ? SPT_GROUP_RUNNING : SPT_GROUP_DONE;
                // an output time equal to the start time fires here (batched_rk45.py:191-209)
                if (prm.n_outputs > 0) {
                    const int last = count_le(prm.output_times, prm.n_outputs, gs.t) - 1;
                    if (last >= 0 && prm.output_times[last] == gs.t) gs.fire_out = last;
                }
            }
        }
        __syncthreads();
        if (gs.fire_out >= 0) {
            for (int i = tid; i < E; i += nt) {
                if (c.tb[i] <= gs.t) {
                    const double sv[6] = {Y0[i], Y0[Emax + i], Y0[2 * Emax + i], Y0[3 * Emax + i], Y0[4 * Emax + i],
                                          Y0[5 * Emax + i]};
                    write_output(prm, st.n_particles, gs.fire_out, base + i, gs.t, sv);
                }
            }
        }
        for (long long att = 0; att < prm.max_attempts; ++att) {
            if (gs.status != SPT_GROUP_RUNNING) break;
            if (tid == 0) {
                // next checkpoint (batched_rk45.py:228-242)
                int lo = 0, hi = E;
                while (lo < hi) { const int mid = (lo + hi) >> 1; if (c.cps[mid] <= gs.t) lo = mid + 1; else hi = mid; }
                gs.exhausted = lo >= E;
                gs.next_cp = gs.exhausted ? prm.t_max : c.cps[lo];
                double target = fmin(gs.next_cp, prm.t_max);
                if (prm.n_outputs > 0) {
                    const int optr = count_le(prm.output_times, prm.n_outputs, gs.t);
                    gs.out_ptr = optr;
                    gs.out_exh = optr >= prm.n_outputs;
                    gs.next_out = gs.out_exh ? prm.t_max : prm.output_times[optr];
                    target = fmin(target, gs.next_out);
                }
                gs.hr = fmin(gs.h, target - gs.t);
                if (!(gs.hr > 0.0) || !isfinite(gs.hr)) gs.status = SPT_GROUP_NONFINITE;
            }
            __syncthreads();
            if (gs.status != SPT_GROUP_RUNNING) break;
            const double t = gs.t, hr = gs.hr;
            for (int i = tid; i < E; i += nt) c.live[i] = (t >= c.tb[i]) && (t < c.td[i]);
            __syncthreads();
            list_live(c);  // (the stages' first barrier orders it)
            // seven stage evaluations through one call site of stage_accel (a second
            // inlined copy of the stage code would double the kernel's instruction footprint)
            for (int s = 0; s < 7; ++s) {
                double* const kps = KP(s);
                if (s < 6) {
                    for (int i = tid; i < E; i += nt) {
                        double p[6];
#pragma unroll
                        for (int k = 0; k < 6; ++k) p[k] = Y0[k * Emax + i];
                        for (int j = 0; j < s; ++j) {
                            const double a = kA[s][j];
                            if (a == 0.0) continue;
                            const double ha = __dmul_rn(hr, a);
                            const double* kpj = KP(j);
                            const double* kvj = KV(j);
#pragma unroll
                            for (int k = 0; k < 3; ++k) {
                                p[k] = __dadd_rn(p[k], __dmul_rn(ha, kpj[k * E + i]));
                                p[3 + k] = __dadd_rn(p[3 + k], __dmul_rn(ha, kvj[k * E + i]));
                            }
                        }
                        const bool lv = c.live[i];
#pragma unroll
                        for (int k = 0; k < 3; ++k) {
                            c.sp[k * E + i] = p[k];
                            kps[k * E + i] = lv ? p[3 + k] : 0.0;
                        }
                    }
                } else {
                    // 5th-order solution and the endpoint stage (batched_rk45.py:365-370)
                    for (int i = tid; i < E; i += nt) {
#pragma unroll
                        for (int k = 0; k < 3; ++k) {
                            double sp = 0.0, sv = 0.0;
#pragma unroll
                            for (int j = 0; j < 6; ++j) {
                                sp = __dadd_rn(sp, __dmul_rn(kB[j], KP(j)[k * E + i]));
                                sv = __dadd_rn(sv, __dmul_rn(kB[j], KV(j)[k * E + i]));
                            }
                            const double pn = __dadd_rn(Y0[k * Emax + i], __dmul_rn(hr, sp));
                            const double vn = __dadd_rn(Y0[(3 + k) * Emax + i], __dmul_rn(hr, sv));
                            NW[k * Emax + i] = pn;
                            NW[(3 + k) * Emax + i] = vn;
                            c.sp[k * E + i] = pn;
                            kps[k * E + i] = c.live[i] ? vn : 0.0;
                        }
                    }
                }
                __syncthreads();
                c.key = (uint32_t)g * 2654435761u ^ (uint32_t)(gs.n_acc + gs.n_rej) * 40503u ^ (uint32_t)s * 97u;
                stage_accel<KIND, FORM, FAR>(c, KV(s), &s_flag);
            }
            // embedded error norm (batched_rk45.py:372-393)
            double part = 0.0;
            for (int i = tid; i < E; i += nt) {
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    double ep = 0.0, ev = 0.0;
#pragma unroll
                    for (int j = 0; j < 7; ++j) {
                        ep = __dadd_rn(ep, __dmul_rn(kE[j], KP(j)[k * E + i]));
                        ev = __dadd_rn(ev, __dmul_rn(kE[j], KV(j)[k * E + i]));
                    }
                    ep = __dmul_rn(hr, ep);
                    ev = __dmul_rn(hr, ev);
                    const double y0p = Y0[k * Emax + i], nwp = NW[k * Emax + i];
                    const double y0v = Y0[(3 + k) * Emax + i], nwv = NW[(3 + k) * Emax + i];
                    const double scp = __dadd_rn(prm.atol, __dmul_rn(prm.rtol, fmax(fabs(y0p), fabs(nwp))));
                    const double scv = __dadd_rn(kSpeedOfLight * prm.atol, __dmul_rn(prm.rtol, fmax(fabs(y0v), fabs(nwv))));
                    const double a = __ddiv_rn(ep, scp), b = __ddiv_rn(ev, scv);
                    part = __dadd_rn(part, __dadd_rn(__dmul_rn(a, a), __dmul_rn(b, b)));
                }
            }
            part = warp_sum(part);
            if ((tid & 31) == 0) s_red[tid >> 5] = part;
            __syncthreads();
            if (tid == 0) {
                double sq = 0.0;
                for (int w = 0; w < c.nw; ++w) sq += s_red[w];
                double err = sqrt(sq / (double)(6 * E));
                if (err == 0.0) err = kTiny;
                const bool acc = err <= 1.0;
                double fac = prm.safety * pow(err, -1.0 / 5.0);
                fac = fmin(fmax(fac, prm.min_factor), prm.max_factor);
                gs.err = err;
                gs.accepted = acc;
                gs.h_next = hr * fac;
                const long long k_att = gs.n_acc + gs.n_rej;
                if (prm.log_capacity > 0 && k_att < prm.log_capacity) {
                    prm.log_h[(size_t)g * prm.log_capacity + k_att] = hr;
                    prm.log_err[(size_t)g * prm.log_capacity + k_att] = err;
                }
                c.cnt[SPT_CNT_ATTEMPTS] += 1;
                c.cnt[SPT_CNT_STAGE_EVALS] += 7ull * E;
            }
            __syncthreads();
            if (gs.accepted) {
                const double t_new = t + hr;
                const double dt = t_new - t;
                const double tol_out = 1e-9 * fmax(prm.t_max, 1e-30);
                const bool hit = prm.n_outputs > 0 && !gs.out_exh && t_new >= gs.next_out - tol_out;
                unsigned long long n_live = 0;
                for (int i = tid; i < E; i += nt) {
                    const bool was = c.live[i];
                    n_live += was;
                    if (was && kill_test<KIND>(NW[i], NW[Emax + i], NW[2 * Emax + i], geo)) c.td[i] = t_new;
                    if (hit || prm.n_screens > 0) {
                        double o[6], nv[6];
                        for (int k = 0; k < 6; ++k) { o[k] = Y0[k * Emax + i]; nv[k] = NW[k * Emax + i]; }
                        if (hit && c.tb[i] <= t_new) write_output(prm, st.n_particles, gs.out_ptr, base + i, t_new, nv);
                        if (prm.n_screens > 0) screen_crossings(prm, o, nv, t, dt, base + i);
                    }
#pragma unroll
                    for (int k = 0; k < 6; ++k) Y0[k * Emax + i] = NW[k * Emax + i];
                }
                count_add(c, SPT_CNT_LIVE_STEPS, n_live);
                if (tid == 0) {
                    gs.t = t_new;
                    gs.n_acc += 1;
                    const double tol = 1e-9 * fmax(prm.t_max, 1e-30);
                    if (!gs.exhausted && t_new >= gs.next_cp - tol)
                        gs.h = (prm.t_max - t_new) * prm.initial_step_fraction;
                    else
                        gs.h = gs.h_next;
                    if (!(t_new < prm.t_max * (1 - 1e-14))) gs.status = SPT_GROUP_DONE;
                    c.cnt[SPT_CNT_ACCEPTED] += 1;
                    c.cnt[SPT_CNT_PARTICLE_STEPS] += (unsigned long long)E;
                }
            } else if (tid == 0) {
                gs.h = gs.h_next;
                gs.n_rej += 1;
            }
            if (tid == 0) {
                if (isnan(gs.err)) gs.status = SPT_GROUP_NONFINITE;
                if (s_flag) gs.status = s_flag;
            }
            __syncthreads();
        }
        // write back
        for (int i = tid; i < E; i += nt) {
            st.x[base + i] = Y0[i]; st.y[base + i] = Y0[Emax + i]; st.z[base + i] = Y0[2 * Emax + i];
            st.vx[base + i] = Y0[3 * Emax + i]; st.vy[base + i] = Y0[4 * Emax + i]; st.vz[base + i] = Y0[5 * Emax + i];
            st.t_death[base + i] = c.td[i];
        }
        if (tid == 0) {
            st.t[g] = gs.t;
            st.h[g] = gs.h;
            st.status[g] = gs.status;
            st.n_accepted[g] = gs.n_acc;
            st.n_rejected[g] = gs.n_rej;
        }
        count_add(c, SPT_CNT_PAIR_EVALS, c.pairs);
        c.pairs = 0;
        __syncthreads();
        flush_counters(c, prm.counters);
        __syncthreads();
        // A timed-out barrier wait leaves this CTA's barrier phases unknown:
        // stop taking groups (the remaining ones stay NEW/RUNNING for the host).
        if (s_flag == SPT_GROUP_TIMEOUT) break;
    }
    if constexpr (sur) release_surrogate(c);
}

// one stage evaluation per group (spt_accel), one CTA per group; GIVEN: ax, ay,
// az hold the perturbation field (of the particles that take one) on entry
template <int KIND, int FORM, int FAR, bool GIVEN>
__global__ void __launch_bounds__(kMaxThreads, 2)
accel_kernel(const __grid_constant__ SptAccelArgs a, const __grid_constant__ SptGeometry geo,
             const __grid_constant__ SptBem bem) {
    extern __shared__ __align__(16) double smem[];
    __shared__ int s_flag;
    __shared__ unsigned long long s_cnt[SPT_N_COUNTERS];
    const int tid = threadIdx.x;
    const int g = blockIdx.x;
    Ctx c(geo, bem);
    c.cm = a.charge_to_mass;
    c.kc = a.coulomb_constant;
    c.soft2 = a.plummer_radius * a.plummer_radius;
    const int Emax = a.max_group_size;
    bind(c, smem, Emax, FAR, nullptr, s_cnt, false, !GIVEN, false);
    init_barriers(c);
    const long long base = a.group_offset[g];
    const int E = (int)(a.group_offset[g + 1] - base);
    c.E = E;
    if (tid == 0) s_flag = 0;
    for (int i = tid; i < E; i += c.nt) {
        c.sp[i] = a.x[base + i];
        c.sp[E + i] = a.y[base + i];
        c.sp[2 * E + i] = a.z[base + i];
        c.live[i] = a.active[base + i];
        c.q[i] = a.charge[base + i];
        c.m[i] = a.mass[base + i];
        if constexpr (GIVEN) {
            c.fld[3 * i + 0] = a.ax[base + i];
            c.fld[3 * i + 1] = a.ay[base + i];
            c.fld[3 * i + 2] = a.az[base + i];
        }
    }
    __syncthreads();
    list_live(c);
    __syncthreads();
    double* out = c.kv;
    stage_accel<KIND, FORM, FAR, GIVEN>(c, out, &s_flag);
    for (int i = tid; i < E; i += c.nt) {
        a.ax[base + i] = out[i];
        a.ay[base + i] = out[E + i];
        a.az[base + i] = out[2 * E + i];
    }
}

// ---------------------------------------------------------------------------
// One group per warp, several groups per CTA, the CTA's BEM points pooled
// (groups of at most 32 particles, BEM geometries without the BEM
// image-charge force, float64 form, adaptive far rule).
//
// Lane i of a warp is particle i of the warp's group: stage combination,
// pair sums (one target per lane, sources in order), error norm, controller,
// kills, screens and output times run per warp, with the group scalars held
// alike by every lane (sums over the group taken in lane 0 and broadcast).
// The CTA's warps advance their groups through each stage in step, and the
// BEM points of all of them go into one CTA-wide task pool that every warp
// draws from (closest segment, near quadrature, adaptive far sum -- the CTA
// team's warp routines, so the same field to the bit -- and the rotation,
// written back to the owning group).  With one group per CTA, warps that had
// finished their share of a stage's points idled at the barrier behind the
// slowest point; with one free-running group per warp, the warps' scattered
// positions in the stage code thrashed the instruction cache.  Here the pool
// of ~W x 17 points balances to within one point, warps share their
// instruction stream, and warps whose group is done help with the others'
// points until the work queue is empty.  The step's state -- y0, the
// 5th-order solution and the seven stage slopes -- lives in a per-warp slot
// in global memory (component k of lane i at slot[k * 32 + i], coalesced),
// read and written past L1 so that L1 keeps the BEM tables.

constexpr int kWarpSlotComps = 54;  // y0 6, 5th-order solution 6, stage velocities 21, stage accelerations 21
constexpr int kWarpSlotDoubles = kWarpSlotComps * 32;
// per-warp shared doubles: BEM record 8, stage positions and charges 4 x 32,
// sphere images 4 x 32, BEM fields 3 x 32, live list 32 ints
constexpr int kWarpTeamDoubles = 8 + 4 * 32 + 4 * 32 + 3 * 32 + 16;

__host__ __device__ inline size_t warp_team_smem(int warps) {
    return (size_t)warps * ((size_t)kWarpScratchInts * 4 + (size_t)kWarpTeamDoubles * 8) +
           (size_t)split_doubles(warps) * 8;
}

__device__ __forceinline__ double warp_min_all(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;  // min is exact and order-free: every lane holds the same value
}

// per-warp shared region of warp w
struct WarpTeam {
    double *rec, *sx, *sy, *sz, *q, *img, *fld;
    int* lidx;
    __device__ WarpTeam(double* smem, int nw, int w) {
        double* t = smem + (size_t)nw * kWarpScratchInts / 2 + (size_t)w * kWarpTeamDoubles;
        rec = t;
        sx = t + 8;
        sy = sx + 32;
        sz = sy + 32;
        q = sz + 32;
        img = q + 32;
        fld = img + 128;
        lidx = reinterpret_cast<int*>(fld + 96);
    }
};

// The CTA's BEM task pool of one stage: entries (warp << 5 | particle), drawn
// one per warp task, or each shared by 2 or 4 warps while there are few; every
// warp calls, between the barriers that close the appends and open the next
// stage.  Shared points' slots end in `part` (pool_totals adds them).
__device__ __forceinline__ void pool_bem_points(Ctx& c, double* smem, const int* entries, int count, int* next,
                                                double* part, PointCounts& n) {
    const int lane = threadIdx.x & 31;
    const int shares = split_shares(count, c.nw);
    for (;;) {
        int t = 0;
        if (lane == 0) t = atomicAdd(next, 1);
        t = __shfl_sync(0xffffffffu, t, 0);
        if (t >= count * shares) break;
        const int e = entries[t / shares];
        const WarpTeam own(smem, c.nw, e >> 5);
        const int k = e & 31;
        PointSums S(t & (shares - 1), shares);
        direct_sums<SPT_FORM_FP64>(c, own.sx[k], own.sy[k], own.sz[k], S, n);
        if (shares == 1) {
            double er, ez, ex, ey;
            S.total(er, ez);
            if (lane == 0) {
                rotate_rho(own.sx[k], own.sy[k], hypot(own.sx[k], own.sy[k]), er, ex, ey);
                own.fld[3 * k + 0] = ex;
                own.fld[3 * k + 1] = ey;
                own.fld[3 * k + 2] = ez;
            }
        } else {
            split_store(S, part + 256 * (t / shares));
        }
        __syncwarp();
    }
}

// The shared points of this warp's own group (after the barrier).
__device__ __forceinline__ void pool_totals(Ctx& c, const WarpTeam& w, const int* entries, int count,
                                            const double* part) {
    if (split_shares(count, c.nw) == 1) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int t = 0; t < count; ++t) {
        if ((entries[t] >> 5) != warp) continue;
        const int k = entries[t] & 31;
        double er, ez, ex, ey;
        split_total(part + 256 * t, er, ez);
        if (lane == 0) {
            rotate_rho(w.sx[k], w.sy[k], hypot(w.sx[k], w.sy[k]), er, ex, ey);
            w.fld[3 * k + 0] = ex;
            w.fld[3 * k + 1] = ey;
            w.fld[3 * k + 2] = ez;
        }
    }
    __syncwarp();
}

// The rest of a stage for this warp's group, after the pool: images, pair
// sums and the blended external field into this lane's acceleration.
template <int KIND>
__device__ __forceinline__ void stage_finish_warp(Ctx& c, const WarpTeam& w, bool live, bool need, double xi,
                                                  double yi, double zi, double mi, double& ax, double& ay,
                                                  double& az) {
    const int lane = threadIdx.x & 31, E = c.E;
    const SptGeometry& g = c.g;
    // image sources of the sphere-on-plane construction (forces.py:170-183)
    const bool three_img = KIND == SPT_GEOM_POST_BEM && g.has_image;
    const double zc = (KIND == SPT_GEOM_POST_BEM) ? g.L : 0.0;
    if (three_img) {
        if (lane < E) {
            const double a = g.R - g.z0;
            const double x = xi, y = yi, z = zi - zc;
            const double d = sqrt(x * x + y * y + z * z);
            const double ds = d > 0.0 ? d : a;
            const double sh = (a * a) / (ds * ds);
            w.img[lane] = x * sh;
            w.img[32 + lane] = y * sh;
            w.img[64 + lane] = z * sh;
            w.img[96 + lane] = -w.q[lane] * (a / ds);
        }
        __syncwarp();
    }
    // Pair sums (forces.py:16-57, 101-191): T lanes a target while the live
    // particles leave lanes free (targets and sources by the live list), the
    // partial sums added with shuffles and handed to the target's lane.
    const unsigned lm = __ballot_sync(0xffffffffu, live);
    const int nl = __popc(lm);
    double fcx = 0.0, fcy = 0.0, fcz = 0.0, fix = 0.0, fiy = 0.0, fiz = 0.0;
    if (nl > 0 && (E > 1 || three_img)) {
        int T = 1;
        while (T * 2 * nl <= 32 && T * 2 <= nl) T *= 2;
        const int at = lane / T, sub = lane & (T - 1);
        const bool on = at < nl;
        const int i = w.lidx[on ? at : 0];
        PairForces f;
        auto real = [&](int jj, double& x, double& y, double& z, double& q) {
            const int j = w.lidx[jj];
            x = w.sx[j]; y = w.sy[j]; z = w.sz[j]; q = w.q[j];
            return j;
        };
        auto sphere = [&](int j, double& x, double& y, double& z, double& q) {
            x = w.img[j]; y = w.img[32 + j]; z = w.img[64 + j]; q = w.img[96 + j];
        };
        const double qk = c.kc * w.q[i];
        const double plane = -2.0 * (zc + g.z0);
        if (three_img)
            pair_forces<4>(on ? nl : 0, sub, T, w.sx[i], w.sy[i], w.sz[i], qk, c.soft2, zc, plane, real, sphere, f);
        else
            pair_forces<1>(on ? nl : 0, sub, T, w.sx[i], w.sy[i], w.sz[i], qk, c.soft2, zc, plane, real, sphere, f);
        const int from = __popc(lm & ((1u << lane) - 1u)) * T;  // the lane that holds this lane's target
        auto hand = [&](double v) { return __shfl_sync(0xffffffffu, group_sum(v, T), from & 31); };
        fcx = hand(E > 1 ? f.cx : 0.0);  // (a lone particle has no Coulomb force)
        fcy = hand(E > 1 ? f.cy : 0.0);
        fcz = hand(E > 1 ? f.cz : 0.0);
        if (three_img) {
            fix = hand((f.ax + f.bx) + f.dx);
            fiy = hand((f.ay + f.by) + f.dy);
            fiz = hand((f.az + f.bz) + f.dz);
        }
    }
    ax = ay = az = 0.0;
    unsigned long long pairs = 0;
    if (live) {
        pairs = (E > 1 ? E : 0) + (three_img ? 3 * E : 0);
        // blend(near, far) with near = where(valid, uniform + pert, 0) (bem/geometry.py:44-55, bem/fields.py:186-211)
        const double wgt = blend_weight(zi, g.z_handoff);
        const bool valid = bem_valid<KIND>(xi, yi, zi, g);
        const double fz = (zi >= 0.0) ? g.E_gun : 0.0;
        double nx = 0.0, ny = 0.0, nz = 0.0;
        if (valid && wgt > 0.0) {
            const double bx = need ? w.fld[3 * lane + 0] : 0.0;
            const double by = need ? w.fld[3 * lane + 1] : 0.0;
            const double bz = need ? w.fld[3 * lane + 2] : 0.0;
            nx = 0.0 + bx;
            ny = 0.0 + by;
            nz = g.E_gun + bz;
        } else if (valid) {
            nx = 0.0; ny = 0.0; nz = g.E_gun;
        }
        const double ex = wgt * nx + (1.0 - wgt) * 0.0;
        const double ey = wgt * ny + (1.0 - wgt) * 0.0;
        const double ez = wgt * nz + (1.0 - wgt) * fz;
        ax = (c.cm * ex + fcx / mi) + fix / mi;
        ay = (c.cm * ey + fcy / mi) + fiy / mi;
        az = (c.cm * ez + fcz / mi) + fiz / mi;
    }
    count_add(c, SPT_CNT_PAIR_EVALS, pairs);
}

template <int KIND, int FORM>
__global__ void __launch_bounds__(kMaxThreads, 2)
trace_warp_kernel(const __grid_constant__ SptState st, const __grid_constant__ SptTraceParams prm,
                  const __grid_constant__ SptGeometry geo, const __grid_constant__ SptBem bem, int* work,
                  double* slots) {
    static_assert(FORM == SPT_FORM_FP64, "the warp team runs the float64 form");
    extern __shared__ __align__(16) double smem[];
    __shared__ unsigned long long s_cnt[SPT_N_COUNTERS];
    __shared__ int s_pool[3][kMaxThreads];  // three stages' task pools, used in turn
    __shared__ int s_pool_n[3], s_pool_next[3];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int k = threadIdx.x; k < SPT_N_COUNTERS; k += blockDim.x) s_cnt[k] = 0;
    if (threadIdx.x < 3) s_pool_n[threadIdx.x] = s_pool_next[threadIdx.x] = 0;
    Ctx c(geo, bem);
    c.cm = prm.charge_to_mass;
    c.kc = prm.coulomb_constant;
    c.soft2 = prm.plummer_radius * prm.plummer_radius;
    c.kappa = prm.kappa_max > 0.0 ? prm.kappa_max : kKappa;
    c.round_pts = 1;
    c.cnt = s_cnt;
    c.nt = blockDim.x;
    c.nw = nw;
    c.tiles = smem;  // far-rule scratch of every warp (far_adaptive_warp takes its own by warp index)
    const WarpTeam w(smem, nw, warp);
    c.wrec = w.rec;
    double* const part = smem + (warp_team_smem(nw) / 8 - split_doubles(nw));
    const double* const map = field_map(bem);
    PointCounts pts;
    double* const slot = slots + ((size_t)blockIdx.x * nw + warp) * kWarpSlotDoubles + lane;
    auto ld = [&](int k) { return __ldcg(slot + 32 * k); };
    auto sto = [&](int k, double v) { __stcg(slot + 32 * k, v); };
    constexpr int Y0 = 0, NW = 6, KP = 12, KV = 33;
    __syncthreads();

    const int n_run = st.n_active ? *st.n_active : st.n_groups;
    // this warp's group and its scalars (alike in every lane)
    bool have = false, queue_empty = false;
    int g = 0, E = 0, status = 0;
    long long base = 0, pi = 0, n_acc = 0, n_rej = 0, att = 0;
    bool in = false;
    double tb = INFINITY, td = INFINITY, mi = 1.0, t = 0.0, h = 0.0;
    auto write_back = [&]() {
        if (in) {
            st.x[pi] = ld(Y0 + 0); st.y[pi] = ld(Y0 + 1); st.z[pi] = ld(Y0 + 2);
            st.vx[pi] = ld(Y0 + 3); st.vy[pi] = ld(Y0 + 4); st.vz[pi] = ld(Y0 + 5);
            st.t_death[pi] = td;
        }
        if (lane == 0) {
            st.t[g] = t;
            st.h[g] = h;
            st.status[g] = status;
            st.n_accepted[g] = n_acc;
            st.n_rejected[g] = n_rej;
        }
        have = false;
    };
    int pp = 0;  // the current stage's pool
    // Single electrons are near the surface, where a point is a direct sum, in
    // the first tenth of their attempts only.  A CTA takes its next ones together,
    // when all it has are done: then either every warp has a direct point or
    // none has (replaced one by one, every stage waited for somebody's).
    const bool together = st.max_group_size == 1;
    for (;;) {
        const bool may_take =
            !together || !__syncthreads_or(have && status == SPT_GROUP_RUNNING && att < prm.max_attempts);
        // ready this warp's group for an attempt: take groups from the work
        // queue until one is running and within this call's attempt budget
        double hr = 0.0, next_cp = 0.0, next_out = 0.0;
        bool exhausted = true, out_exh = true;
        int out_ptr = 0;
        for (;;) {
            if (!have) {
                if (queue_empty || !may_take) break;
                int gi = 0;
                if (lane == 0) gi = atomicAdd(work, 1);
                gi = __shfl_sync(0xffffffffu, gi, 0);
                if (gi >= n_run) { queue_empty = true; break; }
                g = st.group_order ? st.group_order[gi] : gi;
                base = st.group_offset[g];
                E = (int)(st.group_offset[g + 1] - base);
                status = st.status[g];
                if (E <= 0 || E > 32 || status >= SPT_GROUP_DONE) continue;
                in = lane < E;
                pi = base + (in ? lane : 0);
                tb = in ? st.t_birth[pi] : INFINITY;
                td = in ? st.t_death[pi] : INFINITY;
                mi = in ? st.mass[pi] : 1.0;
                __syncwarp();  // the previous group's last pair sums have read q
                w.q[lane] = in ? st.charge[pi] : 0.0;
                if (in) {
                    sto(Y0 + 0, st.x[pi]); sto(Y0 + 1, st.y[pi]); sto(Y0 + 2, st.z[pi]);
                    sto(Y0 + 3, st.vx[pi]); sto(Y0 + 4, st.vy[pi]); sto(Y0 + 5, st.vz[pi]);
                }
                t = st.t[g];
                h = st.h[g];
                n_acc = st.n_accepted[g];
                n_rej = st.n_rejected[g];
                att = 0;
                have = true;
                int fire_out = -1;
                if (status == SPT_GROUP_NEW) {
                    // start at the first birth (batched_rk45.py:164-178)
                    t = warp_min_all(tb);
                    h = (prm.t_max - t) * prm.initial_step_fraction;
                    status = t < prm.t_max ? SPT_GROUP_RUNNING : SPT_GROUP_DONE;
                    if (prm.n_outputs > 0) {
                        const int last = count_le(prm.output_times, prm.n_outputs, t) - 1;
                        if (last >= 0 && prm.output_times[last] == t) fire_out = last;
                    }
                }
                if (fire_out >= 0 && in && tb <= t) {
                    double sv[6];
                    for (int k = 0; k < 6; ++k) sv[k] = ld(Y0 + k);
                    write_output(prm, st.n_particles, fire_out, base + lane, t, sv);
                }
            }
            if (status != SPT_GROUP_RUNNING || att >= prm.max_attempts) {
                write_back();
                continue;
            }
            // next checkpoint: the first birth after t (batched_rk45.py:228-242)
            const double ncp = warp_min_all(tb > t ? tb : INFINITY);
            exhausted = !(ncp < INFINITY);
            next_cp = exhausted ? prm.t_max : ncp;
            double target = fmin(next_cp, prm.t_max);
            out_ptr = 0;
            out_exh = true;
            next_out = prm.t_max;
            if (prm.n_outputs > 0) {
                out_ptr = count_le(prm.output_times, prm.n_outputs, t);
                out_exh = out_ptr >= prm.n_outputs;
                next_out = out_exh ? prm.t_max : prm.output_times[out_ptr];
                target = fmin(target, next_out);
            }
            hr = fmin(h, target - t);
            if (!(hr > 0.0) || !isfinite(hr)) {
                status = SPT_GROUP_NONFINITE;
                write_back();
                continue;
            }
            break;
        }
        const bool run = have;
        if (!__syncthreads_or(run)) {
            // nobody runs: the queue is empty, unless the last running single
            // ended above (no step left), when nobody else was taking groups
            if (may_take) break;
            continue;
        }
        c.E = E;
        const bool live = run && in && (t >= tb) && (t < td);
        // seven stage evaluations (batched_rk45.py:326-370), in step across the CTA
        for (int s = 0; s < 7; ++s, pp = pp == 2 ? 0 : pp + 1) {
            double px = 0.0, py = 0.0, pz = 0.0;
            bool need = false;
            if (run) {
                if (in) {
                    if (s < 6) {
                        double p[6];
#pragma unroll
                        for (int k = 0; k < 6; ++k) p[k] = ld(Y0 + k);
                        for (int j = 0; j < s; ++j) {
                            const double a = kA[s][j];
                            if (a == 0.0) continue;
                            const double ha = __dmul_rn(hr, a);
#pragma unroll
                            for (int k = 0; k < 3; ++k) {
                                p[k] = __dadd_rn(p[k], __dmul_rn(ha, ld(KP + 3 * j + k)));
                                p[3 + k] = __dadd_rn(p[3 + k], __dmul_rn(ha, ld(KV + 3 * j + k)));
                            }
                        }
                        px = p[0]; py = p[1]; pz = p[2];
#pragma unroll
                        for (int k = 0; k < 3; ++k) sto(KP + 3 * s + k, live ? p[3 + k] : 0.0);
                    } else {
                        double pn[3];
#pragma unroll
                        for (int k = 0; k < 3; ++k) {
                            double sp = 0.0, sv = 0.0;
#pragma unroll
                            for (int j = 0; j < 6; ++j) {
                                sp = __dadd_rn(sp, __dmul_rn(kB[j], ld(KP + 3 * j + k)));
                                sv = __dadd_rn(sv, __dmul_rn(kB[j], ld(KV + 3 * j + k)));
                            }
                            pn[k] = __dadd_rn(ld(Y0 + k), __dmul_rn(hr, sp));
                            const double vn = __dadd_rn(ld(Y0 + 3 + k), __dmul_rn(hr, sv));
                            sto(NW + k, pn[k]);
                            sto(NW + 3 + k, vn);
                            sto(KP + 18 + k, live ? vn : 0.0);
                        }
                        px = pn[0]; py = pn[1]; pz = pn[2];
                    }
                }
                w.sx[lane] = px;
                w.sy[lane] = py;
                w.sz[lane] = pz;
                if (s == 0) {  // the live list of this attempt
                    const unsigned lm = __ballot_sync(0xffffffffu, live);
                    if (live) w.lidx[__popc(lm & ((1u << lane) - 1u))] = lane;
                }
                // the BEM field of the live particles inside the valid region
                // with blend weight > 0: mapped points here, by their own
                // warp, the others to the CTA's pool
                need = live && bem_valid<KIND>(px, py, pz, geo) && blend_weight(pz, geo.z_handoff) > 0.0;
                bool direct = need;
                if (map) {
                    const double rho = need ? hypot(px, py) : 0.0;
                    const int leaf = need ? map_find(map, rho, pz) : -1;
                    double er = 0.0, ez = 0.0;
                    map_field_lanes(map, leaf, rho, pz, er, ez);
                    if (leaf >= 0) {
                        direct = false;
                        double ex, ey;
                        rotate_rho(px, py, rho, er, ex, ey);
                        w.fld[3 * lane + 0] = ex;
                        w.fld[3 * lane + 1] = ey;
                        w.fld[3 * lane + 2] = ez;
                        ++pts.cl_evals;
                    }
                }
                const unsigned m = __ballot_sync(0xffffffffu, direct);
                int at = 0;
                if (lane == 0 && m) at = atomicAdd(&s_pool_n[pp], __popc(m));
                at = __shfl_sync(0xffffffffu, at, 0);
                if (direct) s_pool[pp][at + __popc(m & ((1u << lane) - 1u))] = (warp << 5) | lane;
            }
            __syncthreads();
            // The pool after next was last read before this barrier and is
            // next appended to after the next stage's: cleared in between, so
            // a stage without direct points needs no second barrier.
            if (threadIdx.x == 0) {
                const int p2 = pp == 0 ? 2 : pp - 1;
                s_pool_n[p2] = 0;
                s_pool_next[p2] = 0;
            }
            const int n_direct = s_pool_n[pp];
            if (n_direct > 0) {  // alike in every thread
                pool_bem_points(c, smem, s_pool[pp], n_direct, &s_pool_next[pp], part, pts);
                __syncthreads();
                pool_totals(c, w, s_pool[pp], n_direct, part);
            }
            if (run) {
                double ax, ay, az;
                stage_finish_warp<KIND>(c, w, live, need, px, py, pz, mi, ax, ay, az);
                if (in) {
                    sto(KV + 3 * s + 0, ax);
                    sto(KV + 3 * s + 1, ay);
                    sto(KV + 3 * s + 2, az);
                }
                __syncwarp();  // the positions and images are rewritten by the next stage
            }
        }
        if (!run) continue;
        // embedded error norm (batched_rk45.py:372-393); the sum over the
        // group in lane 0, as the CTA kernel's fixed-order block sum
        double part = 0.0;
        if (in) {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                double ep = 0.0, ev = 0.0;
#pragma unroll
                for (int j = 0; j < 7; ++j) {
                    ep = __dadd_rn(ep, __dmul_rn(kE[j], ld(KP + 3 * j + k)));
                    ev = __dadd_rn(ev, __dmul_rn(kE[j], ld(KV + 3 * j + k)));
                }
                ep = __dmul_rn(hr, ep);
                ev = __dmul_rn(hr, ev);
                const double y0p = ld(Y0 + k), nwp = ld(NW + k);
                const double y0v = ld(Y0 + 3 + k), nwv = ld(NW + 3 + k);
                const double scp = __dadd_rn(prm.atol, __dmul_rn(prm.rtol, fmax(fabs(y0p), fabs(nwp))));
                const double scv = __dadd_rn(kSpeedOfLight * prm.atol, __dmul_rn(prm.rtol, fmax(fabs(y0v), fabs(nwv))));
                const double a = __ddiv_rn(ep, scp), b = __ddiv_rn(ev, scv);
                part = __dadd_rn(part, __dadd_rn(__dmul_rn(a, a), __dmul_rn(b, b)));
            }
        }
        const double sq = 0.0 + __shfl_sync(0xffffffffu, warp_sum(part), 0);
        double err = sqrt(sq / (double)(6 * E));
        if (err == 0.0) err = kTiny;
        const bool accepted = err <= 1.0;
        double fac = prm.safety * pow(err, -1.0 / 5.0);
        fac = fmin(fmax(fac, prm.min_factor), prm.max_factor);
        const double h_next = hr * fac;
        if (lane == 0) {
            const long long k_att = n_acc + n_rej;
            if (prm.log_capacity > 0 && k_att < prm.log_capacity) {
                prm.log_h[(size_t)g * prm.log_capacity + k_att] = hr;
                prm.log_err[(size_t)g * prm.log_capacity + k_att] = err;
            }
            atomicAdd(c.cnt + SPT_CNT_ATTEMPTS, 1ull);
            atomicAdd(c.cnt + SPT_CNT_STAGE_EVALS, 7ull * E);
        }
        if (accepted) {
            const double t_new = t + hr;
            const double dt = t_new - t;
            const double tol_out = 1e-9 * fmax(prm.t_max, 1e-30);
            const bool hit = prm.n_outputs > 0 && !out_exh && t_new >= next_out - tol_out;
            if (in) {
                double o[6], nv[6];
#pragma unroll
                for (int k = 0; k < 6; ++k) { o[k] = ld(Y0 + k); nv[k] = ld(NW + k); }
                if (live && kill_test<KIND>(nv[0], nv[1], nv[2], geo)) td = t_new;
                if (hit && tb <= t_new) write_output(prm, st.n_particles, out_ptr, base + lane, t_new, nv);
                if (prm.n_screens > 0) screen_crossings(prm, o, nv, t, dt, base + lane);
#pragma unroll
                for (int k = 0; k < 6; ++k) sto(Y0 + k, nv[k]);
            }
            count_add(c, SPT_CNT_LIVE_STEPS, live ? 1ull : 0ull);
            t = t_new;
            n_acc += 1;
            const double tol = 1e-9 * fmax(prm.t_max, 1e-30);
            if (!exhausted && t_new >= next_cp - tol)
                h = (prm.t_max - t_new) * prm.initial_step_fraction;
            else
                h = h_next;
            if (!(t_new < prm.t_max * (1 - 1e-14))) status = SPT_GROUP_DONE;
            if (lane == 0) {
                atomicAdd(c.cnt + SPT_CNT_ACCEPTED, 1ull);
                atomicAdd(c.cnt + SPT_CNT_PARTICLE_STEPS, (unsigned long long)E);
            }
        } else {
            h = h_next;
            n_rej += 1;
        }
        if (isnan(err)) status = SPT_GROUP_NONFINITE;
        ++att;
    }
    count_points(c, pts);
    __syncthreads();
    flush_counters(c, prm.counters);
}

// ---------------------------------------------------------------------------
// host-side launchers of the kernels above, instantiated per geometry kind in
// spt_trace_<kind>.cu (kept out of the C ABI's translation unit so that the
// kinds compile in parallel)

struct TraceLaunch {
    const SptState* s;
    const SptTraceParams* p;
    const SptGeometry* g;
    SptBem bem;
    int threads;                 // CTA width
    int* work;                   // zeroed work-queue counter
    double* slots;               // big-group slots (or null)
    long long max_slots;         // largest grid: the CTAs the slot buffer holds, or a caller's cap (0: no limit)
    cudaStream_t stream;
    bool warp_team;              // one group per warp (trace_warp_kernel), slope slots at `slots`
};

// Which points a field launch (spt_field.cu) evaluates: points 0 .. n-1
// (active NULL), or of the particles group_offset[0] .. group_offset[n_groups]
// - 1, at most `most`, the active ones in the geometry's valid region below its
// handoff (the others' field is set to zero).
struct FieldMask {
    const uint8_t* active;
    const int64_t* group_offset;
    int n_groups;
    SptGeometry g;
};
int launch_field(const double* x, const double* y, const double* z, long long n, long long most, const SptBem& b,
                 const FieldMask& mask, double* ex, double* ey, double* ez, cudaStream_t st);

// Shared memory and grid of a trace launch; returns 0 or a cudaError_t.
template <int KIND, int FORM, int FAR>
int trace_grid(int max_group_size, int threads, int n_groups, long long max_slots, int img_doubles, size_t* smem,
               int* grid, int* per_sm) {
    const Layout L = make_layout(max_group_size, FAR, FORM == SPT_FORM_SURROGATE, true, threads / 32, img_doubles);
    auto kern = trace_kernel<KIND, FORM, FAR>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L.bytes);
    if (e != cudaSuccess) return (int)e;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, kern, threads, L.bytes);
    if (e != cudaSuccess) return (int)e;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    long long cap = (long long)sms * (*per_sm);
    if (max_slots > 0 && cap > max_slots) cap = max_slots;
    *grid = (int)(n_groups < cap ? n_groups : cap);
    *smem = L.bytes;
    return 0;
}

// Shared memory and grid of a warp-team launch (trace_warp_kernel): as many
// CTAs as the SMs hold, no more than the groups need, capped by max_slots.
template <int KIND, int FORM>
int trace_warp_grid(int threads, int n_groups, long long max_slots, size_t* smem, int* grid, int* per_sm) {
    const size_t bytes = warp_team_smem(threads / 32);
    auto kern = trace_warp_kernel<KIND, FORM>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return (int)e;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, kern, threads, bytes);
    if (e != cudaSuccess) return (int)e;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    long long cap = (long long)sms * (*per_sm);
    if (max_slots > 0 && cap > max_slots) cap = max_slots;
    const long long need = ((long long)n_groups + threads / 32 - 1) / (threads / 32);
    *grid = (int)(need < cap ? need : cap);
    *smem = bytes;
    return 0;
}

template <int KIND, int FORM>
int trace_warp_launch(const TraceLaunch& t, int grid, size_t smem) {
    trace_warp_kernel<KIND, FORM><<<grid, t.threads, smem, t.stream>>>(*t.s, *t.p, *t.g, t.bem, t.work, t.slots);
    return (int)cudaGetLastError();
}

template <int KIND, int FORM, int FAR>
int trace_launch(const TraceLaunch& t, int grid, size_t smem) {
    trace_kernel<KIND, FORM, FAR><<<grid, t.threads, smem, t.stream>>>(*t.s, *t.p, *t.g, t.bem, t.work, t.slots);
    return (int)cudaGetLastError();
}

template <int KIND, int FORM, int FAR, bool GIVEN = false>
int accel_launch(const SptAccelArgs* a, const SptGeometry* g, const SptBem& bem, cudaStream_t stream) {
    const Layout L = make_layout(a->max_group_size, FAR, false, !GIVEN, kMaxWarps,
                                 image_scratch(*g, bem, a->max_group_size, kMaxThreads), false);
    auto kern = accel_kernel<KIND, FORM, FAR, GIVEN>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L.bytes);
    if (e != cudaSuccess) return (int)e;
    kern<<<a->n_groups, kMaxThreads, L.bytes, stream>>>(*a, *g, bem);
    return (int)cudaGetLastError();
}

// Whether an output of spt_accel overlaps an input: then each group's CTA must
// read its inputs before it writes anything, as the one-launch form does.
inline bool accel_in_place(const SptAccelArgs* a) {
    const uintptr_t n = 8 * (uintptr_t)(a->n_particles > 0 ? a->n_particles : (long long)a->n_groups * a->max_group_size);
    const double* in[] = {a->x, a->y, a->z, a->charge, a->mass};
    const double* out[] = {a->ax, a->ay, a->az};
    for (const double* o : out) {
        const uintptr_t p = reinterpret_cast<uintptr_t>(o), act = reinterpret_cast<uintptr_t>(a->active);
        for (const double* i : in) {
            const uintptr_t q = reinterpret_cast<uintptr_t>(i);
            if (p < q + n && q < p + n) return true;
        }
        if (p < act + n / 8 && act < p + n) return true;
    }
    return false;
}

// The float64 form of a BEM geometry in two launches: the field of all
// particles at once into ax, ay, az -- one point a warp or a point split over
// several, whatever fills the SMs, where one CTA per group leaves them idle
// for few groups and waits for its slowest point for many -- then the groups'
// pair sums.  Either far rule: only the first launch depends on it.  Every
// particle of the groups gets its field whatever a caller left in n_particles.
template <int KIND>
int accel_launch_split(const SptAccelArgs* a, const SptGeometry* g, const SptBem& bem, cudaStream_t stream) {
    const FieldMask mask{a->active, a->group_offset, a->n_groups, *g};
    const long long most = (long long)a->n_groups * a->max_group_size;
    const long long n = a->n_particles > 0 && a->n_particles < most ? a->n_particles : most;
    const int e = launch_field(a->x, a->y, a->z, n, most, bem, mask, a->ax, a->ay, a->az, stream);
    if (e == -1) return (int)cudaErrorInvalidValue;
    if (e) return e;
    return accel_launch<KIND, SPT_FORM_FP64, SPT_FAR_REFERENCE, true>(a, g, bem, stream);
}

// Trace dispatch over the (form, far rule) instantiations of one geometry
// kind: with launch false, only the shared memory, grid and occupancy of the
// launch t describes; with launch true, also the launch on that grid.
// Returns 0, a cudaError_t, or -1 for a (form, far rule) this kind does not
// offer.  Defined here, instantiated once per kind in spt_trace_<kind>.cu.
template <int KIND>
int trace_dispatch(const TraceLaunch& t, int form, int far, bool launch, int* grid, size_t* smem, int* per_sm) {
    constexpr bool kBem = KIND == SPT_GEOM_TIP_BEM || KIND == SPT_GEOM_WELL_BEM || KIND == SPT_GEOM_POST_BEM;
    const int n = t.s->n_groups, E = t.s->max_group_size;
    const int img = image_scratch(*t.g, t.bem, E, t.threads);
#define SPT_TRACE_CASE(F, R)                                                                            \
    {                                                                                                   \
        int rc = trace_grid<KIND, F, R>(E, t.threads, n, t.max_slots, img, smem, grid, per_sm);         \
        if (rc || !launch) return rc;                                                                   \
        return trace_launch<KIND, F, R>(t, *grid, *smem);                                               \
    }
    if constexpr (kBem) {
        if (t.warp_team) {
            if (form != SPT_FORM_FP64 || far != SPT_FAR_ADAPTIVE || E > 32 || img > 0) return -1;
            int rc = trace_warp_grid<KIND, SPT_FORM_FP64>(t.threads, n, t.max_slots, smem, grid, per_sm);
            if (rc || !launch) return rc;
            return trace_warp_launch<KIND, SPT_FORM_FP64>(t, *grid, *smem);
        }
        if (form == SPT_FORM_FP64 && far == SPT_FAR_REFERENCE) SPT_TRACE_CASE(SPT_FORM_FP64, SPT_FAR_REFERENCE)
        if (form == SPT_FORM_FP64 && far == SPT_FAR_ADAPTIVE) SPT_TRACE_CASE(SPT_FORM_FP64, SPT_FAR_ADAPTIVE)
        if (form == SPT_FORM_MIXED && far == SPT_FAR_REFERENCE) SPT_TRACE_CASE(SPT_FORM_MIXED, SPT_FAR_REFERENCE)
        if (form == SPT_FORM_MIXED && far == SPT_FAR_ADAPTIVE) SPT_TRACE_CASE(SPT_FORM_MIXED, SPT_FAR_ADAPTIVE)
        if (form == SPT_FORM_SURROGATE && far == SPT_FAR_REFERENCE) SPT_TRACE_CASE(SPT_FORM_SURROGATE, SPT_FAR_REFERENCE)
        if (form == SPT_FORM_SURROGATE && far == SPT_FAR_ADAPTIVE) SPT_TRACE_CASE(SPT_FORM_SURROGATE, SPT_FAR_ADAPTIVE)
    } else {
        // no BEM field: the far rule plays no part
        if (t.warp_team) return -1;
        if (form == SPT_FORM_FP64) SPT_TRACE_CASE(SPT_FORM_FP64, SPT_FAR_REFERENCE)
        if (form == SPT_FORM_MIXED) SPT_TRACE_CASE(SPT_FORM_MIXED, SPT_FAR_REFERENCE)
    }
#undef SPT_TRACE_CASE
    return -1;
}

// spt_accel dispatch, as trace_dispatch (forms FP64 and MIXED).
template <int KIND>
int accel_dispatch(const SptAccelArgs* a, const SptGeometry* g, const SptBem& bem, cudaStream_t stream) {
    constexpr bool kBem = KIND == SPT_GEOM_TIP_BEM || KIND == SPT_GEOM_WELL_BEM || KIND == SPT_GEOM_POST_BEM;
    const int far = kBem ? bem.far_rule : SPT_FAR_REFERENCE;
    if constexpr (kBem) {
        if (a->form == SPT_FORM_FP64 && !accel_in_place(a)) return accel_launch_split<KIND>(a, g, bem, stream);
        if (a->form == SPT_FORM_FP64 && far == SPT_FAR_REFERENCE)
            return accel_launch<KIND, SPT_FORM_FP64, SPT_FAR_REFERENCE>(a, g, bem, stream);
        if (a->form == SPT_FORM_FP64 && far == SPT_FAR_ADAPTIVE)
            return accel_launch<KIND, SPT_FORM_FP64, SPT_FAR_ADAPTIVE>(a, g, bem, stream);
        if (a->form == SPT_FORM_MIXED && far == SPT_FAR_REFERENCE)
            return accel_launch<KIND, SPT_FORM_MIXED, SPT_FAR_REFERENCE>(a, g, bem, stream);
        if (a->form == SPT_FORM_MIXED && far == SPT_FAR_ADAPTIVE)
            return accel_launch<KIND, SPT_FORM_MIXED, SPT_FAR_ADAPTIVE>(a, g, bem, stream);
    } else {
        if (a->form == SPT_FORM_FP64) return accel_launch<KIND, SPT_FORM_FP64, SPT_FAR_REFERENCE>(a, g, bem, stream);
        if (a->form == SPT_FORM_MIXED) return accel_launch<KIND, SPT_FORM_MIXED, SPT_FAR_REFERENCE>(a, g, bem, stream);
    }
    return -1;
}

#define SPT_DECLARE_KIND(KIND)                                                                                  \
    extern template int trace_dispatch<KIND>(const TraceLaunch&, int, int, bool, int*, size_t*, int*);         \
    extern template int accel_dispatch<KIND>(const SptAccelArgs*, const SptGeometry*, const SptBem&, cudaStream_t);
#define SPT_INSTANTIATE_KIND(KIND)                                                                              \
    template int trace_dispatch<KIND>(const TraceLaunch&, int, int, bool, int*, size_t*, int*);                \
    template int accel_dispatch<KIND>(const SptAccelArgs*, const SptGeometry*, const SptBem&, cudaStream_t);

}  // namespace spt
