// pf_slab.cu -- x-slab decomposition of the periodic box over ranks: the
// distributed form of solver_bicgstab.solve (src/solver/pressure.py:196-297)
// and the slab helpers around it.  Replaces the reference's decomposition
// and ghost exchange (decomp, communicate_border,
// src/library/parallel.py:118-414) and its scalar reductions (comms.parallel_sum
// / parallel_max, src/library/parallel.py:60-94) for grids split along x.
//
// A rank holds planes [x0, x0 + nxl) of the global box as a LOCAL EXTENDED
// grid of nxl + 2h planes, [nx][ny][nz] with z fastest like every field of
// this library: h ghost planes, the interior, h ghost planes.  Planes are
// contiguous, so a halo exchange moves h * ny * nz doubles per side with no
// packing.  Kernels that do not reduce (the RK4 predictor, divergence,
// projection) run unchanged on the extended grid: an interior plane depends
// on planes at most one away per stencil, so after an exchange of h planes
// the whole four-stage predictor is exact on the interior (h >= 4); what they
// write on ghost planes is overwritten by the next exchange.
//
// The solve follows the reference's iteration literally -- three global
// reductions per iteration (rho1 = (res, res0); gamma = (vv, res0); (s,t) and
// (t,t)), then max|res| for the stop test -- with every per-element operation
// of the reference (torch's add_(alpha, x) as one fused multiply-add).  Each
// reduction point is: a kernel writes this rank's sums over its interior into
// `send`; the caller gathers every rank's `send` into `recv` (rank order);
// the next phase folds `recv` in rank order on one thread, so every rank
// computes bitwise the same scalars and takes the same branch.  Scalars never
// leave the device; the caller polls the stop flag (pf_slab_bicg_info).
//
// Phases (the caller's loop, one rank):
//   init -> gather -> START;
//   repeat: exchange(pp, 1) -> APPLY_P -> gather -> S -> exchange(s, 1) ->
//           APPLY_S -> gather -> FINAL -> gather -> P (folds the stop test)
// until the stop flag is set; then p += DP (pf_slab_add) and, after an
// exchange of DP, the projection.
#include <algorithm>
#include <cmath>

#include "pf_common.cuh"
#include "pf_gridbar.cuh"
#include "pf_kernels.cuh"
#include "pf_profile.cuh"
#include "pf_sweep.cuh"

namespace pf {
namespace {

struct SlabScalars {
    double rho1, rho2, alpha, omega, max_res0, max_res, min_res;
    int iter, max_it, done, status;
    unsigned int counter;
};

constexpr int kSlabVals = 2;      // values per rank in `send`
constexpr int kSlabMaxRanks = 4096;

struct Slab {
    Dims d;          // the extended local grid
    int h;           // ghost planes per side
    long long off;   // first interior cell: h * ny * nz
    long long nint;  // interior cells: (nx - 2h) * ny * nz
};

struct SlabVecs {
    double *res, *res0, *pp, *vv, *s, *t;
};

struct SlabWs {
    SlabScalars* sc;
    double* part;  // kSlabVals x kMaxPartials block partials
    SlabVecs v;
};

Slab make_slab(const pf_grid* g, int h) {
    Slab s;
    s.d = Dims{g->nx, g->ny, g->nz, (long long)g->nx * g->ny * g->nz};
    s.h = h;
    s.off = (long long)h * g->ny * g->nz;
    s.nint = (long long)(g->nx - 2 * h) * g->ny * g->nz;
    return s;
}

size_t slab_ws_bytes(const pf_grid* g) {
    const size_t n = (size_t)g->nx * g->ny * g->nz;
    return align256(sizeof(SlabScalars)) + align256(kSlabVals * kMaxPartials * sizeof(double)) +
           6 * align256(n * sizeof(double));
}

SlabWs carve_slab(const pf_grid* g, void* ws) {
    const size_t n = (size_t)g->nx * g->ny * g->nz;
    char* p = (char*)ws;
    SlabWs w;
    w.sc = (SlabScalars*)p;
    p += align256(sizeof(SlabScalars));
    w.part = (double*)p;
    p += align256(kSlabVals * kMaxPartials * sizeof(double));
    double** vs[6] = {&w.v.res, &w.v.res0, &w.v.pp, &w.v.vv, &w.v.s, &w.v.t};
    for (double** q : vs) {
        *q = (double*)p;
        p += align256(n * sizeof(double));
    }
    return w;
}

int pointwise_blocks(long long n) {
    const long long b = (n + kBlock * 4 - 1) / (kBlock * 4);
    return (int)std::max<long long>(1, std::min<long long>(b, std::min(num_sms() * 8, kMaxPartials)));
}

__device__ __forceinline__ bool slab_last(SlabScalars* sc) {
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (tid0()) last = atomicAdd(&sc->counter, 1u) == gridDim.x - 1;
    __syncthreads();
    if (last) __threadfence();
    return last;
}

// the last block sums (or maxes) the partials in block order and writes send[slot]
template <bool MAX>
__device__ double finish_blocks(const double* part, int nblocks, double* sh) {
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    double v = 0.0;
    for (int b = tid; b < nblocks; b += kBlock) {
        const double x = ((volatile const double*)part)[b];
        v = MAX ? nanmax(v, x) : v + x;
    }
    return MAX ? block_max<kBlock>(v, sh) : block_sum<kBlock>(v, sh);
}

// ------------------------------------------------------------------ init
// res = res0 = (div * rho/dt) * (-vol) on the interior (the reference's
// source_P *= rho/dt; source_P *= -vol; src/solver/pressure.py:205-212);
// DP, pp, vv, s, t = 0 on every plane.  send = [(res, res0), max|res|].
__global__ void __launch_bounds__(kBlock)
slab_init(Slab sl, SlabWs w, const double* __restrict__ div, double c1, double c2,
          double* __restrict__ DP, double* __restrict__ send, double min_res, int max_it) {
    __shared__ double sh[32];
    double s = 0.0, m = 0.0;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < sl.d.n; q += stride) {
        DP[q] = 0.0;
        w.v.pp[q] = 0.0;
        w.v.vv[q] = 0.0;
        w.v.s[q] = 0.0;
        w.v.t[q] = 0.0;
        double r = 0.0;
        if (q >= sl.off && q < sl.off + sl.nint) {
            r = (div[q] * c1) * c2;
            s += r * r;
            m = nanmax(m, fabs(r));
        }
        w.v.res[q] = r;
        w.v.res0[q] = r;
    }
    const double bs = block_sum<kBlock>(s, sh);
    const double bm = block_max<kBlock>(m, sh);
    if (tid0()) { w.part[blockIdx.x] = bs; w.part[kMaxPartials + blockIdx.x] = bm; }
    if (slab_last(w.sc)) {
        const double tot = finish_blocks<false>(w.part, gridDim.x, sh);
        const double mx = finish_blocks<true>(w.part + kMaxPartials, gridDim.x, sh);
        if (tid0()) {
            send[0] = tot;
            send[1] = mx;
            SlabScalars* sc = w.sc;
            sc->rho1 = 1.0; sc->rho2 = 1.0; sc->alpha = 0.0; sc->omega = 1.0;
            sc->max_res0 = 0.0; sc->max_res = 0.0; sc->min_res = min_res;
            sc->iter = 0; sc->max_it = max_it; sc->done = 0; sc->status = PF_OK;
            sc->counter = 0u;
        }
    }
}

// ------------------------------------------------------------------ folds
// One thread folds the gathered values of every rank in rank order.
enum { kFoldStart = 0, kFoldNext = 1, kFoldGamma = 2, kFoldOmega = 3 };

__global__ void slab_fold(SlabScalars* sc, const double* __restrict__ recv, int world, int mode) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    if (mode != kFoldStart && sc->done) return;
    double a = 0.0, b = 0.0;
    for (int r = 0; r < world; ++r) {
        a += recv[r * kSlabVals];
        b = (mode == kFoldOmega) ? b + recv[r * kSlabVals + 1] : nanmax(b, recv[r * kSlabVals + 1]);
    }
    if (mode == kFoldStart) {
        // max_res0 (src/solver/pressure.py:213) and rho1 of iteration 1
        sc->max_res0 = b;
        sc->rho1 = a;
    } else if (mode == kFoldNext) {
        // end of an iteration (src/solver/pressure.py:276-289): rho2 = rho1,
        // the stop test on max|res| / max_res0, then rho1 of the next one
        sc->rho2 = sc->rho1;
        sc->rho1 = a;
        const double mr = b / sc->max_res0;
        sc->max_res = mr;
        sc->iter += 1;
        if (!(mr == mr)) { sc->done = 1; sc->status = PF_NONFINITE; }
        else if (mr <= sc->min_res) { sc->done = 1; sc->status = PF_OK; }
        else if (sc->iter >= sc->max_it) { sc->done = 1; sc->status = PF_MAXIT; }
    } else if (mode == kFoldGamma) {
        // gamma = (vv, res0); gamma == 0 leaves the loop before DP changes
        if (a == 0.0) { sc->done = 1; sc->status = PF_BREAKDOWN; }
        else sc->alpha = sc->rho1 / a;
    } else {
        // omega = (s, t) / (t, t); (t, t) == 0 leaves after DP += alpha pp
        if (b == 0.0) { sc->done = 1; sc->status = PF_BREAKDOWN; }
        else sc->omega = a / b;
    }
}

// ------------------------------------------------------------------ pointwise
// pp = (pp - omega vv) beta + res, beta = alpha rho1 / (rho2 omega)
// (src/solver/pressure.py:229-234)
__global__ void __launch_bounds__(kBlock)
slab_pupdate(Slab sl, SlabWs w) {
    const SlabScalars* sc = w.sc;
    if (sc->done) return;
    const double omega = sc->omega;
    const double beta = sc->alpha * sc->rho1 / (sc->rho2 * omega);
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long q = sl.off + blockIdx.x * (long long)blockDim.x + threadIdx.x;
         q < sl.off + sl.nint; q += stride) {
        double p = fma(-omega, w.v.vv[q], w.v.pp[q]);
        p = p * beta;
        w.v.pp[q] = p + w.v.res[q];
    }
}

// DP += alpha pp; s = res - alpha vv (src/solver/pressure.py:250-255)
__global__ void __launch_bounds__(kBlock)
slab_supdate(Slab sl, SlabWs w, double* __restrict__ DP) {
    const SlabScalars* sc = w.sc;
    if (sc->done) return;
    const double alpha = sc->alpha;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long q = sl.off + blockIdx.x * (long long)blockDim.x + threadIdx.x;
         q < sl.off + sl.nint; q += stride) {
        DP[q] = fma(alpha, w.v.pp[q], DP[q]);
        w.v.s[q] = fma(-alpha, w.v.vv[q], w.v.res[q]);
    }
}

// DP += omega s; res = s - omega t; send = [(res, res0), max|res|]
// (src/solver/pressure.py:269-283)
__global__ void __launch_bounds__(kBlock)
slab_final(Slab sl, SlabWs w, double* __restrict__ DP, double* __restrict__ send) {
    __shared__ double sh[32];
    SlabScalars* sc = w.sc;
    if (sc->done) return;
    const double omega = sc->omega;
    double s = 0.0, m = 0.0;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long q = sl.off + blockIdx.x * (long long)blockDim.x + threadIdx.x;
         q < sl.off + sl.nint; q += stride) {
        const double sv = w.v.s[q];
        DP[q] = fma(omega, sv, DP[q]);
        const double r = fma(-omega, w.v.t[q], sv);
        w.v.res[q] = r;
        s += r * w.v.res0[q];
        m = nanmax(m, fabs(r));
    }
    const double bs = block_sum<kBlock>(s, sh);
    const double bm = block_max<kBlock>(m, sh);
    if (tid0()) { w.part[blockIdx.x] = bs; w.part[kMaxPartials + blockIdx.x] = bm; }
    if (slab_last(sc)) {
        const double tot = finish_blocks<false>(w.part, gridDim.x, sh);
        const double mx = finish_blocks<true>(w.part + kMaxPartials, gridDim.x, sh);
        if (tid0()) { send[0] = tot; send[1] = mx; sc->counter = 0u; }
    }
}

// ------------------------------------------------------------------ operator
// out = A in on the interior (Pressure_Base.applyOperator,
// src/solver/pressure.py:54-84, the terms in the order of laplace_kernel):
// x neighbours from the planes beside the interior (ghost planes at its
// ends), y and z wrap.  APPLY_P: vv = A pp, send = [(vv, res0), 0];
// APPLY_S: t = A s, send = [(s, t), (t, t)].  A block of 32 x 8 threads walks
// 32 (z) x 8 (y) tiles of the interior planes, tile index += grid size.
template <bool S_PHASE>
__global__ void __launch_bounds__(kBlock)
slab_apply(Slab sl, SlabWs w, LapCoef<double> cf, double* __restrict__ send) {
    __shared__ double sh[32];
    SlabScalars* sc = w.sc;
    if (sc->done) return;
    const Dims d = sl.d;
    const double* A = S_PHASE ? w.v.s : w.v.pp;
    double* B = S_PHASE ? w.v.t : w.v.vv;
    const int tz = (d.nz + 31) / 32, ty = (d.ny + 7) / 8;
    const long long ntiles = (long long)tz * ty * (d.nx - 2 * sl.h);
    double s1 = 0.0, s2 = 0.0;
    for (long long t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const int k = (int)(t % tz) * 32 + threadIdx.x;
        const int j = (int)((t / tz) % ty) * 8 + threadIdx.y;
        const int i = sl.h + (int)(t / ((long long)tz * ty));
        if (k >= d.nz || j >= d.ny) continue;
        const long long q = idx(d, i, j, k);
        const double c = A[q];
        double b = 0.0;
        b += A[idx(d, i - 1, j, k)] * cf.c[0][0];
        b += c * cf.c[0][1];
        b += A[idx(d, i + 1, j, k)] * cf.c[0][2];
        b += A[idx(d, i, wrap(j - 1, d.ny), k)] * cf.c[1][0];
        b += c * cf.c[1][1];
        b += A[idx(d, i, wrap(j + 1, d.ny), k)] * cf.c[1][2];
        b += A[idx(d, i, j, wrap(k - 1, d.nz))] * cf.c[2][0];
        b += c * cf.c[2][1];
        b += A[idx(d, i, j, wrap(k + 1, d.nz))] * cf.c[2][2];
        B[q] = b;
        if (S_PHASE) { s1 += c * b; s2 += b * b; }
        else s1 += b * w.v.res0[q];
    }
    const double b1 = block_sum<kBlock>(s1, sh);
    const double b2 = S_PHASE ? block_sum<kBlock>(s2, sh) : 0.0;
    if (tid0()) { w.part[blockIdx.x] = b1; w.part[kMaxPartials + blockIdx.x] = b2; }
    if (slab_last(sc)) {
        const double t1 = finish_blocks<false>(w.part, gridDim.x, sh);
        const double t2 = S_PHASE ? finish_blocks<false>(w.part + kMaxPartials, gridDim.x, sh) : 0.0;
        if (tid0()) { send[0] = t1; send[1] = t2; sc->counter = 0u; }
    }
}

// p += DP on the interior (src/solver/pressure.py:293-294)
__global__ void __launch_bounds__(kBlock)
slab_add(Slab sl, const double* __restrict__ DP, double* __restrict__ p) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long q = sl.off + blockIdx.x * (long long)blockDim.x + threadIdx.x;
         q < sl.off + sl.nint; q += stride)
        p[q] = p[q] + DP[q];
}

__global__ void slab_info(const SlabScalars* sc, double* out) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    out[0] = sc->max_res;
    out[1] = (double)sc->iter;
    out[2] = (double)sc->status;
    out[3] = (double)sc->done;
}

// blocks of the apply kernel: every SM busy, at most kMaxPartials
int apply_blocks(const Slab& sl) {
    const long long nt = (long long)((sl.d.nz + 31) / 32) * ((sl.d.ny + 7) / 8) * (sl.d.nx - 2 * sl.h);
    return (int)std::max<long long>(1, std::min<long long>(nt, std::min(num_sms() * 8, kMaxPartials)));
}


// --------------------------------------------------- all slabs in one process
// The whole solve of R slabs held by one process as one cooperative launch
// (per kGroupIters iterations).  Driven from the host, an iteration is 16
// launches and copies per slab.  Per iteration, phases -> this kernel, on one
// B200: two slabs of 48x64x64 270 -> 28.7 us, three of 16x40x40 383 -> 19.4,
// two of 64x128x128 277 -> 97, two of 128x256x256 835 -> 759.  What is left at
// the small sizes is latency: each grid barrier with its fold takes 3.5 us,
// and after it every load goes to L2.  An iteration is three phases separated
// by grid barriers:
//   P1  pp' = (pp - omega vv) beta + res at the seven points, vv' = A pp',
//       (vv', res0)
//   P2  s = res - alpha vv' at the seven points, t = A s, (s,t), (t,t)
//       (and DP += alpha pp' while the barrier behind it is under way)
//   P3  DP += omega s, res = s - omega t, (res,res0), max|res|
// The x neighbours of a slab's end planes are read where they lie, in the
// next slab, so nothing is exchanged; pp and vv alternate between two buffers
// each (the phase kernels' s and the just-consumed t are the second ones).
// Every element's operations, and every sum -- per virtual block of the phase
// kernels' grids, then blocks in block order, then slabs in rank order, which
// each physical block folds for itself -- are those of the phase kernels, so
// the solve is bitwise the one the phases give.
constexpr int kGroupMax = 24;     // slabs of one launch (its arguments are passed by value)
constexpr int kGroupIters = 256;  // iterations per launch
constexpr int kGroupParts = kSlabVals * kMaxPartials / 5;  // partial slots per sum and slab

struct GroupSlab {
    int nxl, ab, nb;  // interior planes; virtual blocks of the operator and the pointwise phases
    double *res, *res0, *pp[2], *vv[2], *DP, *part;
    const double* send;
    SlabScalars* sc;
};

struct Group {
    int R, h, ny, nz;
    int nab, nnb;  // virtual blocks over all slabs
    int one;       // every virtual block of the operator is one tile
    LapCoef<double> cf;
    unsigned* bar;
    GroupSlab s[kGroupMax];
};

// A physical block is four groups of 256 threads, each working through
// virtual blocks on its own (named barriers 1-4); the grid barrier then has
// 148 arrivals instead of 592.
constexpr int kGroups = 4;

__device__ __forceinline__ void group_sync(int grp) {
    asm volatile("bar.sync %0, 256;" ::"r"(grp + 1) : "memory");
}

// Sums (or, second value with MAX2, maxima) of U pairs of values over the
// group, in the order of block_sum / block_max; pair u valid in lane 0 of the
// group's warp u.
template <int U, bool TWO, bool MAX2>
__device__ __forceinline__ void group_pairs(double* a, double* b, double* sh, int grp) {
    const int t = threadIdx.x & 255, lane = t & 31, wid = t >> 5;
    auto add2 = [](double x, double y) { return MAX2 ? nanmax(x, y) : x + y; };
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int u = 0; u < U; ++u) {
            a[u] += __shfl_down_sync(0xffffffffu, a[u], o);
            if (TWO) b[u] = add2(b[u], __shfl_down_sync(0xffffffffu, b[u], o));
        }
    if (lane == 0)
#pragma unroll
        for (int u = 0; u < U; ++u) {
            sh[u * 16 + wid] = a[u];
            if (TWO) sh[u * 16 + 8 + wid] = b[u];
        }
    group_sync(grp);
    if (wid < U) {
        double x = lane < 8 ? sh[wid * 16 + lane] : 0.0;
        double y = TWO && lane < 8 ? sh[wid * 16 + 8 + lane] : 0.0;
        for (int o = 16; o > 0; o >>= 1) {
            x += __shfl_down_sync(0xffffffffu, x, o);
            if (TWO) y = add2(y, __shfl_down_sync(0xffffffffu, y, o));
        }
        a[0] = x;
        if (TWO) b[0] = y;
    }
    group_sync(grp);
}

// The partials of every slab folded in rank order, by every block for itself;
// the result in thread 0.  which: the first of the sum's two slots.  The
// groups take one value of one slab each (all in one group, one after another,
// the folds took longer than the barriers).
template <bool TWO, bool MAX2>
__device__ __forceinline__ void group_fold(const Group& G, int which, bool apply, double* sh,
                                           double& A, double& B) {
    const int grp = threadIdx.x >> 8, t = threadIdx.x & 255, lane = t & 31, wid = t >> 5;
    double* ws = sh + grp * 8;       // this group's warp sums
    double* val = sh + 8 * kGroups;  // the values, slab by slab
    const int n = G.R * (TWO ? 2 : 1);
    for (int c = grp; c < n; c += kGroups) {
        const int r = TWO ? c >> 1 : c, second = TWO ? c & 1 : 0;
        const bool mx = MAX2 && second;
        const int nv = apply ? G.s[r].ab : G.s[r].nb;
        const double* pa = G.s[r].part + (which + second) * kGroupParts;
        double x = 0.0;
#pragma unroll 4
        for (int q = t; q < nv; q += 256) {
            const double y = __ldcg(pa + q);
            x = mx ? nanmax(x, y) : x + y;
        }
        for (int o = 16; o > 0; o >>= 1) {
            const double y = __shfl_down_sync(0xffffffffu, x, o);
            x = mx ? nanmax(x, y) : x + y;
        }
        if (lane == 0) ws[wid] = x;
        group_sync(grp);
        if (wid == 0) {
            x = lane < 8 ? ws[lane] : 0.0;
            for (int o = 16; o > 0; o >>= 1) {
                const double y = __shfl_down_sync(0xffffffffu, x, o);
                x = mx ? nanmax(x, y) : x + y;
            }
            if (lane == 0) val[c] = x;
        }
        group_sync(grp);
    }
    __syncthreads();
    A = B = 0.0;
    if (threadIdx.x == 0)
        for (int r = 0; r < G.R; ++r) {
            A += val[TWO ? 2 * r : r];
            if (TWO) B = MAX2 ? nanmax(B, val[2 * r + 1]) : B + val[2 * r + 1];
        }
}

// A x at (j, k) of plane i of slab s: `at(slab, offset)` is the operand.
template <class At>
__device__ __forceinline__ double group_stencil(const Group& G, const GroupSlab& s,
                                                const GroupSlab& sl, const GroupSlab& sr, int i,
                                                int j, int k, At at, double& ctr) {
    const int ny = G.ny, nz = G.nz, h = G.h;
    const int plane = ny * nz, p = (h + i) * plane, c = j * nz + k;
    ctr = at(s, p + c);
    // (the slab is chosen before the loads: in a branch of its own each
    // operand would be waited for before the next is asked for)
    const GroupSlab& bm = i ? s : sl;
    const GroupSlab& bp = i + 1 < s.nxl ? s : sr;
    const double xm = at(bm, (i ? p - plane : (h + sl.nxl - 1) * plane) + c);
    const double xp = at(bp, (i + 1 < s.nxl ? p + plane : h * plane) + c);
    const double ym = at(s, p + wrap(j - 1, ny) * nz + k);
    const double yp = at(s, p + wrap(j + 1, ny) * nz + k);
    const double zm = at(s, p + j * nz + wrap(k - 1, nz));
    const double zp = at(s, p + j * nz + wrap(k + 1, nz));
    double o = 0.0;
    o += xm * G.cf.c[0][0];
    o += ctr * G.cf.c[0][1];
    o += xp * G.cf.c[0][2];
    o += ym * G.cf.c[1][0];
    o += ctr * G.cf.c[1][1];
    o += yp * G.cf.c[1][2];
    o += zm * G.cf.c[2][0];
    o += ctr * G.cf.c[2][1];
    o += zp * G.cf.c[2][2];
    return o;
}

// One operator phase: the operand is `at(slab, q)`; `put(slab, q, centre,
// A operand, sum a, sum b)` consumes a cell.  A block takes a run of virtual
// blocks; where each is one tile (up to 1184 tiles per slab) the run goes
// through the planes of a tile column, so its groups work on neighbouring
// planes and find each other's operands in the SM's L1.
template <bool TWO, class At, class Put>
__device__ __forceinline__ void group_apply(const Group& G, int which, double* sh, At at, Put put) {
    const int grp = threadIdx.x >> 8, wid = (threadIdx.x & 255) >> 5, tx = threadIdx.x & 31;
    const int tz = (G.nz + 31) / 32, ty = (G.ny + 7) / 8, plane = G.ny * G.nz;
    const int per = (G.nab + gridDim.x - 1) / gridDim.x;
    const int end = min(G.nab, (int)(blockIdx.x + 1) * per);
    for (int v = blockIdx.x * per + grp; v < end; v += kGroups) {
        int r = 0, vb = v;
        while (vb >= G.s[r].ab) vb -= G.s[r++].ab;
        const GroupSlab& s = G.s[r];
        const GroupSlab& sl = G.s[r ? r - 1 : G.R - 1];
        const GroupSlab& sr = G.s[r + 1 < G.R ? r + 1 : 0];
        if (G.one) {
            const int col = vb / s.nxl;
            vb = (vb - col * s.nxl) * (tz * ty) + col;
        }
        double a = 0.0, b = 0.0;
        const int ntiles = tz * ty * s.nxl;
        for (int t = vb; t < ntiles; t += s.ab) {
            const int t1 = t / tz, i = t1 / ty;
            const int k = (t - t1 * tz) * 32 + tx, j = (t1 - i * ty) * 8 + wid;
            if (k >= G.nz || j >= G.ny) continue;
            double c;
            const double o = group_stencil(G, s, sl, sr, i, j, k, at, c);
            put(s, (G.h + i) * plane + j * G.nz + k, c, o, a, b);
        }
        group_pairs<1, TWO, false>(&a, &b, sh + 80 + grp * 16, grp);
        if ((threadIdx.x & 255) == 0) {
            s.part[which * kGroupParts + vb] = a;
            if (TWO) s.part[(which + 1) * kGroupParts + vb] = b;
        }
    }
}

__global__ void __launch_bounds__(kBlock * kGroups, 1)
slab_group_solve(const __grid_constant__ Group G, int first) {
    __shared__ double sh[80 + kGroups * 16];  // folds: 32 warp sums, 48 values; then the pairs
    // the scalars of the solve, kept (the same) by every block in shared memory
    __shared__ SlabScalars S;
    const int grp = threadIdx.x >> 8, tid = threadIdx.x & 255;
    unsigned round = 0;
    if (threadIdx.x == 0) {
        S = *G.s[0].sc;
        if (first) {
            // max_res0 (src/solver/pressure.py:213) and rho1 of iteration 1
            double a = 0.0, b = 0.0;
            for (int r = 0; r < G.R; ++r) { a += G.s[r].send[0]; b = nanmax(b, G.s[r].send[1]); }
            S.rho1 = a;
            S.max_res0 = b;
        }
    }
    __syncthreads();
    const int plane = G.ny * G.nz;
    // pointwise phases: f(slab, virtual block, first cell, end, step) in the
    // phase kernels' distribution
    auto pointwise = [&](auto f) {
        for (int v = blockIdx.x + grp * gridDim.x; v < G.nnb; v += gridDim.x * kGroups) {
            int r = 0, vb = v;
            while (vb >= G.s[r].nb) vb -= G.s[r++].nb;
            const GroupSlab& s = G.s[r];
            f(s, vb, G.h * plane + vb * kBlock + tid, (G.h + s.nxl) * plane, s.nb * kBlock);
        }
    };
    constexpr int B = 2;  // cells loaded before any is stored
    double x0, x1;
    for (int it = 0; it < kGroupIters && !S.done; ++it) {
        const int o = S.iter & 1, n = o ^ 1;
        {
            const double omega = S.omega, beta = S.alpha * S.rho1 / (S.rho2 * omega);
            group_apply<false>(
                G, 0, sh,
                [&](const GroupSlab& s, int q) {
                    double p = fma(-omega, s.vv[o][q], s.pp[o][q]);
                    p = p * beta;
                    return p + s.res[q];
                },
                [&](const GroupSlab& s, int q, double c, double v, double& a, double&) {
                    s.pp[n][q] = c;
                    s.vv[n][q] = v;
                    a += v * s.res0[q];
                });
        }
        if (!grid_meet(G.bar, ++round)) return;
        group_fold<false, false>(G, 0, true, sh, x0, x1);
        if (threadIdx.x == 0) {
            // gamma == 0 leaves the loop before DP changes
            if (x0 == 0.0) { S.done = 1; S.status = PF_BREAKDOWN; }
            else S.alpha = S.rho1 / x0;
        }
        __syncthreads();
        if (S.done) break;
        const double alpha = S.alpha;
        group_apply<true>(
            G, 1, sh, [&](const GroupSlab& s, int q) { return fma(-alpha, s.vv[n][q], s.res[q]); },
            [&](const GroupSlab& s, int q, double c, double v, double& a, double& b) {
                s.vv[o][q] = v;  // t
                a += c * v;
                b += v * v;
            });
        grid_arrive(G.bar);
        // while the barrier is under way: DP += alpha pp', of cells that only
        // this thread touches (also where (t, t) == 0 ends the solve)
        pointwise([&](const GroupSlab& s, int, int q0, int end, int step) {
            for (; q0 < end; q0 += B * step) {
                double p[B], d[B];
#pragma unroll
                for (int m = 0; m < B; ++m) {
                    const int q = q0 + m * step;
                    if (q >= end) break;
                    p[m] = s.pp[n][q]; d[m] = s.DP[q];
                }
#pragma unroll
                for (int m = 0; m < B; ++m) {
                    const int q = q0 + m * step;
                    if (q >= end) break;
                    s.DP[q] = fma(alpha, p[m], d[m]);
                }
            }
        });
        if (!grid_wait(G.bar, ++round)) return;
        group_fold<true, false>(G, 1, true, sh, x0, x1);
        if (threadIdx.x == 0) {
            // (t, t) == 0 leaves after DP += alpha pp
            if (x1 == 0.0) { S.done = 1; S.status = PF_BREAKDOWN; }
            else S.omega = x0 / x1;
        }
        __syncthreads();
        if (S.done) break;
        const double omega = S.omega;
        pointwise([&](const GroupSlab& s, int vb, int q0, int end, int step) {
            double a = 0.0, b = 0.0;
            for (; q0 < end; q0 += B * step) {
                double d[B], vv[B], rs[B], t[B], r0[B];
#pragma unroll
                for (int m = 0; m < B; ++m) {
                    const int q = q0 + m * step;
                    if (q >= end) break;
                    vv[m] = s.vv[n][q]; rs[m] = s.res[q]; t[m] = s.vv[o][q];
                    r0[m] = s.res0[q]; d[m] = s.DP[q];
                }
#pragma unroll
                for (int m = 0; m < B; ++m) {
                    const int q = q0 + m * step;
                    if (q >= end) break;
                    const double sv = fma(-alpha, vv[m], rs[m]);
                    const double rn = fma(-omega, t[m], sv);
                    s.res[q] = rn;
                    s.DP[q] = fma(omega, sv, d[m]);
                    a += rn * r0[m];
                    b = nanmax(b, fabs(rn));
                }
            }
            group_pairs<1, true, true>(&a, &b, sh + 80 + grp * 16, grp);
            if (tid == 0) {
                s.part[3 * kGroupParts + vb] = a;
                s.part[4 * kGroupParts + vb] = b;
            }
        });
        if (!grid_meet(G.bar, ++round)) return;
        group_fold<true, true>(G, 3, false, sh, x0, x1);
        if (threadIdx.x == 0) {
            // end of the iteration (src/solver/pressure.py:276-289)
            S.rho2 = S.rho1;
            S.rho1 = x0;
            const double mr = x1 / S.max_res0;
            S.max_res = mr;
            S.iter += 1;
            if (!(mr == mr)) { S.done = 1; S.status = PF_NONFINITE; }
            else if (mr <= S.min_res) { S.done = 1; S.status = PF_OK; }
            else if (S.iter >= S.max_it) { S.done = 1; S.status = PF_MAXIT; }
        }
        __syncthreads();
    }
    // every block holds the same scalars, and none reads the stored ones after
    // the first barrier: one block writes them for every slab
    if (!grid_meet(G.bar, ++round)) return;
    if (blockIdx.x == 0 && threadIdx.x < G.R) *G.s[threadIdx.x].sc = S;
}

}  // namespace
}  // namespace pf

using namespace pf;

static bool slab_ok(const pf_grid* g, int halo) {
    return g && g->ny >= 2 && g->nz >= 2 && halo >= 1 && g->nx - 2 * halo >= 1 &&
           g->dx > 0 && g->dy > 0 && g->dz > 0;
}

static int rc_of(cudaError_t e) { return e == cudaSuccess ? PF_OK : PF_ERR_CUDA; }

extern "C" {

size_t pf_slab_workspace_bytes(const pf_grid* g) {
    if (!g || g->nx < 1 || g->ny < 1 || g->nz < 1) return 0;
    return slab_ws_bytes(g);
}

int pf_slab_bicg_vectors(const pf_grid* g, void* ws, double** pp, double** s) {
    if (!g || !ws || !pp || !s) return PF_ERR_BAD_ARG;
    const SlabWs w = carve_slab(g, ws);
    *pp = w.v.pp;
    *s = w.v.s;
    return PF_OK;
}

int pf_slab_bicg_init(const pf_grid* g, int halo, double rho, double dt, double min_res,
                      int max_it, const double* div, double* DP, void* ws, size_t ws_bytes,
                      double* send, void* stream) {
    if (!slab_ok(g, halo) || !div || !DP || !send || !ws || ((uintptr_t)ws & 255) ||
        ws_bytes < slab_ws_bytes(g) || !(rho != 0.0) || !(dt != 0.0) || max_it < 1)
        return PF_ERR_BAD_ARG;
    const Slab sl = make_slab(g, halo);
    const SlabWs w = carve_slab(g, ws);
    cudaStream_t s = (cudaStream_t)stream;
    if (cudaMemsetAsync(&w.sc->counter, 0, sizeof(unsigned int), s) != cudaSuccess)
        return PF_ERR_CUDA;
    const double vol = (g->dx * g->dy) * g->dz;
    PF_LAUNCH("slab_init", s, slab_init<<<pointwise_blocks(sl.d.n), kBlock, 0, s>>>(
        sl, w, div, rho / dt, -1.0 * vol, DP, send, min_res, max_it));
    return rc_of(cudaGetLastError());
}

int pf_slab_bicg_phase(const pf_grid* g, int halo, int phase, const double* recv, int world,
                       double* DP, void* ws, double* send, void* stream) {
    if (!slab_ok(g, halo) || !ws || ((uintptr_t)ws & 255) || phase < PF_SLAB_START ||
        phase > PF_SLAB_FINAL)
        return PF_ERR_BAD_ARG;
    const bool folds = phase == PF_SLAB_START || phase == PF_SLAB_NEXT || phase == PF_SLAB_S ||
                       phase == PF_SLAB_FINAL;
    if (folds && (!recv || world < 1 || world > kSlabMaxRanks)) return PF_ERR_BAD_ARG;
    if ((phase == PF_SLAB_S || phase == PF_SLAB_FINAL) && !DP) return PF_ERR_BAD_ARG;
    if ((phase == PF_SLAB_APPLY_P || phase == PF_SLAB_APPLY_S || phase == PF_SLAB_FINAL) && !send)
        return PF_ERR_BAD_ARG;
    const Slab sl = make_slab(g, halo);
    const SlabWs w = carve_slab(g, ws);
    cudaStream_t s = (cudaStream_t)stream;
    const int nb = pointwise_blocks(sl.nint);
    switch (phase) {
        case PF_SLAB_START:
        case PF_SLAB_NEXT:
            PF_LAUNCH("slab_fold", s, slab_fold<<<1, 32, 0, s>>>(
                w.sc, recv, world, phase == PF_SLAB_START ? kFoldStart : kFoldNext));
            PF_LAUNCH("slab_pupdate", s, slab_pupdate<<<nb, kBlock, 0, s>>>(sl, w));
            break;
        case PF_SLAB_APPLY_P:
        case PF_SLAB_APPLY_S: {
            const int ab = apply_blocks(sl);
            if (phase == PF_SLAB_APPLY_P)
                PF_LAUNCH("slab_apply_p", s, slab_apply<false><<<ab, dim3(32, 8), 0, s>>>(
                    sl, w, lap_coef<double>(g), send));
            else
                PF_LAUNCH("slab_apply_s", s, slab_apply<true><<<ab, dim3(32, 8), 0, s>>>(
                    sl, w, lap_coef<double>(g), send));
            break;
        }
        case PF_SLAB_S:
            PF_LAUNCH("slab_fold", s, slab_fold<<<1, 32, 0, s>>>(w.sc, recv, world, kFoldGamma));
            PF_LAUNCH("slab_supdate", s, slab_supdate<<<nb, kBlock, 0, s>>>(sl, w, DP));
            break;
        case PF_SLAB_FINAL:
            PF_LAUNCH("slab_fold", s, slab_fold<<<1, 32, 0, s>>>(w.sc, recv, world, kFoldOmega));
            PF_LAUNCH("slab_final", s, slab_final<<<nb, kBlock, 0, s>>>(sl, w, DP, send));
            break;
    }
    return rc_of(cudaGetLastError());
}

int pf_slab_local_solve(int count, const pf_grid* g, int halo, double rho, double dt,
                        double min_res, int max_it, const double* const* div, double* const* DP,
                        void* const* ws, const size_t* ws_bytes, double* const* send,
                        void* stream, pf_solve_info* info) {
    if (count < 1 || !g || !div || !DP || !ws || !ws_bytes || !send || !info) return PF_ERR_BAD_ARG;
    if (count > kGroupMax || prof_on()) return PF_ERR_TOO_LARGE;
    cudaStream_t st = (cudaStream_t)stream;
    Group G;
    G.R = count;
    G.h = halo;
    G.nab = G.nnb = 0;
    G.one = 1;
    for (int r = 0; r < count; ++r) {
        if (!slab_ok(&g[r], halo) || g[r].ny != g[0].ny || g[r].nz != g[0].nz || !ws[r] ||
            ((uintptr_t)ws[r] & 255) || ws_bytes[r] < slab_ws_bytes(&g[r]))
            return PF_ERR_BAD_ARG;
        const Slab sl = make_slab(&g[r], halo);
        const SlabWs w = carve_slab(&g[r], ws[r]);
        GroupSlab& q = G.s[r];
        q.nxl = g[r].nx - 2 * halo;
        q.ab = apply_blocks(sl);
        q.nb = pointwise_blocks(sl.nint);
        if (std::max(q.ab, q.nb) > kGroupParts || sl.d.n >= (1LL << 30)) return PF_ERR_TOO_LARGE;
        q.res = w.v.res; q.res0 = w.v.res0;
        q.pp[0] = w.v.pp; q.pp[1] = w.v.s;
        q.vv[0] = w.v.vv; q.vv[1] = w.v.t;
        q.DP = DP[r]; q.part = w.part; q.send = send[r]; q.sc = w.sc;
        if ((long long)((g[r].nz + 31) / 32) * ((g[r].ny + 7) / 8) * q.nxl != q.ab) G.one = 0;
        G.nab += q.ab;
        G.nnb += q.nb;
    }
    G.ny = g[0].ny; G.nz = g[0].nz;
    G.cf = lap_coef<double>(&g[0]);
    G.bar = (unsigned*)((char*)G.s[0].sc + 128);
    static_assert(sizeof(SlabScalars) <= 128, "the barrier words lie behind the scalars");
    int per = 0, coop = 0, dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, slab_group_solve, kBlock * kGroups, 0) != cudaSuccess)
        return PF_ERR_CUDA;
    if (!coop || per < 1) return PF_ERR_TOO_LARGE;
    for (int r = 0; r < count; ++r) {
        const int rc = pf_slab_bicg_init(&g[r], halo, rho, dt, min_res, max_it, div[r], DP[r], ws[r],
                                         ws_bytes[r], send[r], stream);
        if (rc) return rc;
    }
    const int nb = std::min(num_sms(), (std::max(G.nab, G.nnb) + kGroups - 1) / kGroups);
    struct { SlabScalars sc; char pad[128 - sizeof(SlabScalars)]; unsigned bar[kGridBarWords]; } hs;
    for (int first = 1;; first = 0) {
        if (cudaMemsetAsync(G.bar, 0, kGridBarWords * sizeof(unsigned), st) != cudaSuccess)
            return PF_ERR_CUDA;
        void* args[] = {&G, &first};
        if (cudaLaunchCooperativeKernel((const void*)slab_group_solve, dim3(nb), dim3(kBlock * kGroups), args, 0,
                                        st) != cudaSuccess ||
            cudaMemcpyAsync(&hs, G.s[0].sc, sizeof(hs), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
            cudaStreamSynchronize(st) != cudaSuccess)
            return PF_ERR_CUDA;
        if (hs.bar[1]) return PF_ERR_CUDA;  // a barrier gave up
        if (hs.sc.done) break;
    }
    info->max_res = hs.sc.max_res;
    info->iterations = hs.sc.iter;
    info->outer = 1;
    info->status = hs.sc.status;
    return PF_OK;
}

int pf_slab_bicg_info(const pf_grid* g, void* ws, double* out_dev, void* stream) {
    if (!g || !ws || !out_dev) return PF_ERR_BAD_ARG;
    const SlabWs w = carve_slab(g, ws);
    cudaStream_t s = (cudaStream_t)stream;
    slab_info<<<1, 32, 0, s>>>(w.sc, out_dev);
    return rc_of(cudaGetLastError());
}

int pf_slab_add(const pf_grid* g, int halo, const double* DP, double* p, void* stream) {
    if (!slab_ok(g, halo) || !DP || !p) return PF_ERR_BAD_ARG;
    const Slab sl = make_slab(g, halo);
    cudaStream_t s = (cudaStream_t)stream;
    PF_LAUNCH("slab_add", s, slab_add<<<pointwise_blocks(sl.nint), kBlock, 0, s>>>(sl, DP, p));
    return rc_of(cudaGetLastError());
}

}  // extern "C"
