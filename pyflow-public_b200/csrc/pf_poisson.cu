// pf_poisson.cu -- pressure Poisson solvers, divergence, projection, stats.
//
// BiCGStab (solver_bicgstab.solve, src/solver/pressure.py:196-297) with the
// operator of Pressure_Base.applyOperator (src/solver/pressure.py:54-84,
// coefficients metric_staggered.py:84-102) runs as TWO fused kernels per
// iteration, one per remaining global reduction:
//
//   kernel CA (iteration k): finish iteration k-1 and start iteration k
//     s   = res - alpha vv            (alpha, omega of iteration k-1)
//     res = s - omega t               (the reference's residual update)
//     DP += alpha pp + omega s        (two fused multiply-adds, same order)
//     pp  = (pp - omega vv) beta + res,  beta = alpha rho1 / (rho2 omega)
//     vv  = A pp,   gamma = (vv, res0),   max|res| -> stop test of k-1
//   kernel B (iteration k):
//     s = res - alpha vv,  t = A s,  (s,t), (t,t), (s,res0), (t,res0)
//     omega = (s,t)/(t,t);  rho1 of iteration k+1 = (s,res0) - omega (t,res0)
//
// Every per-element operation is the reference's (same operands, same fused
// multiply-adds: torch's add_(alpha, x) is one fma); only the scalar rho1 is
// formed from two dot products instead of (res, res0), which changes its
// rounding, not its value.  The reference needs three reductions and 17 field
// passes per iteration; this needs two and 14.
//
// Both kernels evaluate their stencil operand on the fly: a block owns a
// 32 (z) x 8R (y) tile, stages one x-plane of the operand plus its y/z halo in
// shared memory, and marches along x keeping the i-1, i, i+1 operand values of
// its own cells in registers.  The raw inputs of plane i+2 (and the halo of
// plane i+1) are loaded one iteration ahead so each thread keeps 15-30 loads
// in flight.  pp, vv and res, read at neighbours and rewritten by kernel CA,
// live in two buffer sets chosen by the parity of a device-side counter.
//
// All scalars stay in device memory; each reduction is finished by the last
// block to arrive (fixed summation order: bitwise reproducible), which also
// applies the reference's stop tests and sets a `done` flag that makes every
// later kernel of the solve return immediately.  The host only polls it.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "pf_common.cuh"
#include "pf_gridbar.cuh"
#include "pf_kernels.cuh"
#include "pf_sweep.cuh"
#include "pf_grad.cuh"
#include "pf_mg.cuh"
#include "pf_profile.cuh"
#include "pf_spectral.cuh"

namespace pf {


// Solver vectors.  set 0/1: res, pp, vv written by kernel CA of even/odd k.
template <typename T>
struct BicgVecs {
    T* res[2];
    T* pp[2];
    T* vv[2];
    T *t, *res0;
};

// ---------------------------------------------------------------- init
// FP64 path: res = res0 = (source * rho/dt) * (-vol); DP = pp = vv = 0.
// Mixed inner pass: res = res0 = T(r / scale) where r is the FP64 residual.
// Writes buffer set 1 (read by the first kernel CA).
template <typename T, bool FROM_RESIDUAL>
__global__ void __launch_bounds__(kBlock)
bicg_init(Dims d, BicgScalars* sc, double* part, const double* src, double c1,
          double c2, BicgVecs<T> v, T* x, int max_it, double min_res) {
    __shared__ double sh[32];
    double s = 0.0, m = 0.0;
    const double inv = (FROM_RESIDUAL && sc->scale > 0.0) ? 1.0 / sc->scale : 0.0;
    T* res = v.res[1];
    T* pp = v.pp[1];
    T* vv = v.vv[1];
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < d.n;
         q += (long long)gridDim.x * blockDim.x) {
        T r;
        if (FROM_RESIDUAL) r = T(src[q] * inv);
        else r = T((src[q] * c1) * c2);
        res[q] = r;
        v.res0[q] = r;
        x[q] = T(0); pp[q] = T(0); vv[q] = T(0); v.t[q] = T(0);
        s += double(r) * double(r);
        m = nanmax(m, fabs(double(r)));
    }
    const double bs = block_sum<kBlock>(s, sh);
    const double bm = block_max<kBlock>(m, sh);
    if (threadIdx.x == 0) { part[blockIdx.x] = bs; part[kMaxPartials + blockIdx.x] = bm; }
    if (arrive_last(sc)) {
        const double tot = finish<false>(part, sh);
        const double mx = finish<true>(part + kMaxPartials, sh);
        if (threadIdx.x == 0) {
            sc->rho1 = tot; sc->rho2 = 1.0; sc->alpha = 0.0; sc->omega = 1.0;
            sc->max_res0 = mx; sc->max_res = 0.0; sc->k = 0; sc->iter = 0;
            sc->done = 0; sc->status = PF_OK; sc->max_it = max_it;
            sc->min_res = min_res; sc->counter = 0u;
            // the words of the one-launch solve's grid barrier
            unsigned* bar = (unsigned*)((char*)sc + 192);
            bar[0] = bar[1] = 0u;
        }
    }
}

// ---------------------------------------------------------------- kernel CA
template <typename T>
struct PhaseCA {
    static constexpr int R = 2;
    const T *res_o, *pp_o, *vv_o, *t, *res0;
    T *x, *res_n, *pp_n, *vv_n;
    T alpha, omega, beta;
    bool fin;  // finish the previous iteration (k > 0)
    double gam, mx;
    struct Raw { T r, p, v, t; };
    struct Ext { T x, r0; };
    __device__ Raw raw(long long q, int = 0, int = 0, int = 0) const { return Raw{res_o[q], pp_o[q], vv_o[q], t[q]}; }
    __device__ Ext ext(long long q) const { return Ext{fin ? x[q] : T(0), res0[q]}; }
    __device__ T resid(const Raw& a) const {
        if (!fin) return a.r;
        const T s = fma(-alpha, a.v, a.r);  // s = res; s.sub_(alpha, vv)
        return fma(-omega, a.t, s);         // res = s; res.sub_(omega, t)
    }
    __device__ T op(const Raw& a) const {
        const T rn = resid(a);
        T q = fma(-omega, a.v, a.p);        // pp.sub_(omega, vv)
        q = q * beta;                       // pp.mul_(beta)
        return q + rn;                      // pp.add_(res)
    }
    __device__ void epi(long long q, T c, T b, const Raw& a, const Ext& e) {
        T rn = a.r;
        if (fin) {
            const T s = fma(-alpha, a.v, a.r);
            rn = fma(-omega, a.t, s);
            T xv = fma(alpha, a.p, e.x);    // DP.add_(alpha, pp)
            x[q] = fma(omega, s, xv);       // DP.add_(omega, s)
        }
        res_n[q] = rn;
        pp_n[q] = c;
        vv_n[q] = b;
        gam += double(b) * double(e.r0);
        mx = nanmax(mx, fabs(double(rn)));
    }
};

template <typename T>
__global__ void __launch_bounds__(kBlock, 2)
bicg_ca(Dims d, Tiling tl, LapCoef<T> cf, BicgScalars* sc, double* part,
        BicgVecs<T> v, T* __restrict__ x, int use_cond = 0,
        cudaGraphConditionalHandle cond = 0) {
    __shared__ double sh[32];
    const int done = sc->done;
    if (done == 1) {
        if (use_cond && blockIdx.x == 0 && tid0()) cudaGraphSetConditional(cond, 0);
        return;
    }
    const int k = sc->k;
    const bool odd = k & 1;  // CA(k) writes set k&1 and reads the other
    if (done == 2) {
        // (t,t) == 0 breakdown: the reference has applied DP += alpha pp and
        // stops (src/solver/pressure.py:251,266-267)
        const T alpha = T(sc->alpha);
        const T* pp = odd ? v.pp[0] : v.pp[1];
        const long long nt = (long long)gridDim.x * blockDim.x * blockDim.y;
        for (long long q = blockIdx.x * (long long)blockDim.x * blockDim.y +
                           threadIdx.y * blockDim.x + threadIdx.x;
             q < d.n; q += nt)
            x[q] = fma(alpha, pp[q], x[q]);
        if (arrive_last(sc) && tid0()) {
            sc->done = 1;
            sc->counter = 0u;
            if (use_cond) cudaGraphSetConditional(cond, 0);
        }
        return;
    }
    PhaseCA<T> ph;
    ph.res_o = odd ? v.res[0] : v.res[1];
    ph.pp_o = odd ? v.pp[0] : v.pp[1];
    ph.vv_o = odd ? v.vv[0] : v.vv[1];
    ph.t = v.t; ph.res0 = v.res0; ph.x = x;
    ph.res_n = odd ? v.res[1] : v.res[0];
    ph.pp_n = odd ? v.pp[1] : v.pp[0];
    ph.vv_n = odd ? v.vv[1] : v.vv[0];
    ph.alpha = T(sc->alpha);
    ph.omega = T(sc->omega);
    ph.beta = T((sc->alpha * sc->rho1) / (sc->rho2 * sc->omega));
    ph.fin = k > 0;
    ph.gam = 0.0; ph.mx = 0.0;
    sweep<T>(d, tl, cf, ph);
    const double bs = block_sum<kBlock>(ph.gam, sh);
    const double bm = block_max<kBlock>(ph.mx, sh);
    if (tid0()) { part[blockIdx.x] = bs; part[kMaxPartials + blockIdx.x] = bm; }
    if (arrive_last(sc)) {
        const double gamma = finish<false>(part, sh);
        const double mxr = finish<true>(part + kMaxPartials, sh);
        if (tid0()) {
            bool stop = false;
            if (k > 0) {
                // stop tests of iteration k (src/solver/pressure.py:279-287)
                sc->iter = k;
                const double mr = mxr / sc->max_res0;
                sc->max_res = mr;
                if (!(mr == mr) || isinf(mr)) { stop = true; sc->status = PF_NONFINITE; }
                else if (mr <= sc->min_res) { stop = true; sc->status = PF_OK; }
                else if (k >= sc->max_it) { stop = true; sc->status = PF_MAXIT; }
            }
            if (!stop) {
                sc->gamma = gamma;
                if (gamma == 0.0) { stop = true; sc->status = PF_BREAKDOWN; }
                else sc->alpha = sc->rho1 / gamma;
            }
            if (stop) {
                sc->done = 1;
                if (use_cond) cudaGraphSetConditional(cond, 0);
            }
            sc->k = k + 1;
            sc->counter = 0u;
        }
    }
}

// ---------------------------------------------------------------- kernel B
template <typename T>
struct PhaseB {
    static constexpr int R = Rows<T>::R;
    const T *res, *vv, *res0;
    T* t;
    T alpha;
    double st, tt, sr, tr;
    struct Raw { T r, v; };
    struct Ext { T r0; };
    __device__ Raw raw(long long q, int = 0, int = 0, int = 0) const { return Raw{res[q], vv[q]}; }
    __device__ Ext ext(long long q) const { return Ext{res0[q]}; }
    __device__ T op(const Raw& a) const { return fma(-alpha, a.v, a.r); }
    __device__ void epi(long long q, T c, T b, const Raw&, const Ext& e) {
        t[q] = b;
        st += double(c) * double(b);
        tt += double(b) * double(b);
        sr += double(c) * double(e.r0);
        tr += double(b) * double(e.r0);
    }
};

template <typename T>
__global__ void __launch_bounds__(kBlock, 2)
bicg_b(Dims d, Tiling tl, LapCoef<T> cf, BicgScalars* sc, double* part,
       BicgVecs<T> v, int use_cond = 0, cudaGraphConditionalHandle cond = 0) {
    __shared__ double sh[32];
    if (sc->done) {
        if (sc->done == 1 && use_cond && blockIdx.x == 0 && tid0())
            cudaGraphSetConditional(cond, 0);
        return;
    }
    const bool odd = (sc->k - 1) & 1;  // set written by the CA kernel just run
    PhaseB<T> ph;
    ph.res = odd ? v.res[1] : v.res[0];
    ph.vv = odd ? v.vv[1] : v.vv[0];
    ph.res0 = v.res0; ph.t = v.t;
    ph.alpha = T(sc->alpha);
    ph.st = ph.tt = ph.sr = ph.tr = 0.0;
    sweep<T>(d, tl, cf, ph);
    const double b0 = block_sum<kBlock>(ph.st, sh);
    const double b1 = block_sum<kBlock>(ph.tt, sh);
    const double b2 = block_sum<kBlock>(ph.sr, sh);
    const double b3 = block_sum<kBlock>(ph.tr, sh);
    if (tid0()) {
        part[blockIdx.x] = b0;
        part[kMaxPartials + blockIdx.x] = b1;
        part[2 * kMaxPartials + blockIdx.x] = b2;
        part[3 * kMaxPartials + blockIdx.x] = b3;
    }
    if (arrive_last(sc)) {
        const double buf1 = finish<false>(part, sh);
        const double buf2 = finish<false>(part + kMaxPartials, sh);
        const double sr = finish<false>(part + 2 * kMaxPartials, sh);
        const double tr = finish<false>(part + 3 * kMaxPartials, sh);
        if (tid0()) {
            sc->buf1 = buf1; sc->buf2 = buf2;
            if (buf2 == 0.0) {
                sc->done = 2;
                sc->status = PF_BREAKDOWN;
            } else {
                const double omega = buf1 / buf2;
                sc->omega = omega;
                sc->rho2 = sc->rho1;
                sc->rho1 = sr - omega * tr;  // (s - omega t, res0)
            }
            sc->counter = 0u;
        }
    }
}

// ------------------------------------------------- the solve in one launch
// The FP64 iterations of a grid of up to 296 tiles (two per SM) as one
// cooperative launch: kernels CA and B over the same tiles and sums, separated
// by grid barriers (pf_gridbar.cuh) instead of launches.  Per iteration, launch
// pairs -> this kernel, on one B200: 24^3 28.6 -> 12.7 us, 64^3 28.3 -> 12.0,
// 70x90x50 31.7 -> 17.0, 96^3 38.8 -> 27.8.  The pairs spent it on launch gaps,
// the serial last block that finished each reduction, and one L2 round trip
// per plane; left is latency: two barriers (1.6 us each at 128 blocks, 3 us at
// 288), the ring cells' loads, and at 96^3 instruction issue.  Every block
// folds the partials itself, in the order the last block used, one value per
// warp, and all hold the same scalars.  The iterates are bitwise those of the
// two kernels.  Deeper tiles (128^3: 68.4 us) stay with the launch pairs.

// Sums of V values over the block in block_sum's order (the value in bit v of
// MAXES: the maximum, NaN propagating), stored to out[v * kIterParts].
constexpr int kIterParts = 512;     // partial slots per value (at most 2 blocks per SM)
constexpr size_t kIterBar = 192;    // the barrier words lie behind the scalars, in their 256 bytes
static_assert(sizeof(BicgScalars) <= kIterBar, "scalar block");
static_assert(kIterParts <= 2 * kBlock, "fold_values takes two partials per thread");

template <int V, unsigned MAXES>
__device__ __forceinline__ void block_values(const double (&in)[V], double* sh, double* out) {
    const int tid = threadIdx.y * blockDim.x + threadIdx.x, lane = tid & 31, wid = tid >> 5;
    double x[V];
#pragma unroll
    for (int v = 0; v < V; ++v) x[v] = in[v];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const double y = __shfl_down_sync(0xffffffffu, x[v], o);
            x[v] = (MAXES >> v) & 1u ? absmax(x[v], y) : x[v] + y;
        }
    if (lane == 0)
#pragma unroll
        for (int v = 0; v < V; ++v) sh[v * 8 + wid] = x[v];
    __syncthreads();
    if (wid < V) {
        const bool mx = (MAXES >> wid) & 1u;
        double y = lane < kBlock / 32 ? sh[wid * 8 + lane] : 0.0;
        for (int o = 16; o > 0; o >>= 1) {
            const double z = __shfl_down_sync(0xffffffffu, y, o);
            y = mx ? absmax(y, z) : y + z;
        }
        if (lane == 0) out[wid * kIterParts] = y;
    }
}

// The blocks' partials of V values in finish's order, one value per warp; the
// results in sh[0 .. V-1] for all threads.
template <int V, unsigned MAXES>
__device__ __forceinline__ void fold_values(const double* part, double* sh) {
    const int tid = threadIdx.y * blockDim.x + threadIdx.x, lane = tid & 31, wid = tid >> 5;
    constexpr int W = kBlock / 32;
    if (wid < V) {
        const bool mx = (MAXES >> wid) & 1u;
        const double* pv = part + wid * kIterParts;
        // every load before the first sum (one after another each waits for L2)
        double x[W], y2[W];
#pragma unroll
        for (int w = 0; w < W; ++w) {
            const int b = 32 * w + lane;
            x[w] = b < (int)gridDim.x ? __ldcg(pv + b) : 0.0;
            y2[w] = b + kBlock < (int)gridDim.x ? __ldcg(pv + b + kBlock) : 0.0;
        }
#pragma unroll
        for (int w = 0; w < W; ++w) {
            const double y = 0.0 + x[w];
            x[w] = 32 * w + lane + kBlock < (int)gridDim.x
                       ? (mx ? absmax(y, y2[w]) : y + y2[w]) : y;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int w = 0; w < W; ++w) {
                const double y = __shfl_down_sync(0xffffffffu, x[w], o);
                x[w] = mx ? absmax(x[w], y) : x[w] + y;
            }
        // the tree over the W warp sums
#pragma unroll
        for (int o = W / 2; o > 0; o >>= 1)
#pragma unroll
            for (int w = 0; w < o; ++w) x[w] = mx ? absmax(x[w], x[w + o]) : x[w] + x[w + o];
        if (lane == 0) sh[wid] = x[0];
    }
    __syncthreads();
}

// The scalars after kernel CA of iteration k + 1 (its sums gamma, max|res|) and
// after kernel B (its four sums), as the kernels' last blocks form them.
__device__ __forceinline__ void solve_after_ca(BicgScalars& S, int k, double gamma, double mxr) {
    bool stop = false;
    if (k > 0) {
        // stop tests of iteration k (src/solver/pressure.py:279-287)
        S.iter = k;
        const double mr = mxr / S.max_res0;
        S.max_res = mr;
        if (!(mr == mr) || isinf(mr)) { stop = true; S.status = PF_NONFINITE; }
        else if (mr <= S.min_res) { stop = true; S.status = PF_OK; }
        else if (k >= S.max_it) { stop = true; S.status = PF_MAXIT; }
    }
    if (!stop) {
        S.gamma = gamma;
        if (gamma == 0.0) { stop = true; S.status = PF_BREAKDOWN; }
        else S.alpha = S.rho1 / gamma;
    }
    if (stop) S.done = 1;
    S.k = k + 1;
}

__device__ __forceinline__ void solve_after_b(BicgScalars& S, const double* sums) {
    S.buf1 = sums[0]; S.buf2 = sums[1];
    if (S.buf2 == 0.0) {
        S.done = 2;
        S.status = PF_BREAKDOWN;
    } else {
        const double omega = S.buf1 / S.buf2;
        S.omega = omega;
        S.rho2 = S.rho1;
        S.rho1 = sums[2] - omega * sums[3];  // (s - omega t, res0)
    }
}

// One tile per block, its part of the solve kept on the SM for the whole of it:
// res, pp and t in shared memory with the stencil operand and its ring of
// neighbours, vv and x there too (up to 4 planes) or in registers.  (Spilled
// registers are no place for it: after a barrier's acquire every reload from
// local memory goes to L2; with 38 spilled words an iteration took 24 us.)
// Only what neighbouring tiles read travels: a block publishes res, pp, vv and
// t of its boundary cells (in the two kernels' buffer sets) and forms
// the operand of its ring cells from its neighbours' published values.
template <int XC, int PER>
struct TileSolve {
    static constexpr int kRing = 34 * 18;              // one plane of the operand
    // all five fields in shared memory (one block of at most 6 planes per SM,
    // or two of 4), or res, pp and t
    static constexpr bool kAll = PER == 1 || XC <= 4;
    static constexpr size_t bytes = ((kAll ? 5 : 3) * 512 * XC + (XC + 2) * kRing) * sizeof(double);
    static constexpr int kBatch = PER == 1 ? 4 : 2;    // ring cells whose loads are in flight
    static constexpr int kItems = (96 * XC + kBlock - 1) / kBlock;  // ring cells in y and z per thread
};

template <int XC, int PER>
__global__ void __launch_bounds__(kBlock, PER)
bicg_tile_solve(Dims d, Tiling tl, LapCoef<double> cf, BicgScalars* sc, double* part,
                BicgVecs<double> v, double* xg) {
    using TS = TileSolve<XC, PER>;
    constexpr int PL = TS::kRing;
    extern __shared__ __align__(16) double tsm[];
    double* const res = tsm;                 // [plane][16][32]
    double* const pp = tsm + 512 * XC;
    double* const tt = tsm + 2 * 512 * XC;
    double* const vs = tsm + 3 * 512 * XC;   // vv and x if kAll
    double* const xs = tsm + 4 * 512 * XC;
    double* const H = tsm + (TS::kAll ? 5 : 3) * 512 * XC;  // [plane + 1][18][34]: the operand
    constexpr int XR = TS::kAll ? 1 : XC;
    double vr[XR][2], xr[XR][2];             // else
    __shared__ double sh[32];
    __shared__ BicgScalars S;
    int tx = threadIdx.x, ty = threadIdx.y;
    unsigned* const bar = (unsigned*)((char*)sc + kIterBar);
    unsigned round = 0;
    if (tid0()) S = *sc;
    // the tile, as in sweep()
    const int t = blockIdx.x, tz = t % tl.ntz, rr = t / tl.ntz;
    const int k0 = tz * 32, j0 = (rr % tl.nty) * 16, i0 = (rr / tl.nty) * tl.xc;
    const int np = min(tl.xc, d.nx - i0), ez = min(32, d.nz - k0), ey = min(16, d.ny - j0);
    const int plane = d.ny * d.nz;
    // The offsets below are recomputed in every phase: kept across the loop
    // they took the registers of the state and spilled.  fresh() hides where
    // tx and ty come from.
    auto fresh = [&]() { asm volatile("" : "+r"(tx), "+r"(ty)); };
    auto row_ok = [&](int r) { return tx < ez && ty + 8 * r < ey; };
    auto own_q = [&](int p, int r) { return (i0 + p) * plane + (j0 + ty + 8 * r) * d.nz + k0 + tx; };
    auto own_e = [&](int p, int r) { return (p * 16 + ty + 8 * r) * 32 + tx; };
    auto own_h = [&](int p, int r) { return (p + 1) * PL + (ty + 8 * r + 1) * 34 + tx + 1; };
    // cells that a neighbouring tile reads
    auto edge = [&](int p, int r) {
        const int jl = ty + 8 * r;
        return p == 0 || p == np - 1 || jl == 0 || jl == ey - 1 || tx == 0 || tx == ez - 1;
    };
    // ring cell `h` of plane h / 96: 32 below and 32 above in y, 16 and 16 in z;
    // its place in H (0: none) and in the grid
    auto ring = [&](int h, int& e, int& q) {
        const int p = h / 96, c = h - p * 96;
        e = 0;
        if (p >= np) return;
        int row, col;
        if (c < 64) {
            row = c < 32 ? 0 : ey + 1;
            col = (c & 31) + 1;
            if (col > ez) return;
        } else {
            row = ((c - 64) & 15) + 1;
            col = c < 80 ? 0 : ez + 1;
            if (row > ey) return;
        }
        e = (p + 1) * PL + row * 34 + col;
        q = (i0 + p) * plane + wrap(j0 + row - 1, d.ny) * d.nz + wrap(k0 + col - 1, d.nz);
    };
    // the operand of every ring cell, op(q): first the planes beside the tile,
    // then the rows and columns around it
    auto fill_ring = [&](auto load, auto op) {
        const int qm = wrap(i0 - 1, d.nx) * plane, qp = wrap(i0 + np, d.nx) * plane;
        // (at most four cells' values at a time)
#pragma unroll
        for (int m0 = 0; m0 < 4; m0 += TS::kBatch) {
            decltype(load(0)) w[TS::kBatch];
#pragma unroll
            for (int m = m0; m < m0 + TS::kBatch; ++m)
                if (row_ok(m & 1))
                    w[m - m0] = load((m < 2 ? qm : qp) + (j0 + ty + 8 * (m & 1)) * d.nz + k0 + tx);
#pragma unroll
            for (int m = m0; m < m0 + TS::kBatch; ++m)
                if (row_ok(m & 1)) H[own_h(m < 2 ? -1 : np, m & 1)] = op(w[m - m0]);
            fresh();
        }
#pragma unroll
        for (int m0 = 0; m0 < TS::kItems; m0 += TS::kBatch) {
            decltype(load(0)) w[TS::kBatch];
            int e[TS::kBatch];
#pragma unroll
            for (int m = 0; m < TS::kBatch; ++m) {
                int q;
                ring(ty * 32 + tx + (m0 + m) * kBlock, e[m], q);
                if (e[m]) w[m] = load(q);
            }
#pragma unroll
            for (int m = 0; m < TS::kBatch; ++m)
                if (e[m]) H[e[m]] = op(w[m]);
            fresh();
        }
    };
    auto stencil = [&](int h) {
        const double c = H[h];
        double b = 0.0;
        b += H[h - PL] * cf.c[0][0];
        b += c * cf.c[0][1];
        b += H[h + PL] * cf.c[0][2];
        b += H[h - 34] * cf.c[1][0];
        b += c * cf.c[1][1];
        b += H[h + 34] * cf.c[1][2];
        b += H[h - 1] * cf.c[2][0];
        b += c * cf.c[2][1];
        b += H[h + 1] * cf.c[2][2];
        return b;
    };
    // a barrier that gave up ends the solve with an error
    auto failed = [&]() {
        if (tid0()) { sc->status = PF_ERR_CUDA; sc->done = 1; }
    };
    // bicg_init's state (buffer set 1): res = b, pp = vv = t = x = 0
    auto VV = [&](int p, int r) -> double& {
        if constexpr (TS::kAll) return vs[own_e(p, r)]; else return vr[p][r];
    };
    auto X = [&](int p, int r) -> double& {
        if constexpr (TS::kAll) return xs[own_e(p, r)]; else return xr[p][r];
    };
    // f(plane, row) for the thread's cells, one plane after another (the
    // compiler may not mix the planes: their loads would fill the registers)
    auto cells = [&](auto f) {
#pragma unroll
        for (int p = 0; p < XC; ++p) {
            if (PER > 1) asm volatile("" ::: "memory");
#pragma unroll
            for (int r = 0; r < 2; ++r)
                if (p < np && row_ok(r)) f(p, r);
        }
    };
    // the same with res0 of the cell: held in registers by a block that has the
    // SM to itself, else loaded a plane ahead
    double r0s[PER == 1 ? XC : 1][2];
    auto cells_r0 = [&](auto f) {
        double nx[2];
        auto fetch = [&](int p) {
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                if constexpr (PER == 1) nx[r] = r0s[p][r];
                else nx[r] = p < np && row_ok(r) ? __ldg(v.res0 + own_q(p, r)) : 0.0;
            }
        };
        fetch(0);
#pragma unroll
        for (int p = 0; p < XC; ++p) {
            const double r0[2] = {nx[0], nx[1]};
            if (p + 1 < XC) fetch(p + 1);
            if (PER > 1) asm volatile("" ::: "memory");
#pragma unroll
            for (int r = 0; r < 2; ++r)
                if (p < np && row_ok(r)) f(p, r, r0[r]);
        }
    };
    if constexpr (!TS::kAll) {
#pragma unroll
        for (int p = 0; p < XR; ++p)
#pragma unroll
            for (int r = 0; r < 2; ++r) vr[p][r] = xr[p][r] = 0.0;
    }
    cells([&](int p, int r) {
        const int e = own_e(p, r);
        const double b = v.res0[own_q(p, r)];
        res[e] = b;
        if constexpr (PER == 1) r0s[p][r] = b;
        pp[e] = tt[e] = 0.0;
        if constexpr (TS::kAll) vs[e] = xs[e] = 0.0;
    });
    __syncthreads();
    while (!S.done) {
        fresh();
        const int k = S.k;
        const bool odd = k & 1, fin = k > 0;  // CA(k) writes set k&1 and reads the other
        double val[4] = {0.0, 0.0, 0.0, 0.0};
        {
            const double alpha = S.alpha, omega = S.omega;
            const double beta = (S.alpha * S.rho1) / (S.rho2 * S.omega);
            const double* ro = odd ? v.res[0] : v.res[1];
            const double* po = odd ? v.pp[0] : v.pp[1];
            const double* vo = odd ? v.vv[0] : v.vv[1];
            double* rn = odd ? v.res[1] : v.res[0];
            double* pn = odd ? v.pp[1] : v.pp[0];
            double* vn = odd ? v.vv[1] : v.vv[0];
            cells([&](int p, int r) {
                    const int e = own_e(p, r);
                    double rv = res[e];
                    const double pv = pp[e];
                    if (fin) {
                        const double s = fma(-alpha, VV(p, r), rv);
                        rv = fma(-omega, tt[own_e(p, r)], s);
                        X(p, r) = fma(omega, s, fma(alpha, pv, X(p, r)));
                        res[e] = rv;
                    }
                    double q = fma(-omega, VV(p, r), pv);
                    q = q * beta;
                    q = q + rv;
                    pp[e] = q;
                    H[own_h(p, r)] = q;
                    val[1] = absmax(val[1], abs_bits(rv));
                    if (edge(p, r)) { rn[own_q(p, r)] = rv; pn[own_q(p, r)] = q; }
            });
            struct Raw { double r, p, v, t; };
            fresh();
            fill_ring([&](int q) { return Raw{ro[q], po[q], vo[q], v.t[q]}; },
                      [&](const Raw& a) {
                          double rv = a.r;
                          if (fin) rv = fma(-omega, a.t, fma(-alpha, a.v, a.r));
                          double q = fma(-omega, a.v, a.p);
                          q = q * beta;
                          return q + rv;
                      });
            __syncthreads();
            fresh();
            cells_r0([&](int p, int r, double r0) {
                    const double b = stencil(own_h(p, r));
                    VV(p, r) = b;
                    val[0] += b * r0;
                    if (edge(p, r)) vn[own_q(p, r)] = b;
            });
        }
        const double v2[2] = {val[0], val[1]};
        block_values<2, 2u>(v2, sh, part + blockIdx.x);
        if (!grid_meet(bar, ++round)) return failed();
        fold_values<2, 2u>(part, sh);
        if (tid0()) solve_after_ca(S, k, sh[0], sh[1]);
        __syncthreads();
        if (S.done) break;
        {
            fresh();
            const double alpha = S.alpha;
            const double* rn = odd ? v.res[1] : v.res[0];
            const double* vn = odd ? v.vv[1] : v.vv[0];
            cells([&](int p, int r) { H[own_h(p, r)] = fma(-alpha, VV(p, r), res[own_e(p, r)]); });
            fresh();
            fill_ring([&](int q) { return make_double2(rn[q], vn[q]); },
                      [&](const double2& a) { return fma(-alpha, a.y, a.x); });
            __syncthreads();
            val[0] = val[1] = 0.0;
            fresh();
            cells_r0([&](int p, int r, double r0) {
                    const int h = own_h(p, r);
                    const double c = H[h], b = stencil(h);
                    tt[own_e(p, r)] = b;
                    if (edge(p, r)) v.t[own_q(p, r)] = b;
                    val[0] += c * b;
                    val[1] += b * b;
                    val[2] += c * r0;
                    val[3] += b * r0;
            });
        }
        block_values<4, 0u>(val, sh, part + 2 * kIterParts + blockIdx.x);
        if (!grid_meet(bar, ++round)) return failed();
        fold_values<4, 0u>(part + 2 * kIterParts, sh);
        if (tid0()) solve_after_b(S, sh);
        __syncthreads();
        if (S.done == 2) {
            // (t,t) == 0 breakdown: the reference has applied DP += alpha pp and
            // stops (src/solver/pressure.py:251,266-267)
            cells([&](int p, int r) { X(p, r) = fma(S.alpha, pp[own_e(p, r)], X(p, r)); });
        }
    }
    cells([&](int p, int r) { xg[own_q(p, r)] = X(p, r); });
    // every block holds the same scalars: once all have read the stored ones,
    // one block stores them
    if (!grid_meet(bar, ++round)) return failed();
    if (blockIdx.x == 0 && tid0()) { S.done = 1; *sc = S; }
}

typedef void (*TileKernel)(Dims, Tiling, LapCoef<double>, BicgScalars*, double*, BicgVecs<double>,
                           double*);

constexpr int kTilePlanes = 6;  // deepest tile: two blocks' shared memory per SM

template <int PER>
static TileKernel tile_kernel_of(int xc, size_t* smem) {
    switch (xc) {
        case 6: *smem = TileSolve<6, PER>::bytes; return bicg_tile_solve<6, PER>;
        case 5: *smem = TileSolve<5, PER>::bytes; return bicg_tile_solve<5, PER>;
        default: *smem = TileSolve<4, PER>::bytes; return bicg_tile_solve<4, PER>;
    }
}

// One block per SM, with its registers, where the tiles are that few.
static TileKernel tile_kernel(const Tiling& tl, size_t* smem) {
    return tl.ntiles <= num_sms() ? tile_kernel_of<1>(tl.xc, smem) : tile_kernel_of<2>(tl.xc, smem);
}

static cudaError_t tile_attributes() {
    for (int xc = 4; xc <= kTilePlanes; ++xc)
        for (int per = 1; per <= 2; ++per) {
            size_t smem;
            TileKernel k = per == 1 ? tile_kernel_of<1>(xc, &smem) : tile_kernel_of<2>(xc, &smem);
            const cudaError_t e =
                cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (e != cudaSuccess) return e;
        }
    return cudaSuccess;
}

// True when the whole solve runs as one cooperative launch: every block has
// one tile of at most kTilePlanes planes and all are resident at once.
static bool tile_solve_applies(const Dims& d) {
    const Tiling tl = make_tiling(d, 16);
    if (tl.xc > kTilePlanes || tl.ntiles > std::min(2 * num_sms(), kIterParts) || d.n >= (1LL << 30))
        return false;
    if (once_per_context((const void*)&tile_attributes, &tile_attributes) != cudaSuccess) return false;
    size_t smem;
    TileKernel k = tile_kernel(tl, &smem);
    int dev = 0, coop = 0, per = 0;
    return cudaGetDevice(&dev) == cudaSuccess &&
           cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) == cudaSuccess && coop &&
           cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k, kBlock, smem) == cudaSuccess &&
           tl.ntiles <= (long long)per * num_sms();
}

static cudaError_t launch_tile_solve(const Dims& d, const LapCoef<double>& cf, BicgScalars* sc,
                                     double* part, const BicgVecs<double>& v, double* x,
                                     cudaStream_t s) {
    const Tiling tl = make_tiling(d, 16);
    cudaLaunchConfig_t cfg = {};
    TileKernel k = tile_kernel(tl, &cfg.dynamicSmemBytes);
    cfg.gridDim = dim3((unsigned)tl.ntiles);
    cfg.blockDim = dim3(32, 8);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k, d, tl, cf, sc, part, v, x);
}

// ------------------------------------------------ mixed-precision refinement
// b = (source*rho/dt)*(-vol) in FP64, max|b|; DP = 0 unless x is null (a
// solve that starts from the DP it is given).
__global__ void __launch_bounds__(kBlock)
mixed_b_init(Dims d, BicgScalars* sc, double* part, const double* src,
             double c1, double c2, double* b, double* x, double* r_copy) {
    __shared__ double sh[32];
    double m = 0.0;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < d.n;
         q += (long long)gridDim.x * blockDim.x) {
        const double r = (src[q] * c1) * c2;
        b[q] = r;
        if (x) x[q] = 0.0;
        if (r_copy) r_copy[q] = r;
        m = nanmax(m, fabs(r));
    }
    const double bm = block_max<kBlock>(m, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = bm;
    if (arrive_last(sc)) {
        const double mx = finish<true>(part, sh);
        if (threadIdx.x == 0) {
            sc->max_b = mx; sc->scale = mx; sc->true_res = mx;
            sc->outer = 0; sc->total = 0; sc->counter = 0u;
            sc->use64 = 0; sc->prev_ratio = 2.0;
            sc->done = 1;  // no pass is running
        }
    }
}

// Refinement update: x += scale * e (FP64 accumulate of a pass's correction,
// scale = max|r| of the residual the pass solved for).
template <typename T>
__global__ void __launch_bounds__(kBlock)
fold_correction(Dims d, const BicgScalars* sc, const T* e, double* x, int guard = 0) {
    // graph mode: a pass that ended non-finite or in breakdown is discarded
    if (guard && (sc->status == PF_NONFINITE || sc->status == PF_BREAKDOWN)) return;
    // a pass that stopped before its first iteration has e = 0 (and may not
    // have written it)
    if (sc->iter == 0) return;
    const double s = sc->scale;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < d.n;
         q += (long long)gridDim.x * blockDim.x)
        x[q] = x[q] + s * double(e[q]);
}

// r = b - A x in FP64 and max|r| (the refinement's true residual)
struct PhaseResidual {
    static constexpr int R = 4;
    const double *x, *b;
    double* r;
    double mx;
    struct Raw { double x; };
    struct Ext { double b; };
    __device__ Raw raw(long long q, int = 0, int = 0, int = 0) const { return Raw{x[q]}; }
    __device__ Ext ext(long long q) const { return Ext{b[q]}; }
    __device__ double op(const Raw& a) const { return a.x; }
    __device__ void epi(long long q, double, double ax, const Raw&, const Ext& e) {
        const double v = e.b - ax;
        r[q] = v;
        mx = nanmax(mx, fabs(v));
    }
};

__global__ void __launch_bounds__(kBlock, 2)
mixed_residual(Dims d, Tiling tl, LapCoef<double> cf, BicgScalars* sc,
               double* part, const double* __restrict__ b,
               const double* __restrict__ x, double* __restrict__ r, int gated = 0) {
    __shared__ double sh[32];
    if (gated && !sc->done) return;  // the pass is still running
    PhaseResidual ph{x, b, r, 0.0};
    sweep<double>(d, tl, cf, ph);
    const double bm = block_max<kBlock>(ph.mx, sh);
    if (tid0()) part[blockIdx.x] = bm;
    if (arrive_last(sc)) {
        const double mx = finish<true>(part, sh);
        if (tid0()) { sc->true_res = mx; sc->scale = mx; sc->counter = 0u; }
    }
}

// One reduction of V values over the grid, finished by the last block to
// arrive: every block stores its V sums (or, bit v of MAXES, integer maxima of
// non-negative values) at part[v * stride + block]; the last block's folds go
// to res (shared memory), true there.  One barrier per level for all values
// together: value by value, the two levels took 8 us of an 11 us kernel.
template <int V, unsigned MAXES>
__device__ __forceinline__ void block_reduce(double (&x)[V], double* sh, double* res) {
    const int tid = threadIdx.y * blockDim.x + threadIdx.x, lane = tid & 31, wid = tid >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const double y = __shfl_down_sync(0xffffffffu, x[v], o);
            x[v] = (MAXES >> v) & 1u ? absmax(x[v], y) : x[v] + y;
        }
    if (lane == 0)
#pragma unroll
        for (int v = 0; v < V; ++v) sh[v * 8 + wid] = x[v];
    __syncthreads();
    if (wid < V) {
        const bool mx = (MAXES >> wid) & 1u;
        double y = lane < kBlock / 32 ? sh[wid * 8 + lane] : 0.0;
        for (int o = 4; o > 0; o >>= 1) {
            const double z = __shfl_down_sync(0xffffffffu, y, o);
            y = mx ? absmax(y, z) : y + z;
        }
        if (lane == 0) res[wid] = y;
    }
    __syncthreads();
}

template <int V, unsigned MAXES>
__device__ __forceinline__ bool grid_reduce(double (&x)[V], BicgScalars* sc, double* part,
                                            int stride, double* sh, double* res) {
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    block_reduce<V, MAXES>(x, sh, res);
    if (tid < V) part[tid * stride + blockIdx.x] = res[tid];
    if (!arrive_last(sc)) return false;
#pragma unroll
    for (int v = 0; v < V; ++v) x[v] = 0.0;
    for (int b0 = tid; b0 < (int)gridDim.x; b0 += 2 * kBlock) {
        double y[V][2];
#pragma unroll
        for (int v = 0; v < V; ++v)
#pragma unroll
            for (int m = 0; m < 2; ++m)
                y[v][m] = b0 + m * kBlock < (int)gridDim.x ? __ldcg(part + v * stride + b0 + m * kBlock) : 0.0;
#pragma unroll
        for (int v = 0; v < V; ++v)
#pragma unroll
            for (int m = 0; m < 2; ++m) x[v] = (MAXES >> v) & 1u ? absmax(x[v], y[v][m]) : x[v] + y[v][m];
    }
    block_reduce<V, MAXES>(x, sh, res);
    return true;
}

// Blocks of the pointwise kernels that reduce: one wave of four per SM (three
// waves: each wave's arrivals cost a fence, 31.5 against 28.9 us at 128^3).
constexpr int kPassBlocks = 592;

// After a solve, in one pass over the grid:
//   CHECK    max|b| and max|b - A x| of the direct solve's x = DP (b = (src c1)
//            c2 formed on the fly), the end of the solve;
//   CORRECT  p += DP (src/solver/pressure.py:294) and the projection u_d -=
//            scale grad DP (src/data/domain.py:394-402).
// With both, the correction does not wait for the check: where it then fails
// (a source with a mean, a tolerance below the transforms' rounding),
// project_undo takes it back before FP64 BiCGStab passes go on from DP (u and p
// keep at most two roundings of |u| + 2 |scale grad DP| from that).  80
// bytes per cell, 26.6 us at 128^3 and 7.5 at 64^3 (6.3 TB/s of L2 and HBM at
// 128^3); as three kernels (96 bytes) with an IF node between the check and the
// correction it took 57 and 26 us of a step.
// A right-hand side that is not finite (sc->nonfin) gives DP = 0, no
// correction and PF_NONFINITE.  VEC: two cells in z per thread, 16-byte loads.
struct ProjectArgs {
    Dims d;
    int tz, ty;             // tiles of a plane
    long long ntiles;
    LapCoef<double> cf;
    BicgScalars* sc;
    double* part;
    const double* src;
    double c1, c2, min_res;
    int max_it;
    double* DP;
    double scale, dxi, dyi, dzi;
    double *u, *v, *w, *p;
    int use_cond;           // graph: the IF node's handle
    cudaGraphConditionalHandle cond;
};

template <int V>
struct Cells {
    double a[V];
};
template <int V>
__device__ __forceinline__ Cells<V> ld_cells(const double* p) {
    Cells<V> c;
    if constexpr (V == 2) {
        const double2 t = *(const double2*)p;
        c.a[0] = t.x;
        c.a[1] = t.y;
    } else {
        c.a[0] = *p;
    }
    return c;
}
template <int V>
__device__ __forceinline__ void st_cells(double* p, const Cells<V>& c) {
    if constexpr (V == 2) *(double2*)p = make_double2(c.a[0], c.a[1]);
    else *p = c.a[0];
}

template <int V, bool CHECK, bool CORRECT>
__global__ void __launch_bounds__(kBlock, 4)
project_kernel(ProjectArgs A) {
    __shared__ double sh[16], res[2];
    pdl_wait();
    const Dims d = A.d;
    const bool bad = CHECK && A.sc->nonfin != 0;
    double mx = 0.0, mb = 0.0;
    const long long plane = (long long)d.ny * d.nz;
    for (long long t = blockIdx.x; t < A.ntiles; t += gridDim.x) {
        const int t1 = (int)(t / A.tz), i = t1 / A.ty;
        const int k = ((int)(t - (long long)t1 * A.tz) * 32 + threadIdx.x) * V;
        const int j = (t1 - i * A.ty) * 8 + threadIdx.y;
        if (k >= d.nz || j >= d.ny) continue;
        const long long row = i * plane + (long long)j * d.nz, q = row + k;
        if (bad) {
            Cells<V> z;
#pragma unroll
            for (int m = 0; m < V; ++m) z.a[m] = 0.0;
            st_cells<V>(A.DP + q, z);
            continue;
        }
        const Cells<V> c = ld_cells<V>(A.DP + q);
        const Cells<V> xm = ld_cells<V>(A.DP + wrap(i - 1, d.nx) * plane + (long long)j * d.nz + k);
        const Cells<V> ym = ld_cells<V>(A.DP + i * plane + (long long)wrap(j - 1, d.ny) * d.nz + k);
        const double zm = A.DP[row + wrap(k - 1, d.nz)];
        Cells<V> xp, yp, src;
        double zp = 0.0;
        if (CHECK) {
            xp = ld_cells<V>(A.DP + wrap(i + 1, d.nx) * plane + (long long)j * d.nz + k);
            yp = ld_cells<V>(A.DP + i * plane + (long long)wrap(j + 1, d.ny) * d.nz + k);
            zp = A.DP[row + wrap(k + V, d.nz)];
            src = ld_cells<V>(A.src + q);
        }
        Cells<V> u, v, w, p;
        if (CORRECT) {
            u = ld_cells<V>(A.u + q);
            v = ld_cells<V>(A.v + q);
            w = ld_cells<V>(A.w + q);
            p = ld_cells<V>(A.p + q);
        }
#pragma unroll
        for (int m = 0; m < V; ++m) {
            const double x = c.a[m], zl = m ? c.a[m - 1] : zm;
            if (CHECK) {
                const double zr = m + 1 < V ? c.a[m + 1 < V ? m + 1 : m] : zp;
                double ax = 0.0;
                ax += xm.a[m] * A.cf.c[0][0];
                ax += x * A.cf.c[0][1];
                ax += xp.a[m] * A.cf.c[0][2];
                ax += ym.a[m] * A.cf.c[1][0];
                ax += x * A.cf.c[1][1];
                ax += yp.a[m] * A.cf.c[1][2];
                ax += zl * A.cf.c[2][0];
                ax += x * A.cf.c[2][1];
                ax += zr * A.cf.c[2][2];
                const double b = (src.a[m] * A.c1) * A.c2;
                mx = absmax(mx, abs_bits(b - ax));
                mb = absmax(mb, abs_bits(b));
            }
            if (CORRECT) {
                p.a[m] = p.a[m] + x;
                u.a[m] = fma(-A.scale, (x - xm.a[m]) * A.dxi, u.a[m]);  // var.sub_(scale, grad)
                v.a[m] = fma(-A.scale, (x - ym.a[m]) * A.dyi, v.a[m]);
                w.a[m] = fma(-A.scale, (x - zl) * A.dzi, w.a[m]);
            }
        }
        if (CORRECT) {
            st_cells<V>(A.p + q, p);
            st_cells<V>(A.u + q, u);
            st_cells<V>(A.v + q, v);
            st_cells<V>(A.w + q, w);
        }
    }
    if (!CHECK) return;
    BicgScalars* sc = A.sc;
    double red[2] = {mx, mb};
    if (grid_reduce<2, 3u>(red, sc, A.part, kPassBlocks, sh, res)) {
        const double fx = res[0], fb = res[1];
        if (tid0()) {
            const double nan = __longlong_as_double(0x7ff8000000000000LL);
            const double ratio = bad ? nan : (fb == 0.0 ? 0.0 : fx / fb);
            sc->max_b = fb; sc->scale = fx; sc->true_res = fx; sc->max_res = ratio;
            sc->outer = 1;
            sc->total = sc->iter = fb == 0.0 && !bad ? 0 : 1;
            sc->use64 = 1; sc->prev_ratio = ratio;
            bool more = false;
            if (!(ratio == ratio) || isinf(ratio)) sc->status = PF_NONFINITE;
            else if (ratio <= A.min_res) sc->status = PF_OK;
            else if (A.max_it <= 1) sc->status = PF_MAXIT;
            else more = true;
            sc->done = more ? 0 : 1;
            sc->redo = more ? 1 : 0;
            sc->nonfin = 0;
            sc->counter = 0u;
            if (A.use_cond) cudaGraphSetConditional(A.cond, more ? 1u : 0u);
        }
    }
}

// Takes project_kernel's correction back (to rounding).
__global__ void __launch_bounds__(256)
project_undo(Dims d, const double* __restrict__ DP, double scale, double dxi, double dyi,
             double dzi, double* __restrict__ u, double* __restrict__ v, double* __restrict__ w,
             double* __restrict__ p) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int i = blockIdx.z;
    if (k >= d.nz || j >= d.ny) return;
    const long long q = idx(d, i, j, k);
    const double c = DP[q];
    u[q] = fma(scale, (c - DP[idx(d, wrap(i - 1, d.nx), j, k)]) * dxi, u[q]);
    v[q] = fma(scale, (c - DP[idx(d, i, wrap(j - 1, d.ny), k)]) * dyi, v[q]);
    w[q] = fma(scale, (c - DP[idx(d, i, j, wrap(k - 1, d.nz))]) * dzi, w[q]);
    p[q] = p[q] - c;
}

template <bool CHECK, bool CORRECT>
static void launch_project(const char* name, const pf_grid* g, ProjectArgs A, cudaStream_t s) {
    A.d = Dims{g->nx, g->ny, g->nz, (long long)g->nx * g->ny * g->nz};
    A.cf = lap_coef<double>(g);
    A.dxi = 1.0 / g->dx; A.dyi = 1.0 / g->dy; A.dzi = 1.0 / g->dz;
    uintptr_t bits = (uintptr_t)A.DP;
    if (CHECK) bits |= (uintptr_t)A.src;
    if (CORRECT) bits |= (uintptr_t)A.u | (uintptr_t)A.v | (uintptr_t)A.w | (uintptr_t)A.p;
    const bool vec = g->nz % 2 == 0 && (bits & 15) == 0;
    const int zt = vec ? 64 : 32;
    A.tz = (g->nz + zt - 1) / zt;
    A.ty = (g->ny + 7) / 8;
    A.ntiles = (long long)A.tz * A.ty * g->nx;
    const int blocks = (int)std::min<long long>(A.ntiles, kPassBlocks);
    if (vec)
        PF_LAUNCH(name, s, launch_pdl(project_kernel<2, CHECK, CORRECT>, dim3(blocks), dim3(32, 8), 0, s, A));
    else
        PF_LAUNCH(name, s, launch_pdl(project_kernel<1, CHECK, CORRECT>, dim3(blocks), dim3(32, 8), 0, s, A));
}

// b = (src c1) c2
__global__ void __launch_bounds__(kBlock)
scaled_source(long long n, const double* src, double c1, double c2, double* b) {
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n;
         q += (long long)gridDim.x * blockDim.x)
        b[q] = (src[q] * c1) * c2;
}

// p += DP (src/solver/pressure.py:294)
__global__ void __launch_bounds__(kBlock)
add_inplace(long long n, const double* a, double* p) {
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n;
         q += (long long)gridDim.x * blockDim.x)
        p[q] = p[q] + a[q];
}

// ------------------------------------------------------------ workspace

static constexpr int kNumPartials = 4;

size_t poisson_ws_bytes(const pf_grid* g, int prec) {
    const size_t n = (size_t)g->nx * g->ny * g->nz;
    size_t b = align256(sizeof(BicgScalars)) +
               align256(kNumPartials * kMaxPartials * sizeof(double));
    if (prec == PF_FP64) {
        b += 8 * align256(n * sizeof(double));  // res[2] pp[2] vv[2] t res0
    } else {
        // inner vectors + correction: FP32 passes, or FP64 passes after an
        // FP32 pass fails (the two sets share one region), then b and r
        b += 9 * align256(n * sizeof(double));
        b += 2 * align256(n * sizeof(double));
    }
    return b;
}

template <typename T>
static BicgVecs<T> carve(char*& p, size_t n) {
    BicgVecs<T> v;
    T** f[8] = {&v.res[0], &v.res[1], &v.pp[0], &v.pp[1], &v.vv[0], &v.vv[1], &v.t, &v.res0};
    for (auto ptr : f) { *ptr = (T*)p; p += align256(n * sizeof(T)); }
    return v;
}

static LapCoef<double> cf64(const pf_grid* g) { return lap_coef<double>(g); }

static int read_scalars(BicgScalars* dev, BicgScalars* host, cudaStream_t s) {
    if (cudaMemcpyAsync(host, dev, sizeof(BicgScalars), cudaMemcpyDeviceToHost, s) != cudaSuccess)
        return PF_ERR_CUDA;
    if (cudaStreamSynchronize(s) != cudaSuccess) return PF_ERR_CUDA;
    return PF_OK;
}

// Enqueue BiCGStab iterations in chunks, polling the device `done` flag
// between chunks; kernels of a finished solve return at once.  Launch order:
// CA(0), then pairs (B(k), CA(k+1)), so every chunk ends with a CA and the
// last iteration of a chunk is finished before polling.
template <typename T>
static int run_iterations(const Dims& d, const LapCoef<T>& cf,
                          BicgScalars* sc, double* part, const BicgVecs<T>& v,
                          T* x, cudaStream_t s, BicgScalars* hs) {
    const Tiling ta = make_tiling(d, 8 * PhaseCA<T>::R);
    const Tiling tb = make_tiling(d, 8 * PhaseB<T>::R);
    const int ga = tiled_grid(ta), gb = tiled_grid(tb);
    if constexpr (sizeof(T) == 8) {
        // (the per-kernel timers count the two kernels)
        if (!prof_on() && tile_solve_applies(d)) {
            if (launch_tile_solve(d, cf, sc, part, v, x, s) != cudaSuccess) return PF_ERR_CUDA;
            const int rc = read_scalars(sc, hs, s);
            return rc ? rc : (hs->status == PF_ERR_CUDA ? PF_ERR_CUDA : PF_OK);
        }
    }
    dim3 blk2(32, 8);
    const char* nca = sizeof(T) == 8 ? "bicg_ca_f64" : "bicg_ca_f32";
    const char* nb = sizeof(T) == 8 ? "bicg_b_f64" : "bicg_b_f32";
    PF_LAUNCH(nca, s, bicg_ca<T><<<ga, blk2, 0, s>>>(d, ta, cf, sc, part, v, x));
    // with per-kernel timing on, poll after every iteration so no launch of
    // a finished solve (which returns at once) enters the kernel averages
    const bool exact = prof_on();
    int chunk = exact ? 1 : 4;
    for (int guard = 0; guard < (1 << 20); ++guard) {
        for (int c = 0; c < chunk; ++c) {
            PF_LAUNCH(nb, s, bicg_b<T><<<gb, blk2, 0, s>>>(d, tb, cf, sc, part, v));
            PF_LAUNCH(nca, s, bicg_ca<T><<<ga, blk2, 0, s>>>(d, ta, cf, sc, part, v, x));
        }
        if (cudaGetLastError() != cudaSuccess) return PF_ERR_CUDA;
        const int rc = read_scalars(sc, hs, s);
        if (rc) return rc;
        if (hs->done == 1) return PF_OK;
        chunk = exact ? 1 : std::min(chunk * 2, 32);
    }
    return PF_ERR_CUDA;
}

// PF_MIXED_MG grids that keep the V-cycle iterations where the direct solve
// would serve too: all that coarsen when PF_MG_COOP asks for them, and those of
// at most 2^15 cells.  The bound keeps the results that such requests had before
// there was a direct solve; it is not the faster choice (a captured 32^3 step
// takes 0.55 ms with the V-cycles, 0.10 ms direct) nor the more accurate one.
// Any change of DP, however small, flips roundings of the FP32 stages, and the
// flips grow: at 32^3, the one size measured below the bound, the velocities of
// the two solvers differ by up to 3e-9 after 10 steps (2-norm; 8e-15 after the
// first), where either is 1.6e-8 from the FP64 form.  Measured above it: 9e-11 after 5
// steps at 128^3, 1.9e-10 after 3 at 90x77x63, 2e-10 after 4 in ensembles up to
// 192^3 (single cells beside a flip at a large velocity by up to 8e-8).
// PF_MIXED, and grids of any size that do not coarsen, solve directly.
constexpr long long kCyclesMaxCells = 1LL << 15;

static bool mg_cycles_serve(const pf_grid* g, int prec) {
    if (prec != PF_MIXED_MG || mg_region_bytes(g) == 0) return false;
    return mg_cycles_requested() || (long long)g->nx * g->ny * g->nz <= kCyclesMaxCells;
}

int bicgstab_solve(const pf_grid* g, int prec, double rho, double dt,
                   double min_res, int max_it, const double* source,
                   double* DP, double* p, void* ws, cudaStream_t s,
                   pf_solve_info* info) {
    // PF_WARM_START (mixed forms): the refinement starts from the DP given
    bool warm = (prec & PF_WARM_START) != 0 && (prec & 0xFF) != PF_FP64;
    const bool direct = (prec & PF_DIRECT_SOLVE) != 0 || (prec & 0xFF) != PF_FP64;
    prec &= 0xFF;
    Dims d{g->nx, g->ny, g->nz, (long long)g->nx * g->ny * g->nz};
    const size_t n = (size_t)d.n;
    char* ptr = (char*)ws;
    BicgScalars* sc = (BicgScalars*)ptr; ptr += align256(sizeof(BicgScalars));
    double* part = (double*)ptr; ptr += align256(kNumPartials * kMaxPartials * sizeof(double));
    const int gp = pointwise_grid(d.n);
    const double vol = (g->dx * g->dy) * g->dz;
    const double c1 = rho / dt, c2 = -1.0 * vol;
    BicgScalars hs;
    std::memset(&hs, 0, sizeof(hs));
    if (cudaMemsetAsync(sc, 0, sizeof(BicgScalars), s) != cudaSuccess) return PF_ERR_CUDA;
    pf_solve_info out{0.0, 0, 1, PF_OK};
    // the reference loop always runs at least one iteration
    max_it = std::max(max_it, 1);
    bool solved = false, use64 = false;
    int outer = 0, total = 0;
    // the direct solve's check reads the source again when DP is there: a DP in
    // the source's own buffer goes to the iterations, which keep b themselves
    if (direct && source != DP && !mg_cycles_serve(g, prec) && spectral_applies(g, min_res, DP, ptr)) {
        // the tables sit in the region of the iterative solver's vectors
        SpectralPlan sp;
        if (spectral_setup(g, ptr, &sp) != cudaSuccess ||
            spectral_enqueue_tables(sp, s) != cudaSuccess ||
            spectral_enqueue_solve(sp, source, c1 * c2, DP, &sc->nonfin, s) != cudaSuccess)
            return PF_ERR_CUDA;
        ProjectArgs A{};
        A.sc = sc; A.part = part; A.src = source; A.c1 = c1; A.c2 = c2;
        A.min_res = min_res; A.max_it = max_it; A.DP = DP;
        launch_project<true, false>("spectral_check", g, A, s);
        if (cudaGetLastError() != cudaSuccess || read_scalars(sc, &hs, s)) return PF_ERR_CUDA;
        if (hs.status == PF_NONFINITE && hs.max_b != 0.0) {
            // a finite source (else max_b is 0 and DP was cleared) whose
            // transforms or right-hand side overflow: the whole iterative
            // solve, which scales its vectors, from DP = 0
            warm = false;
        } else {
            solved = hs.done != 0;
            outer = hs.max_b == 0.0 ? 0 : 1;
            total = hs.total;
            out.max_res = hs.max_res; out.iterations = total; out.outer = outer; out.status = hs.status;
            // the mixed forms go on from here, in FP64; PF_FP64 starts over
            warm = use64 = prec != PF_FP64;
        }
    }
    if (solved) {
        // nothing more to iterate
    } else if (prec == PF_FP64) {
        BicgVecs<double> v = carve<double>(ptr, n);
        const LapCoef<double> cf = lap_coef<double>(g);
        PF_LAUNCH("bicg_init_f64", s, bicg_init<double, false><<<gp, kBlock, 0, s>>>(
            d, sc, part, source, c1, c2, v, DP, max_it, min_res));
        int rc = run_iterations<double>(d, cf, sc, part, v, DP, s, &hs);
        if (rc) return rc;
        out.max_res = hs.max_res; out.iterations = hs.iter; out.status = hs.status;
    } else {
        // Iterative refinement: each pass solves A e = r / max|r| with BiCGStab
        // on FP32 vectors (FP64 dot products) to kInnerTol, then
        // x += max|r| e and r = b - A x in FP64, until max|r| / max|b| reaches
        // the reference's tolerance.  A pass that ends non-finite or in
        // breakdown is discarded, and a pass that gains less than 2x switches
        // the solve to FP64 inner passes, so the refinement always converges
        // like the FP64 solver.
        char* region = ptr;
        BicgVecs<float> v32 = carve<float>(ptr, n);
        float* e32 = (float*)ptr;
        ptr = region + 9 * align256(n * sizeof(double));
        char* r64 = region;
        BicgVecs<double> v64 = carve<double>(r64, n);
        double* e64 = (double*)r64;
        double* b = (double*)ptr; ptr += align256(n * sizeof(double));
        double* r = (double*)ptr; ptr += align256(n * sizeof(double));
        const Tiling tld = make_tiling(d, 8 * PhaseResidual::R);
        const LapCoef<float> cf = lap_coef<float>(g);
        const LapCoef<double> cfd = lap_coef<double>(g);
        const double kInnerTol = 1e-4;
        const int kMaxOuter = 40;
        // PF_MIXED_MG: the FP32 passes run the multigrid-preconditioned solver
        // (its vectors share the same region) when the grid coarsens
        MgPlan mg;
        if (prec == PF_MIXED_MG && mg_region_bytes(g) <= 9 * align256(n * sizeof(double))) {
            const int rc = mg_setup(g, region, &mg);
            if (rc != PF_OK && rc != PF_ERR_BAD_ARG) return rc;
            if (mg.L && mg_enqueue_setup(mg, s) != PF_OK) return PF_ERR_CUDA;
        }
        PF_LAUNCH("mixed_b_init", s, mixed_b_init<<<gp, kBlock, 0, s>>>(d, sc, part, source, c1, c2, b,
                                                                       warm ? nullptr : DP, nullptr));
        if (read_scalars(sc, &hs, s)) return PF_ERR_CUDA;
        const double max_b = hs.max_b;
        int status = PF_OK;
        double ratio = max_b > 0 ? 1.0 : 0.0, prev_ratio = 2.0;
        if (!(max_b == max_b)) status = PF_NONFINITE;
        while (status == PF_OK && max_b > 0.0) {
            if (outer > 0 || warm) {
                PF_LAUNCH("mixed_residual", s, mixed_residual<<<tiled_grid(tld), dim3(32, 8), 0, s>>>(
                    d, tld, cfd, sc, part, b, DP, r));
                if (read_scalars(sc, &hs, s)) return PF_ERR_CUDA;
                ratio = hs.true_res / max_b;
            }
            if (!(ratio == ratio) || std::isinf(ratio)) { status = PF_NONFINITE; break; }
            if (ratio <= min_res) break;
            if (outer >= kMaxOuter || total >= max_it) { status = PF_MAXIT; break; }
            if (!use64 && outer > 1 && ratio > 0.5 * prev_ratio) use64 = true;
            prev_ratio = ratio;
            const double* rhs = (outer == 0 && !warm) ? b : r;
            ++outer;
            if (!use64) {
                float* e = e32;
                if (mg.L) {
                    const int rc = mg_inner_solve(mg, sc, part, rhs, kInnerTol, max_it - total, s,
                                                  &hs, min_res);
                    if (rc) return rc;
                    e = mg.e;
                } else {
                    PF_LAUNCH("bicg_init_f32", s, bicg_init<float, true><<<gp, kBlock, 0, s>>>(
                        d, sc, part, rhs, 0.0, 0.0, v32, e32, max_it - total, kInnerTol));
                    const int rc = run_iterations<float>(d, cf, sc, part, v32, e32, s, &hs);
                    if (rc) return rc;
                }
                total += hs.iter;
                if (hs.status == PF_NONFINITE || hs.status == PF_BREAKDOWN) {
                    use64 = true;  // discard this pass: x is unchanged
                    continue;
                }
                PF_LAUNCH("fold_correction", s, fold_correction<float><<<gp, kBlock, 0, s>>>(d, sc, e, DP));
            } else {
                // an FP64 pass finishes the solve: its tolerance is the
                // remaining reduction
                const double tol64 = std::min(0.5, 0.5 * min_res / ratio);
                PF_LAUNCH("bicg_init_f64", s, bicg_init<double, true><<<gp, kBlock, 0, s>>>(
                    d, sc, part, rhs, 0.0, 0.0, v64, e64, max_it - total, tol64));
                const int rc = run_iterations<double>(d, cf64(g), sc, part, v64, e64, s, &hs);
                if (rc) return rc;
                total += hs.iter;
                if (hs.status == PF_NONFINITE) { status = PF_NONFINITE; break; }
                PF_LAUNCH("fold_correction", s, fold_correction<double><<<gp, kBlock, 0, s>>>(d, sc, e64, DP));
            }
        }
        out.max_res = ratio; out.iterations = total; out.outer = outer; out.status = status;
    }
    PF_LAUNCH("add_inplace", s, add_inplace<<<gp, kBlock, 0, s>>>(d.n, DP, p));
    if (cudaGetLastError() != cudaSuccess) return PF_ERR_CUDA;
    if (info) *info = out;
    return PF_OK;
}

// ------------------------------------------------------------------ Jacobi
// One sweep of solver_jacobi.solve (src/solver/pressure.py:141-147).
__global__ void __launch_bounds__(kBlock)
jacobi_sweep(Dims d, const double* __restrict__ pold, const double* __restrict__ src,
             double* __restrict__ pnew) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int i = blockIdx.z;
    if (k >= d.nz || j >= d.ny) return;
    const double DInv = -1.0 / 6.0;
    double x = -pold[idx(d, wrap(i + 1, d.nx), j, k)];
    x = x - pold[idx(d, wrap(i - 1, d.nx), j, k)];
    x = x - pold[idx(d, i, wrap(j + 1, d.ny), k)];
    x = x - pold[idx(d, i, wrap(j - 1, d.ny), k)];
    x = x - pold[idx(d, i, j, wrap(k + 1, d.nz))];
    x = x - pold[idx(d, i, j, wrap(k - 1, d.nz))];
    x = x + src[idx(d, i, j, k)];
    pnew[idx(d, i, j, k)] = x * DInv;
}

// scaled source, max|.| for the initial residual, then * dx^2
__global__ void __launch_bounds__(kBlock)
jacobi_prep(Dims d, BicgScalars* sc, double* part, const double* src, double c1,
            double dx2, double* s_out, double* p, double* pold) {
    __shared__ double sh[32];
    double m = 0.0;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < d.n;
         q += (long long)gridDim.x * blockDim.x) {
        const double a = src[q] * c1;
        m = nanmax(m, fabs(a));
        s_out[q] = a * dx2;
        p[q] = 0.0;
        if (pold) pold[q] = 0.0;
    }
    const double bm = block_max<kBlock>(m, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = bm;
    if (arrive_last(sc)) {
        const double mx = finish<true>(part, sh);
        if (threadIdx.x == 0) { sc->max_res0 = mx; sc->counter = 0u; }
    }
}

// res = (A p) * -1 + source/dx^2, max|res| / max_res0
struct PhaseJacobiRes {
    static constexpr int R = 2;
    const double *p, *sdx;
    double dx2, mx;
    struct Raw { double p; };
    struct Ext { double s; };
    __device__ Raw raw(long long q, int = 0, int = 0, int = 0) const { return Raw{p[q]}; }
    __device__ Ext ext(long long q) const { return Ext{sdx[q]}; }
    __device__ double op(const Raw& a) const { return a.p; }
    __device__ void epi(long long, double, double ax, const Raw&, const Ext& e) {
        const double v = ax * -1.0 + e.s / dx2;
        mx = nanmax(mx, fabs(v));
    }
};

__global__ void __launch_bounds__(kBlock, 2)
jacobi_residual(Dims d, Tiling tl, LapCoef<double> cf, BicgScalars* sc,
                double* part, const double* __restrict__ sdx, double dx2,
                const double* __restrict__ p) {
    __shared__ double sh[32];
    PhaseJacobiRes ph{p, sdx, dx2, 0.0};
    sweep<double>(d, tl, cf, ph);
    const double bm = block_max<kBlock>(ph.mx, sh);
    if (tid0()) part[blockIdx.x] = bm;
    if (arrive_last(sc)) {
        const double mx = finish<true>(part, sh);
        if (tid0()) { sc->max_res = mx / sc->max_res0; sc->counter = 0u; }
    }
}

int jacobi_solve(const pf_grid* g, double rho, double dt, int n_it,
                 const double* source, double* pold, double* p, void* ws,
                 cudaStream_t s, double* max_res) {
    Dims d{g->nx, g->ny, g->nz, (long long)g->nx * g->ny * g->nz};
    const size_t n = (size_t)d.n;
    char* ptr = (char*)ws;
    BicgScalars* sc = (BicgScalars*)ptr; ptr += align256(sizeof(BicgScalars));
    double* part = (double*)ptr; ptr += align256(kNumPartials * kMaxPartials * sizeof(double));
    double* sdx = (double*)ptr; ptr += align256(n * sizeof(double));
    double* tmp = (double*)ptr;
    const int gp = pointwise_grid(d.n);
    const double dx2 = std::pow(g->dx, 2.0);
    if (cudaMemsetAsync(sc, 0, sizeof(BicgScalars), s) != cudaSuccess) return PF_ERR_CUDA;
    PF_LAUNCH("jacobi_prep", s, jacobi_prep<<<gp, kBlock, 0, s>>>(d, sc, part, source, rho / dt, dx2, sdx, p, nullptr));
    dim3 blk(32, 8), grd((d.nz + 31) / 32, (d.ny + 7) / 8, d.nx);
    // iterate: pold <- p; p <- sweep(pold).  Ping-pong between p and tmp so
    // that the last two iterates land in p (last) and pold (previous).
    for (int it = 0; it < n_it; ++it) {
        const bool last = (it == n_it - 1);
        double* src_buf = (it == 0) ? p : ((it & 1) ? tmp : p);
        double* dst_buf = (it & 1) ? p : tmp;
        if (last) {
            cudaMemcpyAsync(pold, src_buf, n * sizeof(double), cudaMemcpyDeviceToDevice, s);
            PF_LAUNCH("jacobi_sweep", s, jacobi_sweep<<<grd, blk, 0, s>>>(d, pold, sdx, p));
        } else {
            PF_LAUNCH("jacobi_sweep", s, jacobi_sweep<<<grd, blk, 0, s>>>(d, src_buf, sdx, dst_buf));
        }
    }
    const Tiling tl = make_tiling(d, 8 * PhaseJacobiRes::R);
    PF_LAUNCH("jacobi_residual", s, jacobi_residual<<<tiled_grid(tl), dim3(32, 8), 0, s>>>(d, tl, lap_coef<double>(g), sc, part, sdx, dx2, p));
    if (cudaGetLastError() != cudaSuccess) return PF_ERR_CUDA;
    BicgScalars hs;
    if (read_scalars(sc, &hs, s)) return PF_ERR_CUDA;
    if (max_res) *max_res = hs.max_res;
    return PF_OK;
}

// ------------------------------------------------------- small operators
__global__ void __launch_bounds__(256)
div_kernel(Dims d, const double* __restrict__ u, const double* __restrict__ v,
           const double* __restrict__ w, double dxi, double dyi, double dzi,
           double* __restrict__ out) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int i = blockIdx.z;
    if (k >= d.nz || j >= d.ny) return;
    const long long q = idx(d, i, j, k);
    double a = (u[idx(d, wrap(i + 1, d.nx), j, k)] - u[q]) * dxi;
    a += (v[idx(d, i, wrap(j + 1, d.ny), k)] - v[q]) * dyi;
    a += (w[idx(d, i, j, wrap(k + 1, d.nz))] - w[q]) * dzi;
    out[q] = a;
}

__global__ void __launch_bounds__(256)
laplace_kernel(Dims d, LapCoef<double> cf, const double* __restrict__ A,
               double* __restrict__ B) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int i = blockIdx.z;
    if (k >= d.nz || j >= d.ny) return;
    const double c = A[idx(d, i, j, k)];
    double b = 0.0;
    b += A[idx(d, wrap(i - 1, d.nx), j, k)] * cf.c[0][0];
    b += c * cf.c[0][1];
    b += A[idx(d, wrap(i + 1, d.nx), j, k)] * cf.c[0][2];
    b += A[idx(d, i, wrap(j - 1, d.ny), k)] * cf.c[1][0];
    b += c * cf.c[1][1];
    b += A[idx(d, i, wrap(j + 1, d.ny), k)] * cf.c[1][2];
    b += A[idx(d, i, j, wrap(k - 1, d.nz))] * cf.c[2][0];
    b += c * cf.c[2][1];
    b += A[idx(d, i, j, wrap(k + 1, d.nz))] * cf.c[2][2];
    B[idx(d, i, j, k)] = b;
}

__global__ void __launch_bounds__(256)
vel_corr_kernel(Dims d, const double* __restrict__ DP, double scale, double dxi,
                double dyi, double dzi, double* __restrict__ u,
                double* __restrict__ v, double* __restrict__ w) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int i = blockIdx.z;
    if (k >= d.nz || j >= d.ny) return;
    const long long q = idx(d, i, j, k);
    const double c = DP[q];
    const double gx = (c - DP[idx(d, wrap(i - 1, d.nx), j, k)]) * dxi;
    const double gy = (c - DP[idx(d, i, wrap(j - 1, d.ny), k)]) * dyi;
    const double gz = (c - DP[idx(d, i, j, wrap(k - 1, d.nz))]) * dzi;
    u[q] = fma(-scale, gx, u[q]);  // var.sub_(scale, grad)
    v[q] = fma(-scale, gy, v[q]);
    w[q] = fma(-scale, gz, w[q]);
}

// max|u|, max|v|, max|w|, sum(u^2+v^2+w^2), max|div u| (and, with DISS, the
// sum of S_ij S_ij of the cell-centred strain rate): 32 x 8 threads per tile of
// a plane, V cells in z per thread (16-byte loads), maxima as integers.
// out[3] = TKE = 0.5 <u^2 + v^2 + w^2>, out[5] = 2 nu <S_ij S_ij>.  INFO (step
// graphs): out[5..9] = max_res, iterations, status of the solve in sc, += its
// iterations, += 1; with unless_redo nothing where sc->redo says that the step
// is not finished.  24.5 -> 18 us at 128^3 and 11.0 -> 8 at 64^3 against one
// warp per row of cells with NaN-propagating floating-point maxima and a
// reduction per value.
template <int V, bool DISS, bool INFO>
__global__ void __launch_bounds__(kBlock, DISS ? 2 : 4)
stats_kernel(Dims d, int tz, int ty, long long ntiles, BicgScalars* sc, double* part,
             const double* __restrict__ u, const double* __restrict__ v,
             const double* __restrict__ w, double dxi, double dyi, double dzi, double nu,
             int mixed, int unless_redo, double* out) {
    constexpr int NC = DISS ? 6 : 5;
    __shared__ double sh[48], f[6];
    if (INFO && unless_redo && sc->redo) return;
    double mu_ = 0, mv = 0, mw = 0, s = 0, md = 0, ss = 0;
    const long long plane = (long long)d.ny * d.nz;
    for (long long t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const int t1 = (int)(t / tz), i = t1 / ty;
        const int k = ((int)(t - (long long)t1 * tz) * 32 + threadIdx.x) * V;
        const int j = (t1 - i * ty) * 8 + threadIdx.y;
        if (k >= d.nz || j >= d.ny) continue;
        const long long row = i * plane + (long long)j * d.nz, q = row + k;
        const Cells<V> a = ld_cells<V>(u + q), b = ld_cells<V>(v + q), c = ld_cells<V>(w + q);
        const Cells<V> ax = ld_cells<V>(u + wrap(i + 1, d.nx) * plane + (long long)j * d.nz + k);
        const Cells<V> by = ld_cells<V>(v + i * plane + (long long)wrap(j + 1, d.ny) * d.nz + k);
        const double cz = w[row + wrap(k + V, d.nz)];
#pragma unroll
        for (int m = 0; m < V; ++m) {
            mu_ = absmax(mu_, abs_bits(a.a[m]));
            mv = absmax(mv, abs_bits(b.a[m]));
            mw = absmax(mw, abs_bits(c.a[m]));
            s += (a.a[m] * a.a[m] + b.a[m] * b.a[m]) + c.a[m] * c.a[m];
            double dv = (ax.a[m] - a.a[m]) * dxi;
            dv += (by.a[m] - b.a[m]) * dyi;
            dv += ((m + 1 < V ? c.a[m + 1 < V ? m + 1 : m] : cz) - c.a[m]) * dzi;
            md = absmax(md, abs_bits(dv));
            if (DISS) {
                const Grad9 g = grad_center(d, u, v, w, i, j, k + m, dxi, dyi, dzi);
                const double s12 = 0.5 * (g.uy + g.vx);
                const double s13 = 0.5 * (g.uz + g.wx);
                const double s23 = 0.5 * (g.vz + g.wy);
                ss += ((g.ux * g.ux + g.vy * g.vy) + g.wz * g.wz) +
                      2.0 * ((s12 * s12 + s13 * s13) + s23 * s23);
            }
        }
    }
    double red[NC];
    red[0] = mu_; red[1] = mv; red[2] = mw; red[3] = s; red[4] = md;
    if constexpr (DISS) red[5] = ss;
    if (grid_reduce<NC, 0x17u>(red, sc, part, kPassBlocks, sh, f)) {
        if (tid0()) {
            out[0] = f[0]; out[1] = f[1]; out[2] = f[2];
            out[3] = f[3] / double(d.n) * 0.5;
            out[4] = f[4];
            if (DISS) out[5] = 2.0 * nu * (f[5] / double(d.n));
            if (INFO) {
                const double it = double(mixed ? sc->total : sc->iter);
                out[5] = sc->max_res;
                out[6] = it;
                out[7] = double(sc->status);
                out[8] += it;
                out[9] += 1.0;
            }
            sc->counter = 0u;
        }
    }
}

size_t stats_ws_bytes(const pf_grid*) {
    return align256(sizeof(BicgScalars)) + align256(6 * kMaxPartials * sizeof(double));
}

template <bool DISS, bool INFO>
static void launch_stats_kernel(const char* name, const pf_grid* g, const double* u,
                                const double* v, const double* w, double nu, BicgScalars* sc,
                                double* part, int mixed, int unless_redo, double* out,
                                cudaStream_t s) {
    const Dims d{g->nx, g->ny, g->nz, (long long)g->nx * g->ny * g->nz};
    const double dxi = 1.0 / g->dx, dyi = 1.0 / g->dy, dzi = 1.0 / g->dz;
    const bool vec = g->nz % 2 == 0 && (((uintptr_t)u | (uintptr_t)v | (uintptr_t)w) & 15) == 0;
    const int zt = vec ? 64 : 32, tz = (g->nz + zt - 1) / zt, ty = (g->ny + 7) / 8;
    const long long nt = (long long)tz * ty * g->nx;
    const int nb = (int)std::min<long long>(nt, kPassBlocks);
    if (vec)
        PF_LAUNCH(name, s, stats_kernel<2, DISS, INFO><<<nb, dim3(32, 8), 0, s>>>(
            d, tz, ty, nt, sc, part, u, v, w, dxi, dyi, dzi, nu, mixed, unless_redo, out));
    else
        PF_LAUNCH(name, s, stats_kernel<1, DISS, INFO><<<nb, dim3(32, 8), 0, s>>>(
            d, tz, ty, nt, sc, part, u, v, w, dxi, dyi, dzi, nu, mixed, unless_redo, out));
}

static cudaError_t launch_stats_impl(const pf_grid* g, const double* u, const double* v,
                                     const double* w, bool diss, double nu, double* out,
                                     void* ws, cudaStream_t s) {
    Dims d{g->nx, g->ny, g->nz, (long long)g->nx * g->ny * g->nz};
    char* ptr = (char*)ws;
    BicgScalars* sc = (BicgScalars*)ptr; ptr += align256(sizeof(BicgScalars));
    double* part = (double*)ptr;
    cudaMemsetAsync(sc, 0, sizeof(BicgScalars), s);
    if (diss) launch_stats_kernel<true, false>("flow_stats", g, u, v, w, nu, sc, part, 0, 0, out, s);
    else launch_stats_kernel<false, false>("stats", g, u, v, w, 0.0, sc, part, 0, 0, out, s);
    return cudaGetLastError();
}

// A step graph's statistics: sc and part are the solver's (their contents but
// the solve's result are spent by then).
static void launch_step_stats(const pf_grid* g, const double* u, const double* v, const double* w,
                              BicgScalars* sc, double* part, bool mixed, bool unless_redo,
                              double* out, cudaStream_t s) {
    launch_stats_kernel<false, true>("stats", g, u, v, w, 0.0, sc, part, mixed, unless_redo, out, s);
}

cudaError_t launch_stats(const pf_grid* g, const double* u, const double* v,
                         const double* w, double* out, void* ws, cudaStream_t s) {
    return launch_stats_impl(g, u, v, w, false, 0.0, out, ws, s);
}

cudaError_t launch_flow_stats(const pf_grid* g, const double* u, const double* v,
                              const double* w, double nu, double* out, void* ws,
                              cudaStream_t s) {
    return launch_stats_impl(g, u, v, w, true, nu, out, ws, s);
}

static dim3 cgrid(const Dims& d) { return dim3((d.nz + 31) / 32, (d.ny + 7) / 8, d.nx); }

cudaError_t launch_div(const pf_grid* g, const double* u, const double* v,
                       const double* w, double* div, cudaStream_t s) {
    Dims d{g->nx, g->ny, g->nz, (long long)g->nx * g->ny * g->nz};
    PF_LAUNCH("div_vel", 0, div_kernel<<<cgrid(d), dim3(32, 8), 0, s>>>(d, u, v, w, 1.0 / g->dx, 1.0 / g->dy, 1.0 / g->dz, div));
    return cudaGetLastError();
}

cudaError_t launch_laplace(const pf_grid* g, const double* A, double* B, cudaStream_t s) {
    Dims d{g->nx, g->ny, g->nz, (long long)g->nx * g->ny * g->nz};
    PF_LAUNCH("laplace_apply", 0, laplace_kernel<<<cgrid(d), dim3(32, 8), 0, s>>>(d, lap_coef<double>(g), A, B));
    return cudaGetLastError();
}

cudaError_t launch_vel_corr(const pf_grid* g, const double* DP, double scale,
                            double* u, double* v, double* w, cudaStream_t s) {
    Dims d{g->nx, g->ny, g->nz, (long long)g->nx * g->ny * g->nz};
    PF_LAUNCH("vel_corr", 0, vel_corr_kernel<<<cgrid(d), dim3(32, 8), 0, s>>>(d, DP, scale, 1.0 / g->dx, 1.0 / g->dy,
                                                     1.0 / g->dz, u, v, w));
    return cudaGetLastError();
}


// Projection of a velocity field (pf_project): statistics, divergence, direct
// solve and its check go out together and the host waits once for all of
// their results; then the correction.
int project_solve(const pf_grid* g, double* u, double* v, double* w, double* DP, double* p,
                  double rho, double dt, double min_res, int max_it, void* ws, cudaStream_t s,
                  pf_solve_info* info, int* skipped) {
    const Dims d{g->nx, g->ny, g->nz, (long long)g->nx * g->ny * g->nz};
    const size_t n = (size_t)d.n;
    double* div = (double*)ws;
    char* ptr = (char*)ws + align256(n * sizeof(double));
    char* rest = ptr;
    BicgScalars* sc = (BicgScalars*)ptr; ptr += align256(sizeof(BicgScalars));
    double* part = (double*)ptr; ptr += align256(kNumPartials * kMaxPartials * sizeof(double));
    const double vol = (g->dx * g->dy) * g->dz;
    const double hmin = std::min(g->dx, std::min(g->dy, g->dz));
    struct { BicgScalars sc; char pad[192 - sizeof(BicgScalars)]; double st[5]; } h;
    double* st = (double*)((char*)sc + 192);  // behind the scalars, in their 256 bytes
    static_assert(sizeof(BicgScalars) <= 192, "scalar block");
    const bool direct = spectral_applies(g, min_res, DP, ptr);
    if (cudaMemsetAsync(sc, 0, sizeof(BicgScalars), s) != cudaSuccess) return PF_ERR_CUDA;
    launch_stats_kernel<false, false>("stats", g, u, v, w, 0.0, sc, part, 0, 0, st, s);
    launch_div(g, u, v, w, div, s);
    if (direct) {
        SpectralPlan sp;
        if (spectral_setup(g, ptr, &sp) != cudaSuccess ||
            spectral_enqueue_tables(sp, s) != cudaSuccess ||
            spectral_enqueue_solve(sp, div, rho / dt * (-1.0 * vol), DP, &sc->nonfin, s) != cudaSuccess)
            return PF_ERR_CUDA;
        ProjectArgs A{};
        A.sc = sc; A.part = part; A.src = div; A.c1 = rho / dt; A.c2 = -1.0 * vol;
        A.min_res = min_res; A.max_it = std::max(max_it, 1); A.DP = DP;
        launch_project<true, false>("spectral_check", g, A, s);
    }
    if (cudaGetLastError() != cudaSuccess ||
        cudaMemcpyAsync(&h, sc, sizeof(h), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
        return PF_ERR_CUDA;
    const double vmax = std::max(h.st[0], std::max(h.st[1], h.st[2]));
    *skipped = h.st[4] <= 1e-9 * vmax / hmin;
    *info = pf_solve_info{0.0, 0, 1, PF_OK};
    if (*skipped)
        return cudaMemsetAsync(DP, 0, n * sizeof(double), s) == cudaSuccess ? PF_OK : PF_ERR_CUDA;
    if (direct && h.sc.done && h.sc.status == PF_OK) {
        info->max_res = h.sc.max_res;
        info->iterations = h.sc.total;
        ProjectArgs A{};
        A.DP = DP; A.scale = dt / rho;
        A.u = u; A.v = v; A.w = w; A.p = p;
        launch_project<false, true>("project", g, A, s);
        return cudaGetLastError() == cudaSuccess ? PF_OK : PF_ERR_CUDA;
    }
    // what the direct solve does not settle: the whole solve with its iterations
    const int rc = bicgstab_solve(g, PF_FP64, rho, dt, min_res, max_it, div, DP, p, rest, s, info);
    if (rc) return rc;
    if (info->status == PF_NONFINITE) return PF_OK;
    return launch_vel_corr(g, DP, dt / rho, u, v, w, s) == cudaSuccess ? PF_OK : PF_ERR_CUDA;
}

// ============================================================================
// Whole time step as one CUDA graph.
//
// The step (predictor, divergence, Poisson solve, p += DP, projection,
// statistics) is captured once per plan; the BiCGStab iteration loop is a
// conditional WHILE node whose body is (kernel B, kernel CA): kernel CA clears
// the condition when the solve stops (converged, iteration limit, breakdown,
// non-finite), so a whole step runs without any host synchronisation.  The
// mixed-precision refinement is an outer WHILE node (inner pass, fold,
// FP64 residual, control) cleared by the control kernel.  A pass that ends
// non-finite or in breakdown is discarded and ends the solve with that status
// (the host-driven solve switches to FP64 passes instead).  Every kernel that
// can find the solve already stopped clears the condition as well, so each
// loop ends after at most max_it iterations.
// ============================================================================

// Refinement control (one thread): after the FP64 residual of a pass, count the
// pass and its inner iterations and decide whether another pass runs, with
// the host-driven solve's rules: an FP32 pass that ended non-finite or in
// breakdown was discarded (its fold skipped) and the solve continues with
// FP64 passes, as it does once two FP32 passes in a row gain less than 2x.
// gated: nothing while the pass is running, and FP64 passes are left to the
// IF node of handle if64.
__global__ void mixed_control(BicgScalars* sc, double min_res, int max_outer,
                              int max_it, cudaGraphConditionalHandle cond, int gated = 0,
                              cudaGraphConditionalHandle if64 = 0) {
    if (threadIdx.x != 0 || blockIdx.x != 0 || (gated && !sc->done)) return;
    sc->outer += 1;
    sc->total += sc->iter;
    // max|b| == 0: nothing to solve; a NaN max|b| gives a NaN ratio
    const double ratio = sc->max_b == 0.0 ? 0.0 : sc->true_res / sc->max_b;
    const int pass = sc->status;  // status of the inner pass just run
    const bool failed32 = !sc->use64 && (pass == PF_NONFINITE || pass == PF_BREAKDOWN);
    bool stop = true;
    if (sc->use64 && pass == PF_NONFINITE) sc->status = PF_NONFINITE;
    else if (!(ratio == ratio) || isinf(ratio)) sc->status = PF_NONFINITE;
    else if (ratio <= min_res) sc->status = PF_OK;
    else if (sc->outer >= max_outer || sc->total >= max_it) sc->status = PF_MAXIT;
    else stop = false;
    if (!stop) {
        if (failed32 || (!sc->use64 && sc->outer > 1 && ratio > 0.5 * sc->prev_ratio))
            sc->use64 = 1;
        sc->prev_ratio = ratio;
    }
    sc->max_res = ratio;
    const bool leave = gated && !stop && sc->use64;
    if (stop || leave) cudaGraphSetConditional(cond, 0);
    if (leave) cudaGraphSetConditional(if64, 1);
}

// Start of a refinement pass: choose the FP64 or the FP32 pass.
__global__ void pass_branch(const BicgScalars* sc, cudaGraphConditionalHandle if64) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    cudaGraphSetConditional(if64, sc->use64 ? 1u : 0u);
}

// An FP64 pass finishes the solve: its inner tolerance is the remaining
// reduction (set after bicg_init, before the first kernel CA reads it).
__global__ void pass_tol64(BicgScalars* sc, double min_res) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const double ratio = sc->max_b == 0.0 ? 0.0 : sc->true_res / sc->max_b;
    sc->min_res = ratio > 0.0 ? fmin(0.5, 0.5 * min_res / ratio) : 0.5;
}

// x += scale * e of the pass just run (its precision is sc->use64); an FP32
// pass that ended non-finite or in breakdown is discarded.
__global__ void __launch_bounds__(kBlock)
fold_mixed(Dims d, const BicgScalars* sc, const float* e32, const double* e64, double* x,
           int gated = 0) {
    if (gated && !sc->done) return;  // the pass is still running
    const bool f64 = sc->use64 != 0;
    if (!f64 && (sc->status == PF_NONFINITE || sc->status == PF_BREAKDOWN)) return;
    if (f64 && sc->status == PF_NONFINITE) return;
    if (sc->iter == 0) return;  // no iteration ran: e = 0, possibly unwritten
    const double s = sc->scale;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < d.n;
         q += (long long)gridDim.x * blockDim.x)
        x[q] = x[q] + s * (f64 ? e64[q] : double(e32[q]));
}

struct StepPlan {
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
};

static int capture_begin(cudaStream_t cs, cudaGraph_t target) {
    cudaError_t e = target ? cudaStreamBeginCaptureToGraph(cs, target, nullptr, nullptr, 0,
                                                          cudaStreamCaptureModeThreadLocal)
                           : cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
    return e == cudaSuccess ? PF_OK : PF_ERR_CUDA;
}

static int capture_end(cudaStream_t cs, cudaGraph_t* g) {
    return cudaStreamEndCapture(cs, g) == cudaSuccess ? PF_OK : PF_ERR_CUDA;
}

// Re-arms a WHILE condition (the default value is applied only when the
// whole graph is launched, not each time a nested loop is entered).
__global__ void arm_condition(cudaGraphConditionalHandle h) {
    if (threadIdx.x == 0 && blockIdx.x == 0) cudaGraphSetConditional(h, 1);
}

// Adds a WHILE node after `dep` whose body is returned in *body.  With
// `make_handle` the handle (default 1 at every graph launch) is created here
// and written to *handle; otherwise *handle is used as given.
static int add_while(cudaGraph_t g, cudaGraphNode_t dep, cudaGraphNode_t* node,
                     cudaGraph_t* body, cudaGraphConditionalHandle* handle,
                     bool make_handle = true) {
    if (make_handle &&
        cudaGraphConditionalHandleCreate(handle, g, 1, cudaGraphCondAssignDefault) != cudaSuccess)
        return PF_ERR_CUDA;
    cudaGraphNodeParams prm = {cudaGraphNodeTypeConditional};
    prm.conditional.handle = *handle;
    prm.conditional.type = cudaGraphCondTypeWhile;
    prm.conditional.size = 1;
    if (cudaGraphAddNode(node, g, dep ? &dep : nullptr, dep ? 1 : 0, &prm) != cudaSuccess)
        return PF_ERR_CUDA;
    *body = prm.conditional.phGraph_out[0];
    return PF_OK;
}

static int add_child(cudaGraph_t g, cudaGraphNode_t dep, cudaGraph_t child,
                     cudaGraphNode_t* node) {
    return cudaGraphAddChildGraphNode(node, g, dep ? &dep : nullptr, dep ? 1 : 0, child) ==
                   cudaSuccess ? PF_OK : PF_ERR_CUDA;
}

// Plan workspace: [div: n doubles][scalar block][reduction partials][region R]
// R holds, at different times of the step, the predictor's stage buffers, the
// solver vectors and the statistics scratch.  The scalar block is written only
// by the solver kernels.
static constexpr size_t kPlanPinvBytes = (size_t)kMgPinvMax * kMgPinvMax * sizeof(float);

size_t step_plan_ws_bytes(const pf_grid* g, int prec) {
    const size_t n = (size_t)g->nx * g->ny * g->nz;
    size_t vecs = prec == PF_FP64 ? 8 * align256(n * sizeof(double))
                                  : 11 * align256(n * sizeof(double));
    size_t r = std::max(std::max(predictor_ws_bytes(g, prec), vecs), stats_ws_bytes(g));
    // PF_MIXED_MG: the coarsest level's pseudo-inverse in a slot of its own
    // (the region r is reused by the predictor every step), computed once
    const size_t pinv = prec == PF_MIXED_MG ? kPlanPinvBytes + kMgBarrierBytes : 0;
    // mixed forms: the direct solve's tables, filled once too
    const size_t tables = prec == PF_FP64 ? 0 : spectral_table_bytes(g);
    return align256(n * sizeof(double)) + align256(sizeof(BicgScalars)) +
           align256(kNumPartials * kMaxPartials * sizeof(double)) + align256(r) + tables + pinv;
}

// Pointers of one request's plan workspace (see step_plan_ws_bytes).
struct PlanLayout {
    Dims d;
    double* div;
    BicgScalars* sc;
    double* part;
    char* R;
    BicgVecs<double> v64;
    BicgVecs<float> v32;
    float* e32;
    double *bb, *rr;
    MgPlan mg;
    SpectralPlan sp;  // on: the direct solve, with FP64 passes behind it
};

// The two slots at the end of a plan's workspace that are filled once: the
// direct solve's tables, then the coarsest pseudo-inverse and the grid-barrier
// words.  (The region R is rewritten every step.)
static char* plan_tables(const pf_grid* g, int prec, void* ws) {
    return (char*)ws + step_plan_ws_bytes(g, prec) - spectral_table_bytes(g) -
           (prec == PF_MIXED_MG ? kPlanPinvBytes + kMgBarrierBytes : 0);
}

// PF_MIXED_MG: the multigrid of grids that coarsen, its vectors in region R.
static int plan_mg(const pf_grid* g, int prec, void* ws, char* R, MgPlan* mg) {
    const size_t n = (size_t)g->nx * g->ny * g->nz;
    if (prec != PF_MIXED_MG || mg_region_bytes(g) > 9 * align256(n * sizeof(double))) return PF_OK;
    const int e = mg_setup(g, R, mg);
    if (e != PF_OK && e != PF_ERR_BAD_ARG) return e;
    char* end = (char*)ws + step_plan_ws_bytes(g, prec);
    if (mg->L && mg->pinv) mg->pinv = (float*)(end - kPlanPinvBytes - kMgBarrierBytes);
    if (mg->L) mg->gbar = (unsigned*)(end - kMgBarrierBytes);
    return PF_OK;
}

static int plan_layout(const pf_grid* g, int prec, double min_res, const double* DP, void* ws,
                       PlanLayout* L) {
    L->d = Dims{g->nx, g->ny, g->nz, (long long)g->nx * g->ny * g->nz};
    const size_t n = (size_t)L->d.n;
    char* ptr = (char*)ws;
    L->div = (double*)ptr; ptr += align256(n * sizeof(double));
    L->sc = (BicgScalars*)ptr; ptr += align256(sizeof(BicgScalars));
    L->part = (double*)ptr; ptr += align256(kNumPartials * kMaxPartials * sizeof(double));
    L->R = ptr;
    // FP64 vectors, or FP32 vectors + correction followed by b and r (FP64)
    char* vp = L->R;
    L->v64 = carve<double>(vp, n);
    vp = L->R;
    L->v32 = carve<float>(vp, n);
    L->e32 = (float*)vp;
    L->bb = (double*)(L->R + 9 * align256(n * sizeof(double)));
    L->rr = (double*)(L->R + 10 * align256(n * sizeof(double)));
    L->mg = MgPlan();
    L->sp = SpectralPlan();
    if (prec != PF_FP64 && !mg_cycles_serve(g, prec)) {
        char* tables = plan_tables(g, prec, ws);
        if (spectral_applies(g, min_res, DP, tables))
            return spectral_setup(g, tables, &L->sp) == cudaSuccess ? PF_OK : PF_ERR_CUDA;
    }
    return plan_mg(g, prec, ws, L->R, &L->mg);
}

// Fills what the solvers keep in the workspace of a plan: for every solver that
// serves the grid, not only the one P chose, since a later plan of the same
// member (fresh == 0, nothing filled then) may choose another, by its tolerance
// or PF_MG_COOP.
static int plan_fill(const pf_grid* g, int prec, const double* DP, void* ws, const PlanLayout& P,
                     cudaStream_t s) {
    if (prec == PF_FP64) return PF_OK;
    SpectralPlan sp;
    MgPlan mg;
    char* tables = plan_tables(g, prec, ws);
    if (spectral_applies(g, kSpectralMinTol, DP, tables) &&
        (spectral_setup(g, tables, &sp) != cudaSuccess ||
         spectral_enqueue_tables(sp, s) != cudaSuccess))
        return PF_ERR_CUDA;
    const int rc = plan_mg(g, prec, ws, P.R, &mg);
    if (rc != PF_OK) return rc;
    return mg.L ? mg_enqueue_setup(mg, s) : PF_OK;
}

// The monitor statistics with the solve's result next to them, after node
// `dep`; unless_redo: nothing, where the iterations behind the direct solve run.
static int add_stats(cudaGraph_t G, cudaGraphNode_t dep, const pf_grid* g, PlanLayout& P,
                     const double* u, const double* v, const double* w, bool mixed,
                     bool unless_redo, double* stats, cudaStream_t cs, cudaGraphNode_t* end) {
    int rc;
    cudaGraph_t seg = nullptr;
    if ((rc = capture_begin(cs, nullptr))) return rc;
    launch_step_stats(g, u, v, w, P.sc, P.part, mixed, unless_redo, stats, cs);
    if ((rc = capture_end(cs, &seg))) return rc;
    rc = add_child(G, dep, seg, end);
    cudaGraphDestroy(seg);
    return rc;
}

// After the solve (node `dep`): p += DP, the projection, the statistics.
static int add_step_end(cudaGraph_t G, cudaGraphNode_t dep, const pf_grid* g, PlanLayout& P,
                        double* u, double* v, double* w, double* p, double* DP, double rho,
                        double dt, bool mixed, double* stats, cudaStream_t cs,
                        cudaGraphNode_t* end) {
    int rc;
    cudaGraph_t seg = nullptr;
    if ((rc = capture_begin(cs, nullptr))) return rc;
    ProjectArgs A{};
    A.DP = DP; A.scale = dt / rho;
    A.u = u; A.v = v; A.w = w; A.p = p;
    launch_project<false, true>("project", g, A, cs);
    if ((rc = capture_end(cs, &seg))) return rc;
    cudaGraphNode_t np;
    rc = add_child(G, dep, seg, &np);
    cudaGraphDestroy(seg);
    return rc ? rc : add_stats(G, np, g, P, u, v, w, mixed, false, stats, cs, end);
}

// Adds one request's step after the predictor (node `dep`) to graph G:
// divergence and solver set-up, the solver's WHILE loop(s), then p += DP,
// the projection and the monitor statistics.  *end gets the last node.
static int add_solve_chain(cudaGraph_t G, cudaGraphNode_t dep, const pf_grid* g, int prec,
                           PlanLayout& P, double* u, double* v, double* w, double* p,
                           double* DP, double rho, double dt, double min_res, int max_it,
                           double* stats, bool alone, cudaStream_t cs, cudaGraphNode_t* end) {
    const Dims d = P.d;
    BicgScalars* sc = P.sc;
    double* part = P.part;
    const int gp = pointwise_grid(d.n);
    const double vol = (g->dx * g->dy) * g->dz;
    const double c1 = rho / dt, c2 = -1.0 * vol;
    max_it = std::max(max_it, 1);
    dim3 blk2(32, 8);
    int rc = PF_OK;
    // the FP64 solve in one cooperative launch, unless it is one of several
    // parallel branches (their blocks could wait on one another for room)
    const bool one_launch = prec == PF_FP64 && alone && tile_solve_applies(d);
    // ---- divergence, solver set-up
    cudaGraph_t seg1 = nullptr;
    cudaGraph_t C = G;        // the graph that holds the solver's loops
    cudaGraphNode_t nsolved;  // the node after which DP is final
    cudaGraphConditionalHandle hmore = 0;
    if (P.sp.on && cudaGraphConditionalHandleCreate(&hmore, G, 0, cudaGraphCondAssignDefault) !=
                       cudaSuccess)
        return PF_ERR_CUDA;
    if ((rc = capture_begin(cs, nullptr))) return rc;
    launch_div(g, u, v, w, P.div, cs);
    if (P.sp.on) {
        // the direct solve, its check and the correction; beside the statistics
        // an IF node that the check opens: correction taken back, the
        // refinement loop below with FP64 passes only, and the step's end again
        spectral_enqueue_solve(P.sp, P.div, c1 * c2, DP, &sc->nonfin, cs);
        ProjectArgs A{};
        A.sc = sc; A.part = part; A.src = P.div; A.c1 = c1; A.c2 = c2;
        A.min_res = min_res; A.max_it = max_it; A.DP = DP; A.scale = dt / rho;
        A.u = u; A.v = v; A.w = w; A.p = p;
        A.use_cond = 1; A.cond = hmore;
        launch_project<true, true>("project_check", g, A, cs);
        if ((rc = capture_end(cs, &seg1))) return rc;
        cudaGraphNode_t ns;
        rc = add_child(G, dep, seg1, &ns);
        cudaGraphDestroy(seg1);
        if (rc) return rc;
        if ((rc = add_stats(G, ns, g, P, u, v, w, true, true, stats, cs, end))) return rc;
        cudaGraphNodeParams prm = {cudaGraphNodeTypeConditional};
        prm.conditional.handle = hmore;
        prm.conditional.type = cudaGraphCondTypeIf;
        prm.conditional.size = 1;
        cudaGraphNode_t nif;
        if (cudaGraphAddNode(&nif, G, &ns, 1, &prm) != cudaSuccess) return PF_ERR_CUDA;
        C = prm.conditional.phGraph_out[0];
        dep = nullptr;
        if ((rc = capture_begin(cs, nullptr))) return rc;
        project_undo<<<cgrid(d), dim3(32, 8), 0, cs>>>(d, DP, dt / rho, 1.0 / g->dx, 1.0 / g->dy,
                                                      1.0 / g->dz, u, v, w, p);
    }
    if (prec == PF_FP64) {
        const LapCoef<double> cf = lap_coef<double>(g);
        const Tiling ta = make_tiling(d, 8 * PhaseCA<double>::R);
        bicg_init<double, false><<<gp, kBlock, 0, cs>>>(d, sc, part, P.div, c1, c2, P.v64, DP,
                                                       max_it, min_res);
        if (one_launch) {
            const cudaError_t e = launch_tile_solve(d, cf, sc, part, P.v64, DP, cs);
            if ((rc = capture_end(cs, &seg1))) return rc;
            if (e == cudaSuccess) rc = add_child(G, dep, seg1, &nsolved);
            cudaGraphDestroy(seg1);
            if (e != cudaSuccess || rc) return PF_ERR_CUDA;
            return add_step_end(G, nsolved, g, P, u, v, w, p, DP, rho, dt, false, stats, cs, end);
        }
        bicg_ca<double><<<tiled_grid(ta), blk2, 0, cs>>>(d, ta, cf, sc, part, P.v64, DP);
    } else {
        // the refinement starts from the previous step's DP (zero before the
        // first step): its first residual is r = b - A DP, and the stop test
        // stays the reference's, max|b - A DP| <= min_res max|b|
        const Tiling tld = make_tiling(d, 8 * PhaseResidual::R);
        if (P.sp.on)
            scaled_source<<<gp, kBlock, 0, cs>>>(d.n, P.div, c1, c2, P.bb);
        else
            mixed_b_init<<<gp, kBlock, 0, cs>>>(d, sc, part, P.div, c1, c2, P.bb, nullptr, nullptr);
        mixed_residual<<<tiled_grid(tld), blk2, 0, cs>>>(d, tld, lap_coef<double>(g), sc, part,
                                                        P.bb, DP, P.rr);
    }
    if ((rc = capture_end(cs, &seg1))) return rc;
    cudaGraphNode_t n1, nw;
    rc = add_child(C, dep, seg1, &n1);
    cudaGraphDestroy(seg1);
    if (rc) return rc;
    cudaGraph_t body;
    cudaGraphConditionalHandle h;
    if ((rc = add_while(C, n1, &nw, &body, &h))) return rc;
    nsolved = nw;
    if (prec == PF_FP64) {
        const LapCoef<double> cf = lap_coef<double>(g);
        const Tiling ta = make_tiling(d, 8 * PhaseCA<double>::R);
        const Tiling tb = make_tiling(d, 8 * PhaseB<double>::R);
        if ((rc = capture_begin(cs, body))) return rc;
        bicg_b<double><<<tiled_grid(tb), blk2, 0, cs>>>(d, tb, cf, sc, part, P.v64, 1, h);
        bicg_ca<double><<<tiled_grid(ta), blk2, 0, cs>>>(d, ta, cf, sc, part, P.v64, DP, 1, h);
        if ((rc = capture_end(cs, &body))) return rc;
    } else {
        const LapCoef<float> cf = lap_coef<float>(g);
        const LapCoef<double> cfd = lap_coef<double>(g);
        const Tiling ta = make_tiling(d, 8 * PhaseCA<float>::R);
        const Tiling tb = make_tiling(d, 8 * PhaseB<float>::R);
        const Tiling tld = make_tiling(d, 8 * PhaseResidual::R);
        const double kInnerTol = 1e-4;
        const MgPlan& mg = P.mg;
        float* ecorr = mg.L ? mg.e : P.e32;
        // FP64 inner vectors (the same region: a pass uses one set)
        char* r64 = P.R;
        BicgVecs<double> v64 = carve<double>(r64, (size_t)d.n);
        double* e64 = (double*)r64;
        const LapCoef<double> cf64 = lap_coef<double>(g);
        const Tiling ta64 = make_tiling(d, 8 * PhaseCA<double>::R);
        const Tiling tb64 = make_tiling(d, 8 * PhaseB<double>::R);
        // a one-thread kernel node: func(args...) with the given argument list
        auto add_tiny = [](cudaGraph_t gr, void* func, void** args, cudaGraphNode_t* node) {
            cudaKernelNodeParams kp;
            std::memset(&kp, 0, sizeof(kp));
            kp.func = func;
            kp.gridDim = dim3(1);
            kp.blockDim = dim3(32);
            kp.kernelParams = args;
            return cudaGraphAddKernelNode(node, gr, nullptr, 0, &kp) == cudaSuccess ? PF_OK
                                                                                     : PF_ERR_CUDA;
        };
        // One pass in graph `gr`: re-arm its loop, set-up, then the inner
        // WHILE (its handle belongs to the graph that holds the loop).  The
        // FP64 pass runs to the remaining tolerance.
        auto add_pass = [&](cudaGraph_t gr, bool f64, cudaGraphNode_t* cw) -> int {
            cudaGraph_t pre = nullptr, inner_body = nullptr;
            cudaGraphNode_t a0, c1n;
            cudaGraphConditionalHandle hp;
            if (cudaGraphConditionalHandleCreate(&hp, gr, 1, cudaGraphCondAssignDefault) !=
                cudaSuccess)
                return PF_ERR_CUDA;
            void* args[] = {&hp};
            int rc = add_tiny(gr, (void*)arm_condition, args, &a0);
            if (rc || (rc = capture_begin(cs, nullptr))) return rc;
            if (f64) {
                bicg_init<double, true><<<gp, kBlock, 0, cs>>>(d, sc, part, P.rr, 0.0, 0.0, v64,
                                                              e64, max_it, 0.5);
                pass_tol64<<<1, 32, 0, cs>>>(sc, min_res);
                bicg_ca<double><<<tiled_grid(ta64), blk2, 0, cs>>>(d, ta64, cf64, sc, part, v64,
                                                                  e64);
            } else {
                bicg_init<float, true><<<gp, kBlock, 0, cs>>>(d, sc, part, P.rr, 0.0, 0.0, P.v32,
                                                             P.e32, max_it, kInnerTol);
                bicg_ca<float><<<tiled_grid(ta), blk2, 0, cs>>>(d, ta, cf, sc, part, P.v32,
                                                               P.e32);
            }
            if ((rc = capture_end(cs, &pre))) return rc;
            rc = add_child(gr, a0, pre, &c1n);
            cudaGraphDestroy(pre);
            if (rc) return rc;
            if ((rc = add_while(gr, c1n, cw, &inner_body, &hp, false))) return rc;
            if ((rc = capture_begin(cs, inner_body))) return rc;
            if (f64) {
                bicg_b<double><<<tiled_grid(tb64), blk2, 0, cs>>>(d, tb64, cf64, sc, part, v64, 1,
                                                                 hp);
                bicg_ca<double><<<tiled_grid(ta64), blk2, 0, cs>>>(d, ta64, cf64, sc, part, v64,
                                                                  e64, 1, hp);
            } else {
                bicg_b<float><<<tiled_grid(tb), blk2, 0, cs>>>(d, tb, cf, sc, part, P.v32, 1, hp);
                bicg_ca<float><<<tiled_grid(ta), blk2, 0, cs>>>(d, ta, cf, sc, part, P.v32,
                                                               P.e32, 1, hp);
            }
            return capture_end(cs, &inner_body);
        };
        // The refinement loop with FP64 passes in graph `lg` (body of a WHILE
        // whose handle is `lh`): pass, fold, residual, control.
        auto add_loop = [&](cudaGraph_t lg, cudaGraphConditionalHandle lh, cudaGraphNode_t np) -> int {
            cudaGraph_t post = nullptr;
            cudaGraphNode_t b3;
            int rc = capture_begin(cs, nullptr);
            if (rc) return rc;
            fold_mixed<<<gp, kBlock, 0, cs>>>(d, sc, ecorr, e64, DP);
            mixed_residual<<<tiled_grid(tld), blk2, 0, cs>>>(d, tld, cfd, sc, part, P.bb, DP, P.rr);
            mixed_control<<<1, 32, 0, cs>>>(sc, min_res, 40, max_it, lh);
            if ((rc = capture_end(cs, &post))) return rc;
            rc = add_child(lg, np, post, &b3);
            cudaGraphDestroy(post);
            return rc;
        };
        cudaGraphNode_t np;
        if (P.sp.on) {
            // behind the direct solve only FP64 passes make sense
            if ((rc = add_pass(body, true, &np)) || (rc = add_loop(body, h, np))) return rc;
        } else if (mg.L) {
            // One loop for passes and iterations: each turn starts a pass if none
            // is running, runs two iterations (the p buffers alternate), and ends
            // the pass if it has stopped; kernels whose turn it is not return at
            // once (1 us each).  Against the iterations as a WHILE node in an IF
            // node in the passes' WHILE node, the conditional nodes saved outweigh
            // those: ten 32^3 steps 5.88 ms against 6.02, an ensemble with one such
            // member 8.62 against 8.76 (four steps).  FP64 passes, rare, sit behind
            // the loop in an IF node.
            cudaGraphConditionalHandle hif;
            if (cudaGraphConditionalHandleCreate(&hif, C, 0, cudaGraphCondAssignDefault) != cudaSuccess)
                return PF_ERR_CUDA;
            if ((rc = capture_begin(cs, body))) return rc;
            mg_enqueue_init(mg, sc, part, P.rr, kInnerTol, max_it, cs, min_res, 1);
            mg_enqueue_iteration(mg, sc, part, 0, cs);
            mg_enqueue_iteration(mg, sc, part, 1, cs);
            fold_mixed<<<gp, kBlock, 0, cs>>>(d, sc, ecorr, e64, DP, 1);
            mixed_residual<<<tiled_grid(tld), blk2, 0, cs>>>(d, tld, cfd, sc, part, P.bb, DP, P.rr, 1);
            mixed_control<<<1, 32, 0, cs>>>(sc, min_res, 40, max_it, h, 1, hif);
            if ((rc = capture_end(cs, &body))) return rc;
            cudaGraphNodeParams prm = {cudaGraphNodeTypeConditional};
            prm.conditional.handle = hif;
            prm.conditional.type = cudaGraphCondTypeIf;
            prm.conditional.size = 1;
            if (cudaGraphAddNode(&nsolved, C, &nw, 1, &prm) != cudaSuccess) return PF_ERR_CUDA;
            cudaGraph_t lg, if_body = prm.conditional.phGraph_out[0];
            cudaGraphConditionalHandle lh;
            cudaGraphNode_t nl;
            if ((rc = add_while(if_body, nullptr, &nl, &lg, &lh)) || (rc = add_pass(lg, true, &np)) ||
                (rc = add_loop(lg, lh, np)))
                return rc;
        } else {
            // outer body: branch kernel, IF(use64) {FP64 pass} ELSE {FP32 pass},
            // then fold + residual + control
            cudaGraphConditionalHandle hif;
            if (cudaGraphConditionalHandleCreate(&hif, body, 0, cudaGraphCondAssignDefault) !=
                    cudaSuccess)
                return PF_ERR_CUDA;
            cudaGraphNode_t b0, cw;
            BicgScalars* scp = sc;
            void* args[] = {&scp, &hif};
            if ((rc = add_tiny(body, (void*)pass_branch, args, &b0))) return rc;
            cudaGraphNodeParams prm = {cudaGraphNodeTypeConditional};
            prm.conditional.handle = hif;
            prm.conditional.type = cudaGraphCondTypeIf;
            prm.conditional.size = 2;
            if (cudaGraphAddNode(&np, body, &b0, 1, &prm) != cudaSuccess) return PF_ERR_CUDA;
            if ((rc = add_pass(prm.conditional.phGraph_out[1], false, &cw)) ||
                (rc = add_pass(prm.conditional.phGraph_out[0], true, &cw)) || (rc = add_loop(body, h, np)))
                return rc;
        }
    }
    cudaGraphNode_t last;
    return add_step_end(C, nsolved, g, P, u, v, w, p, DP, rho, dt, prec != PF_FP64, stats, cs,
                        P.sp.on ? &last : end);
}

// Captures the body of `enqueue(cs)` as a child node of G (no dependency).
template <class F>
static int add_captured(cudaGraph_t G, cudaStream_t cs, F enqueue, cudaGraphNode_t* node) {
    cudaGraph_t seg = nullptr;
    int rc = capture_begin(cs, nullptr);
    if (rc) return rc;
    const cudaError_t e = enqueue(cs);
    rc = capture_end(cs, &seg);
    if (rc) return rc;
    if (e != cudaSuccess) { cudaGraphDestroy(seg); return PF_ERR_CUDA; }
    rc = add_child(G, nullptr, seg, node);
    cudaGraphDestroy(seg);
    return rc;
}

static void plan_free(StepPlan* plan) {
    if (plan->exec) cudaGraphExecDestroy(plan->exec);
    if (plan->graph) cudaGraphDestroy(plan->graph);
    delete plan;
}

ClosureLayout closure_layout(const pf_grid* g, int prec, int kind) {
    const size_t n = (size_t)g->nx * g->ny * g->nz;
    const size_t tsz = prec == PF_FP64 ? sizeof(double) : sizeof(float);
    ClosureLayout L{0, 0, 0, 0};
    if (kind == PF_CLOSURE_SMAGORINSKY || kind == PF_CLOSURE_GRADIENT) {
        L.bytes = (kind == PF_CLOSURE_SMAGORINSKY ? 1 : 6) * n * tsz;
        return L;
    }
    // MLP: scales + reduction scratch, the FP64 stresses, their float copy
    L.f64 = align256(256 + mlp_scales_ws_bytes());
    L.stage = L.f64;
    L.bytes = L.f64 + align256(6 * n * sizeof(double));
    if (prec != PF_FP64) {
        L.stage = L.bytes;
        L.bytes += align256(6 * n * sizeof(float));
    }
    return L;
}

// the SFS pre-step of a plan (src/data/domain.py:347-355): the closure's
// field from the fields the previous step left, in the stages' type
static cudaError_t enqueue_closure(const pf_grid* g, int prec, const pf_step_closure* c,
                                   double mu, const double* u, const double* v, const double* w,
                                   cudaStream_t st) {
    char* f = (char*)c->field;
    const bool f32 = prec != PF_FP64;
    if (c->kind != PF_CLOSURE_MLP)
        return launch_sgs(g, c->kind - 1, u, v, w, c->coef,
                          c->kind == PF_CLOSURE_SMAGORINSKY ? mu : 0.0, f, f32, st);
    const ClosureLayout L = closure_layout(g, prec, c->kind);
    float* scales = (float*)f;
    cudaError_t e = launch_mlp_scales(g, u, v, w, c->coef, scales, f + 256, st);
    if (e != cudaSuccess) return e;
    e = launch_mlp(g, u, v, w, c->wpack, scales, (double*)(f + L.f64), c->err, st);
    if (e != cudaSuccess || !f32) return e;
    const long long n6 = 6LL * g->nx * g->ny * g->nz;
    return launch_to_float((const double*)(f + L.f64), (float*)(f + L.stage), n6, st);
}

int step_plan_create(const pf_grid* g, int prec, int rk4, double* u, double* v,
                     double* w, double* p, double* DP, double mu, double rho,
                     double dt, double min_res, int max_it, const pf_step_closure* c,
                     void* ws, double* stats, void** out) {
    PlanLayout P;
    int rc = plan_layout(g, prec, min_res, DP, ws, &P);
    if (rc != PF_OK) return rc;
    if (predictor_prepare(prec) != cudaSuccess) return PF_ERR_CUDA;
    if (c && c->kind == PF_CLOSURE_MLP && mlp_prepare() != cudaSuccess) return PF_ERR_CUDA;
    cudaStream_t cs;
    if (cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking) != cudaSuccess) return PF_ERR_CUDA;
    if (plan_fill(g, prec, DP, ws, P, cs) != PF_OK || cudaStreamSynchronize(cs) != cudaSuccess) {
        cudaStreamDestroy(cs);
        return PF_ERR_CUDA;
    }
    prof_suspend(true);
    StepPlan* plan = new StepPlan();
    do {
        if (cudaGraphCreate(&plan->graph, 0) != cudaSuccess) { rc = PF_ERR_CUDA; break; }
        cudaGraph_t G = plan->graph;
        cudaGraphNode_t n0, nend;
        // the SFS pre-step reads the fields the previous step left; the
        // stages read its field in their own type
        const void* cf = c ? (const char*)c->field + closure_layout(g, prec, c->kind).stage : nullptr;
        const void* visc = c && c->kind == PF_CLOSURE_SMAGORINSKY ? cf : nullptr;
        const void* sfs = c && c->kind != PF_CLOSURE_SMAGORINSKY ? cf : nullptr;
        if ((rc = add_captured(G, cs, [&](cudaStream_t st) {
                 if (c) {
                     const cudaError_t e = enqueue_closure(g, prec, c, mu, u, v, w, st);
                     if (e != cudaSuccess) return e;
                 }
                 return launch_predictor(g, prec, rk4, u, v, w, visc, mu, rho, sfs, dt, P.R, st);
             }, &n0)))
            break;
        if ((rc = add_solve_chain(G, n0, g, prec, P, u, v, w, p, DP, rho, dt, min_res, max_it,
                                  stats, true, cs, &nend)))
            break;
        if (cudaGraphInstantiate(&plan->exec, G, 0) != cudaSuccess) { rc = PF_ERR_CUDA; break; }
    } while (0);
    prof_suspend(false);
    if (rc == PF_OK &&
        (cudaMemsetAsync(P.sc, 0, sizeof(BicgScalars), cs) != cudaSuccess ||
         cudaStreamSynchronize(cs) != cudaSuccess))
        rc = PF_ERR_CUDA;
    cudaStreamDestroy(cs);
    if (rc != PF_OK) {
        plan_free(plan);
        cudaGetLastError();
        return rc;
    }
    *out = plan;
    return PF_OK;
}

int batch_plan_create(int prec, int rk4, const pf_batch_member* m, int count, void* table,
                      void** out) {
    if (count < 1 || count > kMaxBatch) return PF_ERR_BAD_ARG;
    PlanLayout* P = new PlanLayout[count];
    int rc = PF_OK;
    for (int r = 0; r < count && rc == PF_OK; ++r)
        rc = plan_layout(&m[r].grid, prec, m[r].min_res, m[r].DP, m[r].ws, &P[r]);
    if (rc != PF_OK) { delete[] P; return rc; }
    // the requests' solves run as parallel branches: their mid levels stay on
    // the per-level kernels (no grid-barrier launches that could wait on one
    // another for room on the SMs)
    for (int r = 0; r < count; ++r) P[r].mg.coop = 0;
    if (predictor_prepare(prec) != cudaSuccess) { delete[] P; return PF_ERR_CUDA; }
    cudaStream_t cs;
    if (cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking) != cudaSuccess) {
        delete[] P;
        return PF_ERR_CUDA;
    }
    // the grouped predictor's members, and each request's one-time set-up
    GroupMember gm[kMaxBatch];
    for (int r = 0; r < count; ++r)
        gm[r] = GroupMember{m[r].grid, m[r].u, m[r].v, m[r].w, m[r].mu, m[r].rho, m[r].dt,
                            P[r].R};
    rc = grouped_predictor_tables(prec, rk4, gm, count, table, cs);
    // one-time set-up of members that join a plan for the first time; a
    // member carried over from an earlier plan may still be computing there
    // and is not touched
    for (int r = 0; r < count && rc == PF_OK; ++r)
        if (m[r].fresh) rc = plan_fill(&m[r].grid, prec, m[r].DP, m[r].ws, P[r], cs);
    if (rc == PF_OK && cudaStreamSynchronize(cs) != cudaSuccess) rc = PF_ERR_CUDA;
    StepPlan* plan = new StepPlan();
    prof_suspend(true);
    do {
        if (rc != PF_OK) break;
        if (cudaGraphCreate(&plan->graph, 0) != cudaSuccess) { rc = PF_ERR_CUDA; break; }
        cudaGraph_t G = plan->graph;
        cudaGraphNode_t n0;
        if ((rc = add_captured(G, cs, [&](cudaStream_t st) {
                 return launch_grouped_predictor(prec, rk4, gm, count, table, st);
             }, &n0)))
            break;
        // the requests' solves run as independent branches of the graph
        for (int r = 0; r < count && rc == PF_OK; ++r) {
            cudaGraphNode_t nend;
            rc = add_solve_chain(G, n0, &m[r].grid, prec, P[r], m[r].u, m[r].v, m[r].w, m[r].p,
                                 m[r].DP, m[r].rho, m[r].dt, m[r].min_res, m[r].max_it,
                                 m[r].stats, false, cs, &nend);
        }
        if (rc != PF_OK) break;
        if (cudaGraphInstantiate(&plan->exec, G, 0) != cudaSuccess) { rc = PF_ERR_CUDA; break; }
    } while (0);
    prof_suspend(false);
    for (int r = 0; r < count && rc == PF_OK; ++r)
        if (m[r].fresh && cudaMemsetAsync(P[r].sc, 0, sizeof(BicgScalars), cs) != cudaSuccess)
            rc = PF_ERR_CUDA;
    if (rc == PF_OK && cudaStreamSynchronize(cs) != cudaSuccess) rc = PF_ERR_CUDA;
    cudaStreamDestroy(cs);
    delete[] P;
    if (rc != PF_OK) {
        plan_free(plan);
        cudaGetLastError();
        return rc;
    }
    *out = plan;
    return PF_OK;
}

int step_plan_launch(void* plan, int nsteps, cudaStream_t s) {
    StepPlan* pl = (StepPlan*)plan;
    for (int i = 0; i < nsteps; ++i)
        if (cudaGraphLaunch(pl->exec, s) != cudaSuccess) return PF_ERR_CUDA;
    return PF_OK;
}

int step_plan_destroy(void* plan) {
    if (plan) plan_free((StepPlan*)plan);
    return PF_OK;
}

}  // namespace pf
