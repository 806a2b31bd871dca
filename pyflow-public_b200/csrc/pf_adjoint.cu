// pf_adjoint.cu -- exact discrete adjoint (vector-Jacobian product) of the
// staggered Navier-Stokes right-hand side, and of its 'tensor' SFS term.
//
// The forward RHS (rhs_NavierStokes.evaluate, src/solver/velocity.py:221-355)
// is a sum of conservative differences of face/edge fluxes:
//   rhs_u +=  dxi (FX[i] - FX[i-1]) + dyi (FXY[j] - FXY[j-1]) + dzi (FXZ[k] - FXZ[k-1])
//   rhs_u -=  dxi (Cxx[i] - Cxx[i-1]) + dyi (Cxy[j+1] - Cxy[j]) + dzi (Cxz[k+1] - Cxz[k])
// (and likewise for v, w), where the viscous fluxes are linear in the
// velocity and the convective ones are products of face averages
// (Cxx = cu^2, Cxy = uy vx, ...; metric_staggered.py:149-188,458-526).  The
// transpose of a flux difference is a difference of the adjoint field, so for
// a given adjoint mu the kernel first forms each flux's adjoint
//   lam_Cxx(p) = dxi (mu_u(p+x) - mu_u(p)),
//   lam_Cxy(p) = dyi (mu_u(p) - mu_u(p-y)) + dxi (mu_v(p) - mu_v(p-x)), ...
// and then gathers lam * dFlux/du over every flux that reads the cell.  The
// result is J(u)^T mu exactly (to round-off), computed per cell from a 3x3x3
// neighbourhood of u and mu: deterministic, no atomics.
//
// The reference's own adjoint (src/solver/adjoint.py:94-227,
// src/metric/metric_staggered.py:537-799) evaluates the same transpose with
// the viscous operator applied as-is (it is symmetric) and its discrete-exact
// convective terms; tests/test_gpu_adjoint.py compares the two.
#include "pf_common.cuh"
#include "pf_kernels.cuh"
#include "pf_profile.cuh"

namespace pf {

struct AdjArgs {
    const double *u, *v, *w;     // forward state at which J is evaluated
    const double *mu, *mv, *mw;  // adjoint input
    double dxi, dyi, dzi;
    double a;   // 2 mu / rho   (diagonal viscous flux factor)
    double e;   // mu_edge / rho (off-diagonal viscous flux factor)
    double scale;  // of the adjoint input
};

// J(state)^T lambda of one cell; lambda = A.scale * (mu, mv, mw), the product
// rounded first (A.scale 1: lambda itself).
__device__ __forceinline__ void rhs_adjoint_cell(const Dims& d, const AdjArgs& A, int i, int j,
                                                 int k, double& ru, double& rv, double& rw) {
    const double dxi = A.dxi, dyi = A.dyi, dzi = A.dzi;
    auto at = [&](const double* f, int di, int dj, int dk) -> double {
        return __ldg(f + idx(d, wrap(i + di, d.nx), wrap(j + dj, d.ny), wrap(k + dk, d.nz)));
    };
    // the adjoint, scaled (its fields may be the state's own)
    auto adj = [&](const double* f, int di, int dj, int dk) { return A.scale * at(f, di, dj, dk); };
    // ---- convective flux adjoints (at flux position p = c + (di,dj,dk))
    auto lamCxx = [&](int di, int dj, int dk) { return dxi * (adj(A.mu, di + 1, dj, dk) - adj(A.mu, di, dj, dk)); };
    auto lamCyy = [&](int di, int dj, int dk) { return dyi * (adj(A.mv, di, dj + 1, dk) - adj(A.mv, di, dj, dk)); };
    auto lamCzz = [&](int di, int dj, int dk) { return dzi * (adj(A.mw, di, dj, dk + 1) - adj(A.mw, di, dj, dk)); };
    auto lamCxy = [&](int di, int dj, int dk) {
        return dyi * (adj(A.mu, di, dj, dk) - adj(A.mu, di, dj - 1, dk)) +
               dxi * (adj(A.mv, di, dj, dk) - adj(A.mv, di - 1, dj, dk));
    };
    auto lamCxz = [&](int di, int dj, int dk) {
        return dzi * (adj(A.mu, di, dj, dk) - adj(A.mu, di, dj, dk - 1)) +
               dxi * (adj(A.mw, di, dj, dk) - adj(A.mw, di - 1, dj, dk));
    };
    auto lamCyz = [&](int di, int dj, int dk) {
        return dzi * (adj(A.mv, di, dj, dk) - adj(A.mv, di, dj, dk - 1)) +
               dyi * (adj(A.mw, di, dj, dk) - adj(A.mw, di, dj - 1, dk));
    };
    // face averages of the state entering the products
    auto cu = [&](int di, int dj, int dk) { return 0.5 * (at(A.u, di + 1, dj, dk) + at(A.u, di, dj, dk)); };
    auto cv = [&](int di, int dj, int dk) { return 0.5 * (at(A.v, di, dj + 1, dk) + at(A.v, di, dj, dk)); };
    auto cw = [&](int di, int dj, int dk) { return 0.5 * (at(A.w, di, dj, dk + 1) + at(A.w, di, dj, dk)); };
    auto uy = [&](int di, int dj, int dk) { return 0.5 * (at(A.u, di, dj, dk) + at(A.u, di, dj - 1, dk)); };
    auto uz = [&](int di, int dj, int dk) { return 0.5 * (at(A.u, di, dj, dk) + at(A.u, di, dj, dk - 1)); };
    auto vx = [&](int di, int dj, int dk) { return 0.5 * (at(A.v, di, dj, dk) + at(A.v, di - 1, dj, dk)); };
    auto vz = [&](int di, int dj, int dk) { return 0.5 * (at(A.v, di, dj, dk) + at(A.v, di, dj, dk - 1)); };
    auto wx = [&](int di, int dj, int dk) { return 0.5 * (at(A.w, di, dj, dk) + at(A.w, di - 1, dj, dk)); };
    auto wy = [&](int di, int dj, int dk) { return 0.5 * (at(A.w, di, dj, dk) + at(A.w, di, dj - 1, dk)); };

    double au = 0.0, av = 0.0, aw = 0.0;
    // Cxx(p) = cu(p)^2 reads u(p), u(p+x): cell c is read by p = c, c-x
    au += lamCxx(0, 0, 0) * cu(0, 0, 0) + lamCxx(-1, 0, 0) * cu(-1, 0, 0);
    // Cxy(p) = uy(p) vx(p): u(c) in uy at p = c, c+y; v(c) in vx at p = c, c+x
    au += 0.5 * (lamCxy(0, 0, 0) * vx(0, 0, 0) + lamCxy(0, 1, 0) * vx(0, 1, 0));
    av += 0.5 * (lamCxy(0, 0, 0) * uy(0, 0, 0) + lamCxy(1, 0, 0) * uy(1, 0, 0));
    // Cxz(p) = uz(p) wx(p)
    au += 0.5 * (lamCxz(0, 0, 0) * wx(0, 0, 0) + lamCxz(0, 0, 1) * wx(0, 0, 1));
    aw += 0.5 * (lamCxz(0, 0, 0) * uz(0, 0, 0) + lamCxz(1, 0, 0) * uz(1, 0, 0));
    // Cyy(p) = cv(p)^2
    av += lamCyy(0, 0, 0) * cv(0, 0, 0) + lamCyy(0, -1, 0) * cv(0, -1, 0);
    // Cyz(p) = vz(p) wy(p)
    av += 0.5 * (lamCyz(0, 0, 0) * wy(0, 0, 0) + lamCyz(0, 0, 1) * wy(0, 0, 1));
    aw += 0.5 * (lamCyz(0, 0, 0) * vz(0, 0, 0) + lamCyz(0, 1, 0) * vz(0, 1, 0));
    // Czz(p) = cw(p)^2
    aw += lamCzz(0, 0, 0) * cw(0, 0, 0) + lamCzz(0, 0, -1) * cw(0, 0, -1);

    // ---- viscous (constant viscosity): diagonal fluxes at centres
    // FX = (ux - D/3) a, FY = (vy - D/3) a, FZ = (wz - D/3) a with D = ux+vy+wz;
    // their adjoints lX = dxi (mu_u(p) - mu_u(p+x)), ...
    auto lX = [&](int di, int dj, int dk) { return dxi * (adj(A.mu, di, dj, dk) - adj(A.mu, di + 1, dj, dk)); };
    auto lY = [&](int di, int dj, int dk) { return dyi * (adj(A.mv, di, dj, dk) - adj(A.mv, di, dj + 1, dk)); };
    auto lZ = [&](int di, int dj, int dk) { return dzi * (adj(A.mw, di, dj, dk) - adj(A.mw, di, dj, dk + 1)); };
    auto sx = [&](int di, int dj, int dk) {
        return A.a * (2.0 * lX(di, dj, dk) - lY(di, dj, dk) - lZ(di, dj, dk)) / 3.0;
    };
    auto sy = [&](int di, int dj, int dk) {
        return A.a * (2.0 * lY(di, dj, dk) - lX(di, dj, dk) - lZ(di, dj, dk)) / 3.0;
    };
    auto sz = [&](int di, int dj, int dk) {
        return A.a * (2.0 * lZ(di, dj, dk) - lX(di, dj, dk) - lY(di, dj, dk)) / 3.0;
    };
    // ux(p) = (u(p+x) - u(p)) dxi reads u(c) at p = c-x (+), c (-)
    au += dxi * (sx(-1, 0, 0) - sx(0, 0, 0));
    av += dyi * (sy(0, -1, 0) - sy(0, 0, 0));
    aw += dzi * (sz(0, 0, -1) - sz(0, 0, 0));
    // off-diagonal fluxes on edges: FXY = ((u(p+y)-u(p)) dyi + (v(p+x)-v(p)) dxi) e
    auto txy = [&](int di, int dj, int dk) {
        return A.e * (dyi * (adj(A.mu, di, dj, dk) - adj(A.mu, di, dj + 1, dk)) +
                      dxi * (adj(A.mv, di, dj, dk) - adj(A.mv, di + 1, dj, dk)));
    };
    auto txz = [&](int di, int dj, int dk) {
        return A.e * (dzi * (adj(A.mu, di, dj, dk) - adj(A.mu, di, dj, dk + 1)) +
                      dxi * (adj(A.mw, di, dj, dk) - adj(A.mw, di + 1, dj, dk)));
    };
    auto tyz = [&](int di, int dj, int dk) {
        return A.e * (dzi * (adj(A.mv, di, dj, dk) - adj(A.mv, di, dj, dk + 1)) +
                      dyi * (adj(A.mw, di, dj, dk) - adj(A.mw, di, dj + 1, dk)));
    };
    au += dyi * (txy(0, -1, 0) - txy(0, 0, 0)) + dzi * (txz(0, 0, -1) - txz(0, 0, 0));
    av += dxi * (txy(-1, 0, 0) - txy(0, 0, 0)) + dzi * (tyz(0, 0, -1) - tyz(0, 0, 0));
    aw += dxi * (txz(-1, 0, 0) - txz(0, 0, 0)) + dyi * (tyz(0, -1, 0) - tyz(0, 0, 0));

    ru = au;
    rv = av;
    rw = aw;
}

__global__ void __launch_bounds__(256, 2)
rhs_adjoint_kernel(Dims d, AdjArgs A, double* __restrict__ ou,
                   double* __restrict__ ov, double* __restrict__ ow) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int i = blockIdx.z;
    if (k >= d.nz || j >= d.ny) return;
    const long long q = idx(d, i, j, k);
    rhs_adjoint_cell(d, A, i, j, k, ou[q], ov[q], ow[q]);
}

// Adjoint of the 'tensor' SFS stresses: the stresses are added to the viscous
// fluxes before the divergence (src/solver/velocity.py:262-267,...), the
// diagonal ones at cell centres and the off-diagonal ones edge-averaged from
// centres one cell below (interp_sc_xy, metric_staggered.py:127-144).
// out[0..5] += adjoint of FXX, FYY, FZZ, FXY, FXZ, FYZ for adjoint mu (scaled
// by `weight`, accumulated so that RK4 stages can be summed).
__device__ __forceinline__ void sfs_adjoint_cell(const Dims& d, const double* mu, const double* mv,
                                                 const double* mw, double scale, double dxi,
                                                 double dyi, double dzi, int i, int j, int k,
                                                 double (&f)[6]) {
    auto at = [&](const double* a, int di, int dj, int dk) -> double {
        return scale * __ldg(a + idx(d, wrap(i + di, d.nx), wrap(j + dj, d.ny), wrap(k + dk, d.nz)));
    };
    // flux adjoints at edge positions p
    auto lxy = [&](int di, int dj) {
        return dyi * (at(mu, di, dj, 0) - at(mu, di, dj + 1, 0)) + dxi * (at(mv, di, dj, 0) - at(mv, di + 1, dj, 0));
    };
    auto lxz = [&](int di, int dk) {
        return dzi * (at(mu, di, 0, dk) - at(mu, di, 0, dk + 1)) + dxi * (at(mw, di, 0, dk) - at(mw, di + 1, 0, dk));
    };
    auto lyz = [&](int dj, int dk) {
        return dzi * (at(mv, 0, dj, dk) - at(mv, 0, dj, dk + 1)) + dyi * (at(mw, 0, dj, dk) - at(mw, 0, dj + 1, dk));
    };
    f[0] = dxi * (at(mu, 0, 0, 0) - at(mu, 1, 0, 0));
    f[1] = dyi * (at(mv, 0, 0, 0) - at(mv, 0, 1, 0));
    f[2] = dzi * (at(mw, 0, 0, 0) - at(mw, 0, 0, 1));
    // S(p) = 0.25 (F(p) + F(p-x) + F(p-y) + F(p-x-y)): F(c) feeds p = c, c+x, c+y, c+x+y
    f[3] = 0.25 * (lxy(0, 0) + lxy(1, 0) + lxy(0, 1) + lxy(1, 1));
    f[4] = 0.25 * (lxz(0, 0) + lxz(1, 0) + lxz(0, 1) + lxz(1, 1));
    f[5] = 0.25 * (lyz(0, 0) + lyz(1, 0) + lyz(0, 1) + lyz(1, 1));
}

__global__ void __launch_bounds__(256)
sfs_adjoint_kernel(Dims d, const double* __restrict__ mu, const double* __restrict__ mv,
                   const double* __restrict__ mw, double dxi, double dyi, double dzi,
                   double weight, double* __restrict__ out) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int i = blockIdx.z;
    if (k >= d.nz || j >= d.ny) return;
    double f[6];
    sfs_adjoint_cell(d, mu, mv, mw, 1.0, dxi, dyi, dzi, i, j, k, f);
    const long long q = idx(d, i, j, k);
#pragma unroll
    for (int c = 0; c < 6; ++c) out[c * d.n + q] += weight * f[c];
}

// One stage of the reversed predictor: m = J(stage state)^T kbar with kbar =
// A.scale * (A.mu, A.mv, A.mw); total = base + m; the next (earlier) stage's
// kbar' = wnext lam + h m; with SFS stresses their adjoint F (+)= of kbar.  As
// separate torch operations the four stages of a step took 70 launches and,
// at 64^3, 0.3 ms of host time against 0.15 ms of these kernels.
struct VjpStage {
    const double* lam[3];   // the projected adjoint field
    const double* base[3];  // total so far (lam at the last stage)
    double* total[3];
    double* next[3];        // null: no earlier stage
    double wnext, h;
    double* F;              // null: no SFS stresses
    int add;                // F holds the later stages' sum
};

__global__ void __launch_bounds__(256, 2)
vjp_stage_kernel(Dims d, AdjArgs A, VjpStage S) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int i = blockIdx.z;
    if (k >= d.nz || j >= d.ny) return;
    const long long q = idx(d, i, j, k);
    double m[3];
    rhs_adjoint_cell(d, A, i, j, k, m[0], m[1], m[2]);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        if (S.next[c]) S.next[c][q] = S.wnext * S.lam[c][q] + S.h * m[c];
        S.total[c][q] = S.base[c][q] + m[c];
    }
    if (S.F) {
        double f[6];
        sfs_adjoint_cell(d, A.mu, A.mv, A.mw, A.scale, A.dxi, A.dyi, A.dzi, i, j, k, f);
#pragma unroll
        for (int c = 0; c < 6; ++c) S.F[c * d.n + q] = S.add ? S.F[c * d.n + q] + f[c] : f[c];
    }
}

}  // namespace pf

extern "C" int pf_rhs_adjoint(const pf_grid* g, const double* u, const double* v,
                              const double* w, const double* mu_u,
                              const double* mu_v, const double* mu_w, double mu,
                              double rho, double* out_u, double* out_v,
                              double* out_w, void* stream) {
    if (!g || g->nx < 2 || g->ny < 2 || g->nz < 2 || !(g->dx > 0) || !(g->dy > 0) ||
        !(g->dz > 0) || !u || !v || !w || !mu_u || !mu_v || !mu_w || !out_u || !out_v ||
        !out_w || !(rho != 0.0))
        return PF_ERR_BAD_ARG;
    pf::Dims d{g->nx, g->ny, g->nz, (long long)g->nx * g->ny * g->nz};
    pf::AdjArgs A{u, v, w, mu_u, mu_v, mu_w, 1.0 / g->dx, 1.0 / g->dy, 1.0 / g->dz,
                  (2.0 * mu) / rho, (0.25 * (((mu + mu) + mu) + mu)) / rho, 1.0};
    cudaStream_t s = (cudaStream_t)stream;
    dim3 blk(32, 8), grd((d.nz + 31) / 32, (d.ny + 7) / 8, d.nx);
    PF_LAUNCH("rhs_adjoint", s, pf::rhs_adjoint_kernel<<<grd, blk, 0, s>>>(d, A, out_u, out_v, out_w));
    return cudaGetLastError() == cudaSuccess ? PF_OK : PF_ERR_CUDA;
}

extern "C" int pf_sfs_adjoint(const pf_grid* g, const double* mu_u,
                              const double* mu_v, const double* mu_w,
                              double weight, double* out, void* stream) {
    if (!g || g->nx < 2 || g->ny < 2 || g->nz < 2 || !(g->dx > 0) || !(g->dy > 0) ||
        !(g->dz > 0) || !mu_u || !mu_v || !mu_w || !out)
        return PF_ERR_BAD_ARG;
    pf::Dims d{g->nx, g->ny, g->nz, (long long)g->nx * g->ny * g->nz};
    cudaStream_t s = (cudaStream_t)stream;
    dim3 blk(32, 8), grd((d.nz + 31) / 32, (d.ny + 7) / 8, d.nx);
    PF_LAUNCH("sfs_adjoint", s, pf::sfs_adjoint_kernel<<<grd, blk, 0, s>>>(
        d, mu_u, mu_v, mu_w, 1.0 / g->dx, 1.0 / g->dy, 1.0 / g->dz, weight, out));
    return cudaGetLastError() == cudaSuccess ? PF_OK : PF_ERR_CUDA;
}

static bool overlap(const void* a, size_t na, const void* b, size_t nb) {
    const uintptr_t x = (uintptr_t)a, y = (uintptr_t)b;
    return x < y + nb && y < x + na;
}

extern "C" size_t pf_predictor_vjp_workspace_bytes(const pf_grid* g) {
    if (!g || g->nx < 2 || g->ny < 2 || g->nz < 2) return 0;
    // three stage states, two sets of stage adjoints
    return (size_t)15 * g->nx * g->ny * g->nz * sizeof(double);
}

extern "C" int pf_predictor_vjp(const pf_grid* g, int rk4, const double* u, const double* v,
                                const double* w, const double* lam_u, const double* lam_v,
                                const double* lam_w, double mu, double rho, double dt,
                                const double* sfs, double* out_u, double* out_v, double* out_w,
                                double* out_sfs, void* ws, size_t ws_bytes, void* stream) {
    if (!g || g->nx < 2 || g->ny < 2 || g->nz < 2 || !(g->dx > 0) || !(g->dy > 0) ||
        !(g->dz > 0) || !u || !v || !w || !lam_u || !lam_v || !lam_w || !out_u || !out_v ||
        !out_w || !(rho != 0.0) || !ws || ((uintptr_t)ws & 7) ||
        ws_bytes < pf_predictor_vjp_workspace_bytes(g) || (out_sfs && !sfs))
        return PF_ERR_BAD_ARG;
    using namespace pf;
    const Dims d{g->nx, g->ny, g->nz, (long long)g->nx * g->ny * g->nz};
    const long long n = d.n;
    // The stages read the state and the adjoint at neighbouring cells after
    // outputs have been written, and the workspace holds stage states and
    // adjoints (RK4): what is written shares memory with none of them.
    {
        struct Range { const void* p; size_t bytes; } r[11];
        int outs = 0, k = 0;
        const size_t b = (size_t)n * sizeof(double);
        for (double* o : {out_u, out_v, out_w}) r[k++] = Range{o, b};
        if (out_sfs) r[k++] = Range{out_sfs, 6 * b};
        if (rk4) r[k++] = Range{ws, pf_predictor_vjp_workspace_bytes(g)};
        outs = k;
        for (const double* x : {u, v, w, lam_u, lam_v, lam_w}) r[k++] = Range{x, b};
        for (int i = 0; i < outs; ++i)
            for (int j = i + 1; j < k; ++j)
                if (overlap(r[i].p, r[i].bytes, r[j].p, r[j].bytes)) return PF_ERR_BAD_ARG;
        // (the stresses are read before any output is written)
        if (rk4 && sfs && overlap(ws, pf_predictor_vjp_workspace_bytes(g), sfs, 6 * b))
            return PF_ERR_BAD_ARG;
    }
    cudaStream_t s = (cudaStream_t)stream;
    double* st = (double*)ws;
    double* kb[2] = {st + 9 * n, st + 12 * n};
    const int stages = rk4 ? 4 : 1;
    if (rk4 && launch_stage_states(g, u, v, w, mu, rho, sfs, dt, st, s) != cudaSuccess)
        return PF_ERR_CUDA;
    const double* lam[3] = {lam_u, lam_v, lam_w};
    double* out[3] = {out_u, out_v, out_w};
    const double wts[4] = {dt / 6.0, dt / 3.0, dt / 3.0, dt / 6.0};
    dim3 blk(32, 8), grd((d.nz + 31) / 32, (d.ny + 7) / 8, d.nx);
    for (int q = stages - 1; q >= 0; --q) {
        const double* x = q ? st + 3 * n * (q - 1) : nullptr;
        const bool first = q == stages - 1;
        const double* kin = kb[q & 1];
        AdjArgs A{x ? x : u, x ? x + n : v, x ? x + 2 * n : w,
                  first ? lam_u : kin, first ? lam_v : kin + n, first ? lam_w : kin + 2 * n,
                  1.0 / g->dx, 1.0 / g->dy, 1.0 / g->dz, (2.0 * mu) / rho,
                  (0.25 * (((mu + mu) + mu) + mu)) / rho,
                  first ? (rk4 ? wts[3] : dt) : 1.0};
        VjpStage S;
        for (int c = 0; c < 3; ++c) {
            S.lam[c] = lam[c];
            S.base[c] = first ? lam[c] : out[c];
            S.total[c] = out[c];
            S.next[c] = q ? kb[(q - 1) & 1] + c * n : nullptr;
        }
        S.wnext = q ? wts[q - 1] : 0.0;
        S.h = 0.5 * dt;
        S.F = out_sfs;
        S.add = first ? 0 : 1;
        PF_LAUNCH("vjp_stage", s, vjp_stage_kernel<<<grd, blk, 0, s>>>(d, A, S));
    }
    return cudaGetLastError() == cudaSuccess ? PF_OK : PF_ERR_CUDA;
}
