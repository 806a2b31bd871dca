// pf_spectral.cu -- direct solve of A x = c src, A = (-vol L) the periodic
// 7-point operator of Pressure_Base.applyOperator (src/solver/pressure.py:54-84).
//
// On the uniform periodic grid A is diagonal in the product of the three
// axes' discrete Hartley bases cas(2 pi j k / n) (cas = cos + sin), with
// eigenvalues sum_q 4 vol/h_q^2 sin^2(pi k_q / n_q).  The Hartley transform is
// real and its own inverse (up to n), so every array of the solve is a real
// [nx][ny][nz] field and the z and y passes back are the passes forward:
//
//   z pass (src -> DP), y pass, x pass (transform, divide by the eigenvalue,
//   transform back), y pass, z pass -- all FP64, in place in DP,
//
// 16 bytes per cell and pass (80 in all), against 174 per iteration of the
// multigrid-preconditioned FP32 BiCGStab that served these solves before,
// whose refinement ran five iterations per step at 512^3.
//
// A block transforms 2L real lines as L complex ones (pairs of lines as real
// and imaginary part; the Hartley values come from Z[k] and Z[n-k]): Stockham
// stages of radix 8, 4, 2, 3, 5, 7 in registers, other primes as direct sums,
// exchanged through one [n][L] shared-memory buffer whose 16-byte slots are
// XOR-swizzled by the element so that neither the line-wise (z) nor the
// element-wise accesses conflict.  A thread holds 8 complex values.  In the x
// and y passes a line pair is two neighbouring cells in z, and a block's L = 8
// pairs read and write runs of 128 bytes; in the z pass the rows themselves
// are contiguous.  The multiples of 32 among 2^k, 3 2^k and 5 2^k up to 1024 have
// kernels of their own (pf_spectral_fast.cu); 48 and 80, for example, do not.
#include <algorithm>
#include <cmath>

#include "pf_common.cuh"
#include "pf_kernels.cuh"
#include "pf_profile.cuh"
#include "pf_spectral_pass.cuh"

namespace pf {
namespace {

// One Stockham stage of radix R (pp: product of the earlier radices): the
// butterfly i of a line reads elements i + q n/R, and writes (i - k) R + k + q pp
// with k = i mod pp.  The values stay in registers across the barrier, so one
// buffer serves.
template <int R, int L>
__device__ __forceinline__ void stage(double2* sm, const double2* tw, int n, int tp,
                                      int pp, unsigned magic, int it, int l, bool act) {
    constexpr int M = kHold / R;
    const int nr = n / R, ts = nr / pp;
    double2 x[M][R];
#pragma unroll
    for (int m = 0; m < M; ++m) {
        // a thread without a butterfly computes the first one and drops it
        const int i = act && it + m * tp < nr ? it + m * tp : 0;
#pragma unroll
        for (int q = 0; q < R; ++q) x[m][q] = sm[slot<L>(i + q * nr, l)];
        if (pp > 1) {
            const int k = i - (int)__umulhi((unsigned)i, magic) * pp;
#pragma unroll
            for (int q = 1; q < R; ++q) x[m][q] = cmul(x[m][q], tw[q * k * ts]);
        }
        Dft<R>::run(x[m]);
    }
    __syncthreads();
#pragma unroll
    for (int m = 0; m < M; ++m) {
        const int i = it + m * tp;
        if (!act || i >= nr) continue;
        const int k = pp > 1 ? i - (int)__umulhi((unsigned)i, magic) * pp : 0;
        const int jo = (i - k) * R + k;
#pragma unroll
        for (int q = 0; q < R; ++q) sm[slot<L>(jo + q * pp, l)] = x[m][q];
    }
    __syncthreads();
}

// A stage of any other (prime) radix R as direct sums, one output at a time:
// output q of butterfly i is sum_r x[i + r n/R] w_n^(r (k n/(R pp) + q n/R)).
template <int L>
__device__ __forceinline__ void stage_any(double2* sm, const double2* tw, int n, int tp, int R,
                                          int pp, unsigned magic, int it, int l, bool act) {
    const int nr = n / R, ts = nr / pp;
    double2 y[kHold];
    int jo[kHold];
#pragma unroll
    for (int m = 0; m < kHold; ++m) {
        const int o = it + m * tp;
        jo[m] = -1;
        if (!act || o >= n) continue;
        const int q = o / nr, i = o - q * nr;
        const int k = pp > 1 ? i - (int)__umulhi((unsigned)i, magic) * pp : 0;
        const int step = (k * ts + q * nr) % n;
        double2 a = sm[slot<L>(i, l)];
        int e = 0;
        for (int r = 1; r < R; ++r) {
            e += step;
            if (e >= n) e -= n;
            const double2 b = sm[slot<L>(i + r * nr, l)], w = tw[e];
            a.x = fma(b.x, w.x, a.x); a.x = fma(-b.y, w.y, a.x);
            a.y = fma(b.x, w.y, a.y); a.y = fma(b.y, w.x, a.y);
        }
        y[m] = a;
        jo[m] = (i - k) * R + k + q * pp;
    }
    __syncthreads();
#pragma unroll
    for (int m = 0; m < kHold; ++m)
        if (jo[m] >= 0) sm[slot<L>(jo[m], l)] = y[m];
    __syncthreads();
}

// DFT of the L complex lines in sm (all threads of the block call it).  The
// odd radices need more registers than the 64 that let two 512-thread blocks
// share an SM, so extents without odd factors have an instance of their own.
template <int L, bool ODD>
__device__ __forceinline__ void transform(double2* sm, const double2* tw, const SpectralAxis& ax,
                                          int it, int l, bool act) {
    int pp = 1;
    for (int s = 0; s < ax.stages; ++s) {
        const int R = ax.radix[s];
        const unsigned mg = ax.magic[s];
        if (R == 8) stage<8, L>(sm, tw, ax.n, ax.tp, pp, mg, it, l, act);
        else if (R == 4) stage<4, L>(sm, tw, ax.n, ax.tp, pp, mg, it, l, act);
        else if (R == 2) stage<2, L>(sm, tw, ax.n, ax.tp, pp, mg, it, l, act);
        else if (ODD) {
            if (R == 3) stage<3, L>(sm, tw, ax.n, ax.tp, pp, mg, it, l, act);
            else if (R == 5) stage<5, L>(sm, tw, ax.n, ax.tp, pp, mg, it, l, act);
            else if (R == 7) stage<7, L>(sm, tw, ax.n, ax.tp, pp, mg, it, l, act);
            else stage_any<L>(sm, tw, ax.n, ax.tp, R, pp, mg, it, l, act);
        }
        pp *= R;
    }
}

template <int L, int KIND, bool ODD>
__global__ void __launch_bounds__(kMaxThreads, ODD ? 1 : 2)
spectral_pass(PassArgs a) {
    extern __shared__ __align__(16) double2 sm[];
    const int n = a.ax.n, tid = threadIdx.x, nt = blockDim.x;
    double2* tw = sm + n * L;
    const int l = tid % L, it = tid / L;
    const bool act = it < a.ax.tp;
    pdl_wait();
    for (int e = tid; e < n; e += nt) tw[e] = a.ax.tw[e];
    // ---- load
    long long base = 0, c0 = 0;
    bool ha = false, hb = false;    // x, y: this thread's pair has a first, second line
    if (KIND == kPassZ) {
        const int lane = tid & 31, nw = nt >> 5;
        const long long r0 = (long long)blockIdx.x * (2 * L);
        double big = 0.0;
        for (int q = tid >> 5; q < L; q += nw) {
            const long long ra = r0 + 2 * q;
            if (ra >= a.nlines) break;
            const bool two = ra + 1 < a.nlines;
            const double* pa = a.src + ra * n;
#pragma unroll 4
            for (int e = lane; e < n; e += 32) {
                const double2 x = make_double2(pa[e], two ? pa[n + e] : 0.0);
                sm[slot<L>(e, q)] = x;
                big = absmax(big, absmax(abs_bits(x.x), abs_bits(x.y)));
            }
        }
        if (a.nonfin && !(big < __longlong_as_double(0x7ff0000000000000LL))) *a.nonfin = 1;
    } else {
        long long plane = 0;
        if (KIND == kPassY) {
            const long long i = blockIdx.x / a.tiles;
            c0 = (long long)(blockIdx.x - i * a.tiles) * (2 * L);
            plane = i * (long long)n * a.stride;
        } else {
            c0 = (long long)blockIdx.x * (2 * L);
        }
        const long long c = c0 + 2 * l;
        ha = c < a.nlines;
        hb = c + 1 < a.nlines;
        base = plane + c;
        const double* p = a.src + base;
        const int es = nt / L;
        if (it < es && ha) {
            if (a.vec && hb) {
#pragma unroll 8
                for (int e = it; e < n; e += es)
                    sm[slot<L>(e, l)] = *(const double2*)(p + e * a.stride);
            } else {
#pragma unroll 4
                for (int e = it; e < n; e += es)
                    sm[slot<L>(e, l)] = make_double2(p[e * a.stride], hb ? p[e * a.stride + 1] : 0.0);
            }
        }
    }
    __syncthreads();
    transform<L, ODD>(sm, tw, a.ax, it, l, act);
    if (KIND == kPassZ) {
        const int lane = tid & 31, nw = nt >> 5;
        const long long r0 = (long long)blockIdx.x * (2 * L);
        for (int q = tid >> 5; q < L; q += nw) {
            const long long ra = r0 + 2 * q;
            if (ra >= a.nlines) break;
            const bool two = ra + 1 < a.nlines;
            double* pa = a.dst + ra * n;
            for (int e = lane; e < n; e += 32) {
                const double2 h = hartley(sm[slot<L>(e, q)], sm[slot<L>(e ? n - e : 0, q)]);
                pa[e] = h.x;
                if (two) pa[n + e] = h.y;
            }
        }
        return;
    }
    double* p = a.dst + base;
    const int es = nt / L;
    if (KIND == kPassY) {
        if (it < es && ha) {
            for (int e = it; e < n; e += es) {
                const double2 h = hartley(sm[slot<L>(e, l)], sm[slot<L>(e ? n - e : 0, l)]);
                double* o = p + e * a.stride;
                if (a.vec && hb) *(double2*)o = h;
                else { o[0] = h.x; if (hb) o[1] = h.y; }
            }
        }
        return;
    }
    // x pass: the transforms of the two lines times their own factors s/lambda
    // (equal at k and n - k): W = (ma + mb)/2 Z[k] + (ma - mb)/2 conj Z[n-k].
    // The inverse DFT of W is the forward one with real and imaginary parts
    // exchanged on the way in and out.
    {
        double la = 0.0, lb = 0.0;
        const long long c = c0 + 2 * l;
        if (ha) {
            const int j = (int)(c / a.nz), k = (int)(c - (long long)j * a.nz);
            la = a.lamy[j] + a.lamz[k];
            const int j2 = k + 1 < a.nz ? j : j + 1, k2 = k + 1 < a.nz ? k + 1 : 0;
            lb = hb ? a.lamy[j2] + a.lamz[k2] : 1.0;
        }
        double2 w[kHold];
#pragma unroll
        for (int m = 0; m < kHold; ++m) {
            const int e = it + m * a.ax.tp;
            if (!act || !ha || e >= n) continue;
            const double2 z = sm[slot<L>(e, l)], y = sm[slot<L>(e ? n - e : 0, l)];
            const double lx = a.ax.lam[e];
            const double va = lx + la, vb = lx + lb;
            // the constant mode (zero eigenvalue) has no part in the solution
            const double ma = va > 0.0 ? a.scale / va : 0.0, mb = vb > 0.0 ? a.scale / vb : 0.0;
            const double s = 0.5 * (ma + mb), t = 0.5 * (ma - mb);
            w[m] = make_double2(fma(s, z.y, -(t * y.y)), fma(s, z.x, t * y.x));
        }
        __syncthreads();
#pragma unroll
        for (int m = 0; m < kHold; ++m) {
            const int e = it + m * a.ax.tp;
            if (act && ha && e < n) sm[slot<L>(e, l)] = w[m];
        }
        __syncthreads();
    }
    transform<L, ODD>(sm, tw, a.ax, it, l, act);
    if (it < es && ha) {
        for (int e = it; e < n; e += es) {
            const double2 h = sm[slot<L>(e, l)];
            double* o = p + e * a.stride;
            if (a.vec && hb) *(double2*)o = make_double2(h.y, h.x);
            else { o[0] = h.y; if (hb) o[1] = h.x; }
        }
    }
}

// Twiddles exp(-2 pi i k / n) and eigenvalues 4 vol/h^2 sin^2(pi k / n) of the
// three axes.
struct TableArgs {
    int n[3];
    double2* tw[3];
    double* lam[3];
    double f[3];
};

__global__ void __launch_bounds__(256) spectral_tables(TableArgs a) {
    pdl_wait();
    const int q = blockIdx.y;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = a.n[q];
    if (k >= n) return;
    // reduced to the first quadrant's mirror images so that equal modes get
    // equal values: k and n - k share their cosine, sine and eigenvalue
    const int m = 2 * k <= n ? k : n - k;
    double s, c;
    sincospi(2.0 * m / n, &s, &c);
    a.tw[q][k] = make_double2(c, m == k ? -s : s);
    const double h = sinpi((double)m / n);
    a.lam[q][k] = 4.0 * a.f[q] * (h * h);
}

size_t pass_smem(const SpectralAxis& ax) { return (size_t)ax.n * (ax.lines + 1) * sizeof(double2); }

int pass_threads(const SpectralAxis& ax) { return (ax.tp * ax.lines + 31) / 32 * 32; }

template <int KIND, bool ODD>
PassKernel pass_kernel_l(int lines) {
    return lines == 8 ? spectral_pass<8, KIND, ODD>
                      : (lines == 4 ? spectral_pass<4, KIND, ODD> : spectral_pass<2, KIND, ODD>);
}

template <int KIND>
PassKernel pass_kernel(const SpectralAxis& ax) {
    return ax.odd ? pass_kernel_l<KIND, true>(ax.lines) : pass_kernel_l<KIND, false>(ax.lines);
}

cudaError_t spectral_attributes() {
    SpectralAxis ax;
    for (int lines : {8, 4, 2})
        for (int odd : {0, 1}) {
            ax.lines = lines;
            ax.odd = odd;
            for (PassKernel k : {pass_kernel<kPassZ>(ax), pass_kernel<kPassY>(ax),
                                 pass_kernel<kPassX>(ax)}) {
                const cudaError_t e = cudaFuncSetAttribute(
                    k, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
                if (e != cudaSuccess) return e;
            }
        }
    return spectral_fast_attributes();
}

template <int KIND>
void launch_pass(const char* name, const PassArgs& a, long long blocks, cudaStream_t s) {
    const PassKernel fast = spectral_fast_kernel(KIND, a.ax.n);
    PF_LAUNCH(name, s, launch_pdl(fast ? fast : pass_kernel<KIND>(a.ax), dim3((unsigned)blocks),
                                  dim3(pass_threads(a.ax)), pass_smem(a.ax), s, a));
}

// Radices of n: 8s and one 4, or two 4s (never a lone 2 beside an 8), then 3,
// 5, 7 and the remaining primes.  Threads per line: every stage's butterflies
// in one go, at most kHold values each.
void axis_plan(int n, SpectralAxis* ax) {
    ax->n = n;
    int m = n, twos = 0, s = 0;
    while (m % 2 == 0) { m /= 2; ++twos; }
    while (twos >= 3 && twos != 4) { ax->radix[s++] = 8; twos -= 3; }
    while (twos >= 2) { ax->radix[s++] = 4; twos -= 2; }
    if (twos) ax->radix[s++] = 2;
    for (int p = 3; m > 1; p += 2)
        while (m % p == 0) { ax->radix[s++] = p; m /= p; }
    ax->stages = s;
    ax->odd = (n & (n - 1)) != 0;
    int pp = 1, tp = 1;
    for (int q = 0; q < s; ++q) {
        const int R = ax->radix[q];
        ax->magic[q] = pp > 1 ? (unsigned)(((1ULL << 32) + pp - 1) / pp) : 0u;
        const bool fast = R <= 8;
        const int per = fast ? kHold / R : kHold, cnt = fast ? n / R : n;
        tp = std::max(tp, (cnt + per - 1) / per);
        pp *= R;
    }
    tp = std::max(tp, (n + kHold - 1) / kHold);  // the x pass's scaling
    ax->tp = tp;
    ax->lines = 8;
    if (spectral_fast_kernel(kPassZ, n)) {  // its own radices, 8 values a thread
        ax->tp = n / 8;
        ax->lines = fast_lines(n);
        return;
    }
    while (ax->lines > 2 && (pass_threads(*ax) > kMaxThreads || pass_smem(*ax) > 113 * 1024))
        ax->lines /= 2;
}

}  // namespace

size_t spectral_table_bytes(const pf_grid* g) {
    return align256((size_t)(g->nx + g->ny + g->nz) * (sizeof(double2) + sizeof(double)));
}

bool spectral_applies(const pf_grid* g, double min_res, const double* DP, const void* tables) {
    if (std::max(g->nx, std::max(g->ny, g->nz)) > kSpectralMaxN) return false;
    if (!(min_res >= kSpectralMinTol)) return false;
    if (((uintptr_t)tables & 15) || ((uintptr_t)DP & 7)) return false;
    SpectralAxis ax;
    for (int n : {g->nx, g->ny, g->nz}) {
        axis_plan(n, &ax);
        if (pass_threads(ax) > kMaxThreads || pass_smem(ax) > 227 * 1024) return false;
    }
    return true;
}

cudaError_t spectral_setup(const pf_grid* g, void* tables, SpectralPlan* P) {
    static const int key = 0;
    const cudaError_t e = once_per_context(&key, spectral_attributes);
    if (e != cudaSuccess) return e;
    P->d = Dims{g->nx, g->ny, g->nz, (long long)g->nx * g->ny * g->nz};
    P->tables = (double2*)tables;
    const double vol = (g->dx * g->dy) * g->dz;
    const double h[3] = {g->dx, g->dy, g->dz};
    const int n[3] = {g->nx, g->ny, g->nz};
    double2* tw = P->tables;
    for (int q = 0; q < 3; ++q) {
        axis_plan(n[q], &P->ax[q]);
        P->ax[q].tw = tw;
        tw += n[q];
        P->vol_d2[q] = vol / (h[q] * h[q]);
    }
    double* lam = (double*)tw;
    for (int q = 0; q < 3; ++q) { P->ax[q].lam = lam; lam += n[q]; }
    P->on = true;
    return cudaSuccess;
}

cudaError_t spectral_enqueue_tables(const SpectralPlan& P, cudaStream_t s) {
    TableArgs t;
    int most = 0;
    for (int q = 0; q < 3; ++q) {
        t.n[q] = P.ax[q].n;
        t.tw[q] = (double2*)P.ax[q].tw;
        t.lam[q] = (double*)P.ax[q].lam;
        t.f[q] = P.vol_d2[q];
        most = std::max(most, t.n[q]);
    }
    PF_LAUNCH("spectral_tables", s, launch_pdl(spectral_tables, dim3((most + 255) / 256, 3), dim3(256),
                                               0, s, t));
    return cudaGetLastError();
}

cudaError_t spectral_enqueue_solve(const SpectralPlan& P, const double* src, double c, double* DP,
                                   int* nonfin, cudaStream_t s) {
    const Dims& d = P.d;
    const bool al = ((uintptr_t)DP & 15) == 0;
    auto pairs = [](long long lines) { return (lines + 1) / 2; };
    PassArgs z{};
    z.ax = P.ax[2];
    z.src = src; z.dst = DP;
    z.nonfin = nonfin;
    z.nlines = (long long)d.nx * d.ny;
    z.stride = 1;
    const long long bz = (pairs(z.nlines) + z.ax.lines - 1) / z.ax.lines;
    PassArgs y{};
    y.ax = P.ax[1];
    y.src = DP; y.dst = DP;
    y.nlines = d.nz;
    y.stride = d.nz;
    y.tiles = (int)((pairs(d.nz) + y.ax.lines - 1) / y.ax.lines);
    y.vec = al && d.nz % 2 == 0;
    const long long by = (long long)d.nx * y.tiles;
    PassArgs x{};
    x.ax = P.ax[0];
    x.src = DP; x.dst = DP;
    x.nlines = (long long)d.ny * d.nz;
    x.stride = x.nlines;
    x.vec = al && x.nlines % 2 == 0;
    x.scale = c / (double)d.n;
    x.lamy = P.ax[1].lam; x.lamz = P.ax[2].lam;
    x.nz = d.nz;
    const long long bx = (pairs(x.nlines) + x.ax.lines - 1) / x.ax.lines;
    launch_pass<kPassZ>("spectral_z", z, bz, s);
    launch_pass<kPassY>("spectral_y", y, by, s);
    launch_pass<kPassX>("spectral_x", x, bx, s);
    launch_pass<kPassY>("spectral_y", y, by, s);
    z.src = DP;
    z.nonfin = nullptr;
    launch_pass<kPassZ>("spectral_z", z, bz, s);
    return cudaGetLastError();
}

}  // namespace pf
