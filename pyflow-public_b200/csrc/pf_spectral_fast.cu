// pf_spectral_fast.cu -- the transform passes of pf_spectral.cu for extents
// 2^k, 3 2^k and 5 2^k that are multiples of 32, up to 1024, with every index
// known at compile time.
//
// The pass of any extent (pf_spectral.cu) is bound by the shared-memory pipe
// (77-81 % busy at 256^3) and by integer instructions: a value goes through
// shared memory once on arrival, once per stage and twice more for the Hartley
// values.  Here the first stage takes its values from global memory, and the
// last one, of radix 4, computes the butterflies k and n/4 - k in one thread,
// whose outputs are each other's mirror images, so the Hartley values are
// formed in registers and stored.  The x pass goes on from there: the scaled
// values are the input of the inverse transform's first butterfly.  At 256
// (8 8 4) a value crosses shared memory twice a transform, not five times.
//
// z, y and x pass, us, this form against the general one: 64^3 2.8 / 3.2 / 7.1
// against 5.9 / 4.0 / 9.3, 128^3 6.5 / 7.1 / 12.1 against 9.4 / 9.5 / 18.1, 192^3
// 27 / 25 / 43 against 52 / 55 / 97, 512^3 430 / 452 / 794 against 614 / 520 / 1072
// (a copy of the data takes 328).  With 80 registers for the x pass in place of
// 64 and a few spills: 15.6 us at 128^3, 1158 at 512^3.
#include "pf_spectral_pass.cuh"

namespace pf {
namespace {

#define PF_FAST_EXTENTS(X) \
    X(32) X(64) X(96) X(128) X(160) X(192) X(256) X(320) X(384) X(512) X(640) X(768) X(1024)

constexpr int kMaxFast = 4;
struct Radices { int n, r[kMaxFast]; };

// Stages of an extent, first to last; the last is a 4.
constexpr Radices radices(int n) {
    switch (n) {
        case 32: return {2, {8, 4}};
        case 64: return {3, {4, 4, 4}};
        case 96: return {3, {8, 3, 4}};
        case 128: return {3, {8, 4, 4}};
        case 160: return {3, {8, 5, 4}};
        case 192: return {4, {4, 3, 4, 4}};
        case 256: return {3, {8, 8, 4}};
        case 320: return {4, {4, 5, 4, 4}};
        case 384: return {4, {8, 3, 4, 4}};
        case 512: return {4, {8, 4, 4, 4}};
        case 640: return {4, {8, 5, 4, 4}};
        case 768: return {4, {8, 3, 8, 4}};
        case 1024: return {4, {8, 8, 4, 4}};
    }
    return {0, {}};
}

// product of the radices before stage s, of the transform forward or (inv) of
// the inverse one, which runs the stages in the other order
constexpr int before(int n, int s, bool inv) {
    const Radices R = radices(n);
    int p = 1;
    for (int q = 0; q < s; ++q) p *= R.r[inv ? R.n - 1 - q : q];
    return p;
}

// Slot of element e of line pair l: distinct banks for the L pairs of an
// element, for L consecutive elements and for L elements 4 or 8 apart.
template <int L>
__device__ __forceinline__ int at(int e, int l) { return e * L + (l ^ ((e ^ (e >> 3)) & (L - 1))); }

// Stage of radix R after PP: M butterflies per thread (N / 8 threads a line).
template <int N, int L, int R, int PP>
struct Stage {
    static constexpr int NR = N / R, TP = N / 8, M = (NR + TP - 1) / TP;
    static constexpr bool kAll = M * TP == NR;
    double2 x[M][R];
    static __device__ __forceinline__ int fly(int m, int it) {
        // a thread without a butterfly computes the first one and drops it
        return kAll || it + m * TP < NR ? it + m * TP : 0;
    }
    __device__ __forceinline__ void dft() {
#pragma unroll
        for (int m = 0; m < M; ++m) Dft<R>::run(x[m]);
    }
    __device__ __forceinline__ void read(const double2* sm, const double2* tw, int it, int l) {
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const int i = fly(m, it), k = i % PP;
#pragma unroll
            for (int q = 0; q < R; ++q) x[m][q] = sm[at<L>(i + q * NR, l)];
#pragma unroll
            for (int q = 1; q < R; ++q) x[m][q] = cmul(x[m][q], tw[q * k * (NR / PP)]);
        }
        dft();
    }
    __device__ __forceinline__ void write(double2* sm, int it, int l) const {
#pragma unroll
        for (int m = 0; m < M; ++m) {
            if (!kAll && it + m * TP >= NR) continue;
            const int i = it + m * TP, k = i % PP, jo = (i - k) * R + k;
#pragma unroll
            for (int q = 0; q < R; ++q) sm[at<L>(jo + q * PP, l)] = x[m][q];
        }
    }
};

// The stages from S up to the last but one, through shared memory.
template <int N, int L, int S, bool INV>
__device__ __forceinline__ void middle(double2* sm, const double2* tw, int it, int l) {
    constexpr Radices R = radices(N);
    if constexpr (S + 1 < R.n) {
        Stage<N, L, R.r[INV ? R.n - 1 - S : S], before(N, S, INV)> st;
        st.read(sm, tw, it, l);
        __syncthreads();
        st.write(sm, it, l);
        __syncthreads();
        middle<N, L, S + 1, INV>(sm, tw, it, l);
    }
}

constexpr int fast_threads(int n) { return n / 8 * fast_lines(n); }

template <int N, int KIND>
__global__ void __launch_bounds__(fast_threads(N), 1024 / fast_threads(N))
spectral_fast(PassArgs a) {
    constexpr int L = fast_lines(N), T = fast_threads(N), TP = N / 8;
    constexpr Radices R = radices(N);
    extern __shared__ __align__(16) double2 sm[];
    double2* tw = sm + N * L;
    const int tid = threadIdx.x;
    // element-wise threads (l, it); a z pass reads and writes its rows with
    // neighbouring threads on neighbouring elements (zl, zi)
    const int l = tid % L, it = tid / L;
    const int gl = KIND == kPassZ ? tid / TP : l, gi = KIND == kPassZ ? tid % TP : it;
    pdl_wait();
#pragma unroll
    for (int e = 0; e < N; e += T)
        if (N % T == 0 || e + tid < N) tw[e + tid] = a.ax.tw[e + tid];
    // lines a and b of this thread's pair: offset of the first, which exist
    long long base;
    bool ha, hb;
    long long col = 0;
    if (KIND == kPassZ) {
        const long long row = (long long)blockIdx.x * (2 * L) + 2 * gl;
        base = row * N;
        ha = row < a.nlines;
        hb = row + 1 < a.nlines;
    } else {
        long long plane = 0;
        int b = blockIdx.x;
        if (KIND == kPassY) {
            const int i = b / a.tiles;
            b -= i * a.tiles;
            plane = (long long)i * N * a.stride;
        }
        col = (long long)b * (2 * L) + 2 * l;
        base = plane + col;
        ha = col < a.nlines;
        hb = col + 1 < a.nlines;
    }
    const long long step = KIND == kPassZ ? 1 : a.stride;  // of elements; a pair's lines are `other` apart
    const long long other = KIND == kPassZ ? N : 1;
    const bool two = KIND != kPassZ && a.vec && hb;
    auto put = [&](int e, double2 h) {
        double* o = a.dst + base + e * step;
        if (two) {
            *(double2*)o = h;
        } else {
            if (ha) o[0] = h.x;
            if (hb) o[other] = h.y;
        }
    };
    {
        Stage<N, L, R.r[0], 1> st;
        const double* p = a.src + base;
#pragma unroll
        for (int m = 0; m < st.M; ++m)
#pragma unroll
            for (int q = 0; q < R.r[0]; ++q) {
                const double* o = p + (st.fly(m, gi) + q * st.NR) * step;
                if (two) st.x[m][q] = *(const double2*)o;
                else st.x[m][q] = make_double2(ha ? o[0] : 0.0, hb ? o[other] : 0.0);
            }
        if (KIND == kPassZ && a.nonfin) {
            double big = 0.0;
#pragma unroll
            for (int m = 0; m < st.M; ++m)
#pragma unroll
                for (int q = 0; q < R.r[0]; ++q)
                    big = absmax(big, absmax(abs_bits(st.x[m][q].x), abs_bits(st.x[m][q].y)));
            if (!(big < __longlong_as_double(0x7ff0000000000000LL))) *a.nonfin = 1;
        }
        st.dft();
        st.write(sm, gi, gl);
    }
    __syncthreads();
    middle<N, L, 1, false>(sm, tw, it, l);
    // last stage, radix 4: the butterflies i and j = n/4 - i (0: 0 and n/8, each
    // its own mirror image)
    constexpr int P = N / 4;
    const int i = gi, j = gi ? P - gi : N / 8;
    double2 x[2][4], y[2][4];
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        const int k = m ? j : i;
#pragma unroll
        for (int q = 0; q < 4; ++q) x[m][q] = sm[at<L>(k + q * P, gl)];
#pragma unroll
        for (int q = 1; q < 4; ++q) x[m][q] = cmul(x[m][q], tw[q * k]);
        Dft<4>::run(x[m]);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        y[0][q] = i ? x[1][3 - q] : x[0][(4 - q) & 3];
        y[1][q] = i ? x[0][3 - q] : x[1][3 - q];
    }
    if (KIND != kPassX) {
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int q = 0; q < 4; ++q) put((m ? j : i) + q * P, hartley(x[m][q], y[m][q]));
        return;
    }
    // x pass: the transforms of the two lines times their own factors s/lambda
    // (equal at k and n - k): W = (ma + mb)/2 Z[k] + (ma - mb)/2 conj Z[n-k].
    // The inverse DFT of W is the forward one with real and imaginary parts
    // exchanged on the way in and out.
    {
        double la = 0.0, lb = 0.0;
        if (ha) {
            const int jy = (int)((unsigned)col / (unsigned)a.nz), kz = (int)col - jy * a.nz;
            la = a.lamy[jy] + a.lamz[kz];
            const int j2 = kz + 1 < a.nz ? jy : jy + 1, k2 = kz + 1 < a.nz ? kz + 1 : 0;
            lb = hb ? a.lamy[j2] + a.lamz[k2] : 1.0;
        }
#pragma unroll
        for (int m = 0; m < 2; ++m) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const double lx = a.ax.lam[(m ? j : i) + q * P];
                const double va = lx + la, vb = lx + lb;
                // the constant mode (zero eigenvalue) has no part in the solution
                const double ma = va > 0.0 ? a.scale / va : 0.0, mb = vb > 0.0 ? a.scale / vb : 0.0;
                const double s = 0.5 * (ma + mb), t = 0.5 * (ma - mb);
                const double2 z = x[m][q], w = y[m][q];
                x[m][q] = make_double2(fma(s, z.y, -(t * w.y)), fma(s, z.x, t * w.x));
            }
        }
        __syncthreads();
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            Dft<4>::run(x[m]);
#pragma unroll
            for (int q = 0; q < 4; ++q) sm[at<L>((m ? j : i) * 4 + q, l)] = x[m][q];
        }
    }
    __syncthreads();
    middle<N, L, 1, true>(sm, tw, it, l);
    Stage<N, L, R.r[0], N / R.r[0]> st;
    st.read(sm, tw, it, l);
#pragma unroll
    for (int m = 0; m < st.M; ++m)
#pragma unroll
        for (int q = 0; q < R.r[0]; ++q)
            put(it + m * TP + q * st.NR, make_double2(st.x[m][q].y, st.x[m][q].x));
}

template <int N>
PassKernel kernel_of(int kind) {
    static_assert(radices(N).r[0] == 8 || radices(N).r[0] == 4, "first stage: no idle butterflies");
    return kind == kPassZ ? spectral_fast<N, kPassZ>
                          : (kind == kPassY ? spectral_fast<N, kPassY> : spectral_fast<N, kPassX>);
}

}  // namespace

PassKernel spectral_fast_kernel(int kind, int n) {
    switch (n) {
#define PF_FAST(N) case N: return kernel_of<N>(kind);
        PF_FAST_EXTENTS(PF_FAST)
#undef PF_FAST
    }
    return nullptr;
}

cudaError_t spectral_fast_attributes() {
#define PF_FAST(N) N,
    for (int n : {PF_FAST_EXTENTS(PF_FAST)})
#undef PF_FAST
        for (int kind : {kPassZ, kPassY, kPassX}) {
            const cudaError_t e =
                cudaFuncSetAttribute(spectral_fast_kernel(kind, n),
                                     cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     n * (fast_lines(n) + 1) * (int)sizeof(double2));
            if (e != cudaSuccess) return e;
        }
    return cudaSuccess;
}

}  // namespace pf
