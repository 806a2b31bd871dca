// pf_spectral_pass.cuh -- what the transform passes of the direct Poisson solve
// share: arguments of a pass, the small DFTs, the shared-memory layout.
#pragma once
#include "pf_common.cuh"
#include "pf_kernels.cuh"
#include "pf_spectral.cuh"

namespace pf {

enum { kPassZ = 0, kPassY = 1, kPassX = 2 };
constexpr int kHold = 8;          // complex values a thread holds
constexpr int kMaxThreads = 512;

struct PassArgs {
    SpectralAxis ax;
    const double* src;
    double* dst;
    long long nlines;   // real lines in all (z: rows; x: ny nz), or nz per i (y)
    long long stride;   // distance of consecutive elements of a line
    int tiles;          // y: tiles per x plane
    int vec;            // pairs of cells are 16-byte aligned
    // x pass
    double scale;       // c / (nx ny nz)
    const double *lamy, *lamz;
    int nz;
    int* nonfin;        // first z pass: set where the input is not finite
};

__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(fma(a.x, b.x, -(a.y * b.y)), fma(a.x, b.y, a.y * b.x));
}

// Forward DFT of R values in place.
template <int R>
struct Dft {
    // odd R: the terms j and R - j share their products
    static __device__ __forceinline__ void run(double2* a) {
        // cos, sin(2 pi m / R), m = 1 .. (R-1)/2
        constexpr double c3[1] = {-0.5}, s3[1] = {0.86602540378443864676};
        constexpr double c5[2] = {0.30901699437494742410, -0.80901699437494742410};
        constexpr double s5[2] = {0.95105651629515357212, 0.58778525229247312917};
        constexpr double c7[3] = {0.62348980185873353053, -0.22252093395631440429,
                                  -0.90096886790241912624};
        constexpr double s7[3] = {0.78183148246802980871, 0.97492791218182360702,
                                  0.43388373911755812048};
        constexpr int H = (R - 1) / 2;
        double2 t[H], u[H];
        double2 y0 = a[0];
#pragma unroll
        for (int j = 0; j < H; ++j) {
            t[j] = cadd(a[j + 1], a[R - 1 - j]);
            u[j] = csub(a[j + 1], a[R - 1 - j]);
            y0 = cadd(y0, t[j]);
        }
        const double2 a0 = a[0];
        a[0] = y0;
#pragma unroll
        for (int k = 1; k <= H; ++k) {
            double2 m = a0, s = make_double2(0.0, 0.0);
#pragma unroll
            for (int j = 0; j < H; ++j) {
                const int q = (j + 1) * k % R;
                const int h = q <= H ? q - 1 : R - q - 1;
                const double c = R == 3 ? c3[h % 1] : (R == 5 ? c5[h % 2] : c7[h % 3]);
                const double sv = R == 3 ? s3[h % 1] : (R == 5 ? s5[h % 2] : s7[h % 3]);
                const double sg = q <= H ? sv : -sv;
                m.x = fma(c, t[j].x, m.x);
                m.y = fma(c, t[j].y, m.y);
                s.x = fma(sg, u[j].x, s.x);
                s.y = fma(sg, u[j].y, s.y);
            }
            a[k] = make_double2(m.x + s.y, m.y - s.x);
            a[R - k] = make_double2(m.x - s.y, m.y + s.x);
        }
    }
};

template <>
struct Dft<2> {
    static __device__ __forceinline__ void run(double2* a) {
        const double2 t = csub(a[0], a[1]);
        a[0] = cadd(a[0], a[1]);
        a[1] = t;
    }
};

template <>
struct Dft<4> {
    static __device__ __forceinline__ void run(double2* a) {
        const double2 t0 = cadd(a[0], a[2]), t1 = csub(a[0], a[2]);
        const double2 t2 = cadd(a[1], a[3]), t3 = csub(a[1], a[3]);
        a[0] = cadd(t0, t2);
        a[2] = csub(t0, t2);
        a[1] = make_double2(t1.x + t3.y, t1.y - t3.x);
        a[3] = make_double2(t1.x - t3.y, t1.y + t3.x);
    }
};

template <>
struct Dft<8> {
    static __device__ __forceinline__ void run(double2* a) {
        double2 e[4] = {a[0], a[2], a[4], a[6]}, o[4] = {a[1], a[3], a[5], a[7]};
        Dft<4>::run(e);
        Dft<4>::run(o);
        const double c = 0.70710678118654752440;
        const double2 o1 = make_double2(c * (o[1].x + o[1].y), c * (o[1].y - o[1].x));
        const double2 o2 = make_double2(o[2].y, -o[2].x);
        const double2 o3 = make_double2(c * (o[3].y - o[3].x), -c * (o[3].x + o[3].y));
        a[0] = cadd(e[0], o[0]); a[4] = csub(e[0], o[0]);
        a[1] = cadd(e[1], o1);   a[5] = csub(e[1], o1);
        a[2] = cadd(e[2], o2);   a[6] = csub(e[2], o2);
        a[3] = cadd(e[3], o3);   a[7] = csub(e[3], o3);
    }
};

// slot of element e of line pair l
template <int L>
__device__ __forceinline__ int slot(int e, int l) { return e * L + (l ^ (e & (L - 1))); }

// Hartley values of the pair of real lines whose DFT is Z, from z = Z[k] and
// y = Z[n - k].
__device__ __forceinline__ double2 hartley(double2 z, double2 y) {
    return make_double2(0.5 * ((z.x + y.x) - (z.y - y.y)), 0.5 * ((z.y + y.y) + (z.x - y.x)));
}

typedef void (*PassKernel)(PassArgs);

// The kernel of an extent whose stages are laid out at compile time
// (pf_spectral_fast.cu), or nullptr.
PassKernel spectral_fast_kernel(int kind, int n);
cudaError_t spectral_fast_attributes();
constexpr int fast_lines(int n) { return n <= 512 ? 8 : 4; }  // line pairs per block

}  // namespace pf
