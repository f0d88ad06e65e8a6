// Host build of the device arithmetic in ldg_common.cuh for comparisons with 64-bit results: the packed and the
// scalar FP32 routines and the FP64 eigen-solver, with one C entry each. The device intrinsics that they use are
// written here as what they are defined to compute (IEEE operations, rounded once).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#undef __device__
#undef __forceinline__
#undef __noinline__
#define __device__
#define __forceinline__ inline
#define __noinline__ __attribute__((noinline))

static inline float2 __ffma2_rn(float2 a, float2 b, float2 c) {
    return make_float2(std::fmaf(a.x, b.x, c.x), std::fmaf(a.y, b.y, c.y));
}
static inline float2 __fadd2_rn(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
static inline float2 __fmul2_rn(float2 a, float2 b) { return make_float2(a.x * b.x, a.y * b.y); }
static inline float __fadd_rn(float a, float b) { return a + b; }
static inline float __fsub_rn(float a, float b) { return a - b; }
static inline float __uint_as_float(unsigned u) {
    float f;
    std::memcpy(&f, &u, 4);
    return f;
}
static inline unsigned __umulhi(unsigned a, unsigned b) { return (unsigned)(((unsigned long long)a * b) >> 32); }
static inline float rsqrtf(float a) { return 1.0f / std::sqrt(a); }
template <class T>
static inline T __shfl_xor_sync(unsigned, T v, int) { return v; }
template <class T>
static inline T __shfl_down_sync(unsigned, T v, int) { return v; }
using std::max;
using std::min;

#include "ldg_common.cuh"

using namespace ldg;

namespace {

// FP32 field of n^3 cells, component-major, centred on a cell.
struct Cell {
    const float* q;
    int n, i, j, k;
    float operator()(int c, int di, int dj, int dk) const {
        const long long o = ((long long)(i + di) * n + j + dj) * n + k + dk, m = (long long)n * n * n;
        return c < 5 ? q[c * m + o] : -(q[o] + q[3 * m + o]);
    }
};
struct Divergence {
    const Cell& A;
    const QsrConst& P;
    float operator()(int c, int di, int dj, int dk) const {
        float D[3];
        dcol_at<false>(A, P, A.i, A.j, A.k, di, dj, dk, D);
        return D[c];
    }
};

QsrConst constants(double dx, const double e[6]) {  // L1, L2, L3, cQ, cQ2, cQ3
    QsrConst P{};
    const double ix2 = 1 / (dx * dx), i2 = 1 / (2 * dx);
    P.ix2 = P.iy2 = P.iz2 = (float)ix2;
    P.i2x = P.i2y = P.i2z = (float)i2;
    P.ix = P.iy = P.iz = (float)(1 / dx);
    P.i4xy = P.i4xz = P.i4yz = (float)(ix2 / 4);
    P.Liso = (float)e[0], P.L2 = (float)e[1], P.L3 = (float)e[2];
    P.cQ = (float)e[3], P.cQ2 = (float)e[4], P.cQ3 = (float)e[5];
    P.lap_c = (float)(-6 * ix2);
    P.L2i2x = P.L2i2y = P.L2i2z = (float)(e[1] * i2);
    P.lx = P.ly = P.lz = (float)(e[0] * ix2);
    for (int m = 0; m < 6; ++m) {
        P.l3m[m] = (float)(0.5 * e[2] * i2 * i2);
        P.l2w[m] = (float)(e[1] * i2 * i2);
        P.l3d[m] = (float)(e[2] * i2 * i2);
    }
    for (int m = 0; m < 3; ++m) P.l3s[m] = (float)(e[2] * ix2), P.l3c[m] = (float)(2 * e[2] * i2 * i2);
    return P;
}

template <bool kL2, bool kL3>
void chem(const float* q, int n, const QsrConst& P, bool packed, float* mu) {
    const long long m = (long long)n * n * n;
    for (int i = 2; i < n - 2; ++i)
        for (int j = 2; j < n - 3; j += 2)
            for (int k = 2; k < n - 2; ++k) {
                const long long o = ((long long)i * n + j) * n + k;
                if (packed) {
                    const Cell A{q, n, i, j, k};
                    F2 c[5], r[5], lap[5];
                    for (int x = 0; x < 5; ++x) c[x] = mk2(A(x, 0, 0, 0), A(x, 0, 1, 0));
                    const InteriorPair<kL2, kL3, Cell> S{A};
                    chem_core<kL2, kL3, false, false, F2>(S, P, c, F2{}, r, lap);
                    for (int x = 0; x < 5; ++x) mu[x * m + o] = r[x].v.x, mu[x * m + o + n] = r[x].v.y;
                } else {
                    for (int y = 0; y < 2; ++y) {
                        const Cell A{q, n, i, j + y, k};
                        const Divergence D{A, P};
                        float c[5], r[5], lap[5];
                        for (int x = 0; x < 5; ++x) c[x] = A(x, 0, 0, 0);
                        chem_potential<kL2, kL3, false>(A, D, P, i, j + y, k, c, false, r, lap);
                        for (int x = 0; x < 5; ++x) mu[x * m + o + y * n] = r[x];
                    }
                }
            }
}

}  // namespace

extern "C" {

// Chemical potential of the interior cells of an n^3 field; packed: the step kernels' two-cell form, else the
// term-by-term form of the one-thread-per-cell kernel.
void dm_chem(const float* q, int n, double dx, const double* e, int packed, float* mu) {
    const QsrConst P = constants(dx, e);
    const bool l2 = e[1] != 0.0, l3 = e[2] != 0.0;
    if (l2 && l3) chem<true, true>(q, n, P, packed, mu);
    else if (l2) chem<true, false>(q, n, P, packed, mu);
    else if (l3) chem<false, true>(q, n, P, packed, mu);
    else chem<false, false>(q, n, P, packed, mu);
}

// S and director of n tensors (five stored components each).
void dm_nematic(const double* q, long long n, double iso_cut, double* out) {
    for (long long t = 0; t < n; ++t) {
        const Nematic f = nematic64(q + 5 * t, iso_cut, Nematic{0.0, 0.0, 0.0, 1.0});
        out[4 * t] = f.S, out[4 * t + 1] = f.nx, out[4 * t + 2] = f.ny, out[4 * t + 3] = f.nz;
    }
}

}  // extern "C"
