// Confined droplet solver: device kernels and the qsr_* C ABI (include/ldg_b200.h).
//
// Device layout: two FP32 SoA field buffers (ping-pong), one uint8 classification per cell,
// an FP32 SoA right-hand side for the IMEX path, and an FP64 AoS staging buffer for the
// host boundary. One fused kernel per explicit step reads each Q component once per cell
// and writes it once (the reference runs 5-7 separate FP64 AoS passes).
#include <omp.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <limits>
#include <new>
#include <random>
#include <vector>

#include "ldg_api_common.h"
#include "ldg_common.cuh"
#include "qsr_tiled.cuh"

using namespace ldg;

namespace {

constexpr double kPi = 3.14159265358979323846;

// ---------------------------------------------------------------------------------------
// Host FP64 geometry: the reference's droplet (QSR.cu:34-185), evaluated once per handle.
// ---------------------------------------------------------------------------------------
struct Geometry {
    double dx, dy, dz, cx, cy, cz, rx, ry, rz, min_spacing, min_radius, shell_half, core_radius;
};

Geometry make_geometry(const qsr_params& p) {
    Geometry g{};
    g.dx = p.dx; g.dy = p.dy; g.dz = p.dz;
    g.cx = 0.5 * ((double)p.Nx - 1.0) * p.dx;
    g.cy = 0.5 * ((double)p.Ny - 1.0) * p.dy;
    g.cz = 0.5 * ((double)p.Nz - 1.0) * p.dz;
    double ridx = 0.5 * ((double)std::min({p.Nx, p.Ny, p.Nz}) - 1.0);
    if (p.droplet_radius_cells > 0.0) ridx = p.droplet_radius_cells;
    g.rx = std::max(ridx * p.dx, 0.5 * p.dx);
    g.ry = std::max(ridx * p.dy, 0.5 * p.dy);
    g.rz = std::max(ridx * p.dz, 0.5 * p.dz);
    g.min_spacing = std::min({p.dx, p.dy, p.dz});
    g.min_radius = std::min({g.rx, g.ry, g.rz});
    g.shell_half = g.min_spacing;
    g.core_radius = g.min_spacing;
    return g;
}

// Signed distance proxy (rho - 1)/|grad rho| and distance from the centre (QSR.cu:70-98).
inline void signed_distance(const Geometry& g, int i, int j, int k, double& sd, double& r) {
    const double x = i * g.dx - g.cx, y = j * g.dy - g.cy, z = k * g.dz - g.cz;
    r = std::sqrt(x * x + y * y + z * z);
    const double sx = x / g.rx, sy = y / g.ry, sz = z / g.rz;
    const double rho_sq = sx * sx + sy * sy + sz * sz;
    if (rho_sq <= 1e-30) { sd = -g.min_radius; return; }
    const double rho = std::sqrt(rho_sq);
    const double gx = x / (g.rx * g.rx), gy = y / (g.ry * g.ry), gz = z / (g.rz * g.rz);
    const double gn = std::sqrt(gx * gx + gy * gy + gz * gz) / rho;
    sd = (gn > 1e-30) ? (rho - 1.0) / gn : r - g.min_radius;
}

// ---------------------------------------------------------------------------------------
// Kernels
// ---------------------------------------------------------------------------------------

// Global-memory neighbour accessor for the direct kernels.
struct GAcc {
    const float* __restrict__ q;
    long long id, si, sc;
    int sj;
    __device__ __forceinline__ float operator()(int c, int di, int dj, int dk) const {
        const long long o = id + di * si + (long long)dj * sj + dk;
        if (c < 5) return __ldg(q + c * sc + o);
        return -(__ldg(q + o) + __ldg(q + 3 * sc + o));
    }
};

// Column divergence computed on the fly from the Q accessor (v1 path).
struct GDAcc {
    const GAcc* A;
    const QsrConst* P;
    int i, j, k;
    __device__ __forceinline__ float operator()(int comp, int di, int dj, int dk) const {
        float D[3];
        dcol_at(*A, *P, i, j, k, di, dj, dk, D);
        return D[comp];
    }
};

// One explicit step (RHS=false) or the IMEX right-hand side (RHS=true) for every cell of
// the box. Block (32, 8): k fastest, then j; grid z runs over i.
template <bool kL2, bool kL3, bool kNoise, bool kRHS>
__global__ void __launch_bounds__(256) k_step_direct(const float* __restrict__ q, float* __restrict__ out,
                                                     const uint8_t* __restrict__ flags, QsrConst P) {
    const int k = blockIdx.x * 32 + threadIdx.x;
    const int j = blockIdx.y * 8 + threadIdx.y;
    const int i = blockIdx.z;
    if (k >= P.Nz || j >= P.Ny) return;
    const long long id = (long long)i * P.si + (long long)j * P.sj + k;
    const uint8_t f = flags[id];
    float c[5], o[5];
#pragma unroll
    for (int m = 0; m < 5; ++m) c[m] = __ldg(q + m * P.sc + id);
    if (!kRHS && (f & kFixed)) {
        surface_q0(P, i, j, k, o);
    } else if (f & kMove) {
        GAcc A{q, id, P.si, P.sc, P.sj};
        GDAcc DA{&A, &P, i, j, k};
        float mu[5], lap[5];
        chem_potential<kL2, kL3>(A, DA, P, i, j, k, c, (f & kAnchor) != 0, mu, lap);
        const uint32_t cell = (uint32_t)(k + P.Nz * (j + P.Ny * i));
        if (kRHS) {
            // computeRhsSemiImplicitKernel (QSR.cu:775-783).
#pragma unroll
            for (int m = 0; m < 5; ++m) o[m] = c[m] - P.mob_dt * mu[m] - P.alpha * lap[m];
            if (kNoise) {
                float g[5];
                normals5(cell, P.instance, P.step, P.key0, P.key1, g);
#pragma unroll
                for (int m = 0; m < 5; ++m) o[m] += P.sigma * g[m];
            }
        } else {
            euler_update(P, c, mu, cell, kNoise, o);
        }
    } else {
#pragma unroll
        for (int m = 0; m < 5; ++m) o[m] = c[m];
    }
#pragma unroll
    for (int m = 0; m < 5; ++m) out[m * P.sc + id] = o[m];
}

// One Jacobi sweep of (I - alpha Lap) Q = rhs with faces and non-moving cells held
// (QSR.cu:786-849). LAST also applies the strong-anchoring rewrite (QSR.cu:851-867).
template <bool kLast>
__global__ void __launch_bounds__(256) k_jacobi(const float* __restrict__ rhs, const float* __restrict__ qo,
                                                float* __restrict__ qn, const uint8_t* __restrict__ flags, QsrConst P) {
    const int k = blockIdx.x * 32 + threadIdx.x;
    const int j = blockIdx.y * 8 + threadIdx.y;
    const int i = blockIdx.z;
    if (k >= P.Nz || j >= P.Ny) return;
    const long long id = (long long)i * P.si + (long long)j * P.sj + k;
    const uint8_t f = flags[id];
    float o[5];
    if (kLast && (f & kFixed)) {
        surface_q0(P, i, j, k, o);
    } else {
        const bool face = (i == 0 || j == 0 || k == 0 || i == P.Nx - 1 || j == P.Ny - 1 || k == P.Nz - 1);
        if (face || !(f & kMove)) {
#pragma unroll
            for (int m = 0; m < 5; ++m) o[m] = __ldg(qo + m * P.sc + id);
        } else {
#pragma unroll
            for (int m = 0; m < 5; ++m) {
                const float* b = qo + m * P.sc + id;
                const float s = P.ix2 * (__ldg(b + P.si) + __ldg(b - P.si)) +
                                P.iy2 * (__ldg(b + P.sj) + __ldg(b - P.sj)) + P.iz2 * (__ldg(b + 1) + __ldg(b - 1));
                o[m] = (__ldg(rhs + m * P.sc + id) + P.alpha * s) * P.jdenom_inv;
            }
        }
    }
#pragma unroll
    for (int m = 0; m < 5; ++m) qn[m * P.sc + id] = o[m];
}

// Host AoS FP64 (reference cell order) <-> device FP32 SoA.
__global__ void k_aos_to_soa(const double* __restrict__ aos, float* __restrict__ a, float* __restrict__ b,
                             int Nx, int Ny, int Nz, int sj, long long si, long long sc, float* __restrict__ la = nullptr,
                             float* __restrict__ lb = nullptr) {
    const long long n = (long long)Nx * Ny * Nz;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        const int k = (int)(t % Nz);
        const long long r = t / Nz;
        const int j = (int)(r % Ny);
        const int i = (int)(r / Ny);
        const long long id = (long long)i * si + (long long)j * sj + k;
#pragma unroll
        for (int m = 0; m < 5; ++m) {
            const double x = aos[5 * t + m];
            const float v = (float)x;
            a[m * sc + id] = v;
            b[m * sc + id] = v;
            if (la) {
                const float r = (float)(x - (double)v);  // low word of compensated storage
                la[m * sc + id] = r;
                lb[m * sc + id] = r;
            }
        }
    }
}

__global__ void k_soa_to_aos(const float* __restrict__ a, double* __restrict__ aos, int Nx, int Ny, int Nz, int sj,
                             long long si, long long sc, const float* __restrict__ lo = nullptr) {
    const long long n = (long long)Nx * Ny * Nz;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        const int k = (int)(t % Nz);
        const long long r = t / Nz;
        const int j = (int)(r % Ny);
        const int i = (int)(r / Ny);
        const long long id = (long long)i * si + (long long)j * sj + k;
#pragma unroll
        for (int m = 0; m < 5; ++m)
            aos[5 * t + m] = (double)a[m * sc + id] + (lo ? (double)lo[m * sc + id] : 0.0);
    }
}

__global__ void k_nematic_out(const float* __restrict__ a, double* __restrict__ out4, int Nx, int Ny, int Nz, int sj,
                              long long si, long long sc) {
    const long long n = (long long)Nx * Ny * Nz;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        const int k = (int)(t % Nz);
        const long long r = t / Nz;
        const int j = (int)(r % Ny);
        const int i = (int)(r / Ny);
        const long long id = (long long)i * si + (long long)j * sj + k;
        double q[5];
#pragma unroll
        for (int m = 0; m < 5; ++m) q[m] = (double)a[m * sc + id];
        const Nematic nf = nematic64(q, 1e-9, Nematic{0.0, 0.0, 0.0, 1.0});
        out4[4 * t + 0] = nf.S;
        out4[4 * t + 1] = nf.nx;
        out4[4 * t + 2] = nf.ny;
        out4[4 * t + 3] = nf.nz;
    }
}

// ---------------------------------------------------------------------------------------
// FP64 observables, one launch: the first blocks take the volume sums, the others the slice metrics.
// Every block writes one partial; the last one to finish adds the partials in block order, so results
// do not depend on scheduling.
// ---------------------------------------------------------------------------------------
enum ObsSum { kBulk, kElastic, kAnch, kRad, kSumS, kEven, kOdd, kXi, kObsSums, kMaxS = kObsSums, kMaxQ, kObsVals };
enum ObsCount { kRadN, kCoreN, kEvenN, kOddN, kNonfinite, kDefects, kPlaq, kEdges, kObsCounts };
struct ObsPartial {
    double v[kObsVals];                  // sums, then maxima
    unsigned long long n[kObsCounts];
};

struct ObsConst {
    QsrConst P;
    double i2x, i2y, i2z;
    double c2, c3, c4;         // bulk energy coefficients (QSR.cu:887-899)
    double Liso, L2, L3;       // kappa if L1 = L2 = L3 = 0, else L1 (QSR.cu:955-987)
    double dV, Weff_half;      // cell volume; 0.5*W/delta_eff
    double S_shell;
    double cx, cy, cz, gx, gy, gz;  // FP64 geometry for normals and radial directions (cell units)
    double hx, hy, hz;               // spacing
    int checker_k;
    int mode;                  // bit 0: defects on slice dk, bit 1: xi proxy on slice xk
    int dk, xk;
    double dthr, dcut, xthr;
    int volume_blocks;
};

constexpr int kObsThreads = 256, kObsWarps = kObsThreads / 32;
// 128 registers: two blocks per SM. (With the FP64 state of a cell in 156 to 255 registers one block
// fitted, and 16 reductions with a block barrier each cost as much as the cells of a 64^3 grid.)
constexpr int kObsPerSM = 2;
constexpr int kObsVolumeBlocks = 148 * 2 * kObsPerSM, kObsSliceBlocks = 148;
constexpr size_t kObsBytes = (kObsVolumeBlocks + kObsSliceBlocks + 1) * sizeof(ObsPartial) + sizeof(unsigned);

// Volume terms of cell (i, j, k).
__device__ __forceinline__ void observe_cell(const float* __restrict__ q, const uint8_t* __restrict__ flags,
                                             const ObsConst& O, int i, int j, int k, double v[kObsVals],
                                             unsigned n[kObsCounts]) {
    const QsrConst& P = O.P;
    const long long id = (long long)i * P.si + (long long)j * P.sj + k;
    const uint8_t f = flags[id];
    const float* b = q + id;
    double c[5];
    unsigned bits = 0;
    bool finite = true;
#pragma unroll
    for (int m = 0; m < 5; ++m) {
        const float x = b[m * P.sc];
        bits |= __float_as_uint(x);
        c[m] = (double)x;
        finite = finite && isfinite(x);
    }
    if (!finite) n[kNonfinite]++;
    const double Qxx = c[0], Qxy = c[1], Qxz = c[2], Qyy = c[3], Qyz = c[4], Qzz = -Qxx - Qyy;
    const double trQ2 = Qxx * Qxx + Qyy * Qyy + Qzz * Qzz + 2 * (Qxy * Qxy + Qxz * Qxz + Qyz * Qyz);
    v[kMaxQ] = fmax(v[kMaxQ], trQ2);  // squared; the root is taken at the end
    const bool interior = (i >= 1 && j >= 1 && k >= 1 && i < P.Nx - 1 && j < P.Ny - 1 && k < P.Nz - 1);
    // Outside the droplet a field that is zero, neighbours included, adds nothing.
    if (interior && !(f & (kInside | kShell))) {
#pragma unroll
        for (int m = 0; m < 5; ++m) {
            const float* p = b + m * P.sc;
            bits |= __float_as_uint(p[P.si]) | __float_as_uint(p[-P.si]) | __float_as_uint(p[P.sj]) |
                    __float_as_uint(p[-P.sj]) | __float_as_uint(p[1]) | __float_as_uint(p[-1]);
        }
    } else {
        bits = 1;
    }
    if (interior && bits != 0) {
        // computeEnergyKernel (QSR.cu:869-992); tr Q^3 = 3 det Q of a traceless Q
        const double det = Qxx * (Qyy * Qzz - Qyz * Qyz) - Qxy * (Qxy * Qzz - Qyz * Qxz) + Qxz * (Qxy * Qyz - Qyy * Qxz);
        v[kBulk] += O.c2 * trQ2 - 3.0 * O.c3 * det + O.c4 * trQ2 * trQ2;
        double d[5][3];
#pragma unroll
        for (int m = 0; m < 5; ++m) {
            const float* p = b + m * P.sc;
            d[m][0] = ((double)p[P.si] - (double)p[-P.si]) * O.i2x;
            d[m][1] = ((double)p[P.sj] - (double)p[-P.sj]) * O.i2y;
            d[m][2] = ((double)p[1] - (double)p[-1]) * O.i2z;
        }
        // M_xy = dQ_kl/dx dQ_kl/dy over all nine entries, dQ_zz = -(dQ_xx + dQ_yy)
        auto M = [&](int x, int y) {
            return 2.0 * (d[0][x] * (d[0][y] + 0.5 * d[3][y]) + d[3][x] * (d[3][y] + 0.5 * d[0][y]) + d[1][x] * d[1][y] +
                          d[2][x] * d[2][y] + d[4][x] * d[4][y]);
        };
        const double m00 = M(0, 0), m11 = M(1, 1), m22 = M(2, 2);
        double fel = 0.5 * O.Liso * (m00 + m11 + m22);
        if (O.L2 != 0.0) {
            const double vx = d[0][0] + d[1][1] + d[2][2];
            const double vy = d[1][0] + d[3][1] + d[4][2];
            const double vz = d[2][0] + d[4][1] - (d[0][2] + d[3][2]);
            fel += 0.5 * O.L2 * (vx * vx + vy * vy + vz * vz);
        }
        if (O.L3 != 0.0)
            fel += 0.5 * O.L3 * (Qxx * m00 + Qyy * m11 + Qzz * m22 +
                                 2.0 * (Qxy * M(0, 1) + Qxz * M(0, 2) + Qyz * M(1, 2)));
        v[kElastic] += fel;
    }
    const double X = ((double)i - O.cx), Y = ((double)j - O.cy), Z = ((double)k - O.cz);
    if (f & kAnchor) {
        // computeAnchoringEnergyKernel (QSR.cu:654-695).
        const double gx = X * O.gx, gy = Y * O.gy, gz = Z * O.gz;
        const double gn = sqrt(gx * gx + gy * gy + gz * gz);
        double nx = 1.0, ny = 0.0, nz = 0.0;
        if (gn > 0.0) { nx = gx / gn; ny = gy / gn; nz = gz / gn; }
        const double S = O.S_shell;
        const double q0xx = S * (nx * nx - 1.0 / 3.0), q0xy = S * (nx * ny), q0xz = S * (nx * nz);
        const double q0yy = S * (ny * ny - 1.0 / 3.0), q0yz = S * (ny * nz), q0zz = -(q0xx + q0yy);
        const double dxx = Qxx - q0xx, dxy = Qxy - q0xy, dxz = Qxz - q0xz, dyy = Qyy - q0yy, dyz = Qyz - q0yz;
        const double dzz = Qzz - q0zz;
        v[kAnch] += dxx * dxx + dyy * dyy + dzz * dzz + 2.0 * (dxy * dxy + dxz * dxz + dyz * dyz);
    }
    if (f & (kRadial | kCore)) {
        const Nematic nf = nematic64(c, 1e-9, Nematic{0.0, 0.0, 0.0, 1.0});
        if (f & kRadial) {
            // computeRadialityKernel (QSR.cu:994-1015): r-hat from the centre.
            const double px = X * O.hx, py = Y * O.hy, pz = Z * O.hz;
            const double rr = sqrt(px * px + py * py + pz * pz);
            v[kRad] += rr > 1e-30 ? fabs(nf.nx * px + nf.ny * py + nf.nz * pz) / rr : fabs(nf.nx);
            n[kRadN]++;
        }
        if (f & kCore) {
            v[kSumS] += nf.S;
            n[kCoreN]++;
            if (isfinite(nf.S)) v[kMaxS] = fmax(v[kMaxS], nf.S);
            if (k == O.checker_k && isfinite(nf.S) && nf.S > 0.01) {
                // Checkerboard sums on the defect slice (QSR.cu:2845-2868).
                if (((i + j) & 1) == 0) { v[kEven] += nf.S; n[kEvenN]++; }
                else { v[kOdd] += nf.S; n[kOddN]++; }
            }
        }
    }
}

__device__ __forceinline__ double wrap_pi(double x) {
    // wrap_to_pi_device (QSR.cu:1027-1035).
    const double two_pi = 2.0 * kPi;
    x = x + kPi;
    x -= floor(x / two_pi) * two_pi;
    return x - kPi;
}

// Plaquette winding (QSR.cu:1114-1176) and wrapped phase-gradient edges (QSR.cu:1042-1106) of cell
// (i, j) with its neighbours at i + 1 and j + 1, on the defect and the xi slice.
__device__ __forceinline__ void observe_slice(const float* __restrict__ q, const ObsConst& O, int i, int j,
                                              double v[kObsVals], unsigned n[kObsCounts]) {
    const QsrConst& P = O.P;
    struct Site {
        double S, psi;
        bool fine;
    };
    auto site = [&](int ii, int jj, int k) {
        double c[5];
        const long long id = (long long)ii * P.si + (long long)jj * P.sj + k;
#pragma unroll
        for (int m = 0; m < 5; ++m) c[m] = (double)q[m * P.sc + id];
        const Nematic f = nematic64(c, 1e-9, Nematic{0.0, 0.0, 0.0, 1.0});
        return Site{f.S, 2.0 * atan2(f.ny, f.nx), isfinite(f.S) && isfinite(f.nx) && isfinite(f.ny)};
    };
    const bool ip = i < P.Nx - 1, jp = j < P.Ny - 1;
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
        const bool dfc = (O.mode & 1) && pass == 0, xi = (O.mode & 2) && (O.xk == O.dk && (O.mode & 1) ? pass == 0 : pass == 1);
        if (!dfc && !xi) continue;
        const int k = pass == 0 ? O.dk : O.xk;
        const Site s00 = site(i, j, k), s10 = ip ? site(i + 1, j, k) : s00, s01 = jp ? site(i, j + 1, k) : s00;
        if (dfc && ip && jp) {
            const Site s11 = site(i + 1, j + 1, k);
            auto ok = [&](const Site& s) { return s.fine && s.S > O.dthr; };
            if (ok(s00) && ok(s10) && ok(s11) && ok(s01)) {
                const double dsum = wrap_pi(s10.psi - s00.psi) + wrap_pi(s11.psi - s10.psi) + wrap_pi(s01.psi - s11.psi) +
                                    wrap_pi(s00.psi - s01.psi);
                n[kPlaq]++;
                if (fabs(0.5 * (dsum * (1.0 / (2.0 * kPi)))) > O.dcut) n[kDefects]++;
            }
        }
        if (xi) {
            auto edge = [&](bool in, const Site& s) {
                if (!(in && s00.fine && s.fine && s00.S > O.xthr && s.S > O.xthr)) return;
                const double d = wrap_pi(s.psi - s00.psi);
                v[kXi] += d * d;
                n[kEdges]++;
            };
            edge(ip, s10);
            edge(jp, s01);
        }
    }
}

// Adds the threads' values of a block in a fixed order; valid in threads 0 .. kObsVals + kObsCounts - 1,
// which write them to `out`. One block barrier.
template <class N>
__device__ __forceinline__ void observe_block(const double v[kObsVals], const N n[kObsCounts], ObsPartial* out) {
    __shared__ double sv[kObsWarps][kObsVals];
    __shared__ unsigned long long sn[kObsWarps][kObsCounts];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int m = 0; m < kObsVals; ++m) {
        const double r = m < kObsSums ? warp_sum(v[m]) : warp_max(v[m]);
        if (lane == 0) sv[w][m] = r;
    }
#pragma unroll
    for (int m = 0; m < kObsCounts; ++m) {
        const unsigned long long r = warp_sum((unsigned long long)n[m]);
        if (lane == 0) sn[w][m] = r;
    }
    __syncthreads();
    const int t = threadIdx.x;
    if (t < kObsVals) {
        double r = 0.0;
        for (int x = 0; x < kObsWarps; ++x) r = t < kObsSums ? r + sv[x][t] : fmax(r, sv[x][t]);
        out->v[t] = r;
    } else if (t < kObsVals + kObsCounts) {
        unsigned long long r = 0;
        for (int x = 0; x < kObsWarps; ++x) r += sn[x][t - kObsVals];
        out->n[t - kObsVals] = r;
    }
}

__global__ void __launch_bounds__(kObsThreads, kObsPerSM) k_observe(const float* __restrict__ q,
                                                                    const uint8_t* __restrict__ flags, ObsConst O,
                                                                    ObsPartial* __restrict__ part,
                                                                    unsigned* __restrict__ ticket,
                                                                    ObsPartial* __restrict__ out) {
    const QsrConst& P = O.P;
    double v[kObsVals] = {};
    unsigned n[kObsCounts] = {};
    if ((int)blockIdx.x < O.volume_blocks) {
        // A warp takes a row of cells at a time: one division per row instead of two per cell.
        const int lane = threadIdx.x & 31;
        const long long rows = (long long)P.Nx * P.Ny, warps = (long long)O.volume_blocks * kObsWarps;
        for (long long r = (long long)blockIdx.x * kObsWarps + (threadIdx.x >> 5); r < rows; r += warps) {
            const int i = (int)(r / P.Ny), j = (int)(r - (long long)i * P.Ny);
            for (int k = lane; k < P.Nz; k += 32) observe_cell(q, flags, O, i, j, k, v, n);
        }
        v[kBulk] *= O.dV;
        v[kElastic] *= O.dV;
        v[kAnch] *= O.Weff_half * O.dV;
        v[kMaxQ] = sqrt(v[kMaxQ]);
    } else {
        const long long cells = (long long)P.Nx * P.Ny, step = (long long)(gridDim.x - O.volume_blocks) * kObsThreads;
        for (long long t = (long long)(blockIdx.x - O.volume_blocks) * kObsThreads + threadIdx.x; t < cells; t += step)
            observe_slice(q, O, (int)(t / P.Ny), (int)(t % P.Ny), v, n);
    }
    observe_block(v, n, &part[blockIdx.x]);
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    double tv[kObsVals] = {};
    unsigned long long tn[kObsCounts] = {};
    for (unsigned b = threadIdx.x; b < gridDim.x; b += kObsThreads) {
#pragma unroll
        for (int m = 0; m < kObsVals; ++m) {
            const double x = __ldcg(&part[b].v[m]);
            tv[m] = m < kObsSums ? tv[m] + x : fmax(tv[m], x);
        }
#pragma unroll
        for (int m = 0; m < kObsCounts; ++m) tn[m] += __ldcg(&part[b].n[m]);
    }
    __syncthreads();  // the shared arrays of the first reduction are read
    observe_block(tv, tn, out);
    if (threadIdx.x == 0) *ticket = 0;
}

}  // namespace

// ---------------------------------------------------------------------------------------
// Handle and C ABI
// ---------------------------------------------------------------------------------------
struct qsr_handle {
    qsr_params p{};
    Geometry g{};
    double delta_eff = 0.0;
    long long shell_cells = 0, evolving_cells = 0, active_cells = 0, written_cells = 0;
    int sj = 0;
    long long si = 0, sc = 0, ncells = 0;
    float* q[2] = {nullptr, nullptr};
    float* lo[2] = {nullptr, nullptr};  // low words of compensated storage (optional)
    float* rhs = nullptr;
    uint8_t* flags = nullptr;
    double* stage = nullptr;       // FP64 AoS staging (5 or 4 doubles per cell)
    bool stage_shared = false;     // staging owned by an ensemble (shared by its droplets)
    ObsPartial* opart = nullptr;   // block partials, the result, then the ticket counter
    TiledPlan tiled{};             // tiled-kernel launch plan
    TiledPlan sweep{};             // plan of the IMEX sweeps (shares the other one's error word)
    CUtensorMap rhs_map;
    int cur = 0;
    bool uploaded = false;
    cudaStream_t stream = nullptr;
    long long launches = 0;
    int device = -1;               // the GPU the handle was created on
};

namespace {

QsrConst make_const(const qsr_handle* h, double T, double S_shell, double dt) {
    const qsr_params& p = h->p;
    QsrConst P{};
    P.Nx = p.Nx; P.Ny = p.Ny; P.Nz = p.Nz;
    P.sj = h->sj; P.si = h->si; P.sc = h->sc;
    P.ix2 = (float)(1.0 / (p.dx * p.dx)); P.iy2 = (float)(1.0 / (p.dy * p.dy)); P.iz2 = (float)(1.0 / (p.dz * p.dz));
    P.i2x = (float)(1.0 / (2.0 * p.dx)); P.i2y = (float)(1.0 / (2.0 * p.dy)); P.i2z = (float)(1.0 / (2.0 * p.dz));
    P.ix = (float)(1.0 / p.dx); P.iy = (float)(1.0 / p.dy); P.iz = (float)(1.0 / p.dz);
    P.i4xy = (float)(1.0 / (4.0 * p.dx * p.dy));
    P.i4xz = (float)(1.0 / (4.0 * p.dx * p.dz));
    P.i4yz = (float)(1.0 / (4.0 * p.dy * p.dz));
    const double dT = T - p.T_star;
    const double cQ = 3.0 * p.a * dT;
    const double cQ2 = (p.bulk_modechoice == 1) ? (9.0 * p.b) / 2.0 : (27.0 * p.b) / 2.0;
    const double cQ3 = (p.bulk_modechoice == 1) ? (9.0 * p.c) / 2.0 : 9.0 * p.c;
    P.cQ = (float)cQ; P.cQ2 = (float)cQ2; P.cQ3 = (float)cQ3;
    const bool all_zero = (p.L1 == 0.0 && p.L2 == 0.0 && p.L3 == 0.0);
    P.Liso = (float)(all_zero ? p.kappa : p.L1);
    P.L2 = (float)p.L2; P.L3 = (float)p.L3;
    P.Weff = (h->delta_eff > 0.0) ? (float)(p.W / h->delta_eff) : 0.0f;
    P.S_shell = (float)S_shell;
    P.mob_dt = (float)((1.0 / p.gamma) * dt);
    P.ci = (float)(0.5 * (p.Nx - 1.0)); P.cj = (float)(0.5 * (p.Ny - 1.0)); P.ck = (float)(0.5 * (p.Nz - 1.0));
    // Surface normal ~ (x/rx^2, y/ry^2, z/rz^2) with x = X dx: scale per axis dx/rx^2 (normalised later),
    // expressed relative to the x axis to stay in FP32 range.
    const double sxn = p.dx / (h->g.rx * h->g.rx);
    P.gnx = 1.0f;
    P.gny = (float)((p.dy / (h->g.ry * h->g.ry)) / sxn);
    P.gnz = (float)((p.dz / (h->g.rz * h->g.rz)) / sxn);
    const double ix2 = 1.0 / (p.dx * p.dx), iy2 = 1.0 / (p.dy * p.dy), iz2 = 1.0 / (p.dz * p.dz);
    P.lap_c = (float)(-2.0 * (ix2 + iy2 + iz2));
    P.L2i2x = (float)(p.L2 / (2.0 * p.dx)); P.L2i2y = (float)(p.L2 / (2.0 * p.dy)); P.L2i2z = (float)(p.L2 / (2.0 * p.dz));
    const double i2[3] = {1.0 / (2.0 * p.dx), 1.0 / (2.0 * p.dy), 1.0 / (2.0 * p.dz)};
    const int ab[6][2] = {{0, 0}, {1, 1}, {2, 2}, {0, 1}, {0, 2}, {1, 2}};
    for (int m = 0; m < 6; ++m) P.l3m[m] = (float)(0.5 * p.L3 * i2[ab[m][0]] * i2[ab[m][1]]);
    for (int m = 0; m < 6; ++m) P.l2w[m] = (float)(p.L2 * i2[ab[m][0]] * i2[ab[m][1]]);
    const double Liso = all_zero ? p.kappa : p.L1;
    P.lx = (float)(Liso * ix2); P.ly = (float)(Liso * iy2); P.lz = (float)(Liso * iz2);
    P.l3s[0] = (float)(p.L3 * ix2); P.l3s[1] = (float)(p.L3 * iy2); P.l3s[2] = (float)(p.L3 * iz2);
    for (int m = 0; m < 3; ++m) P.l3c[m] = (float)(2.0 * p.L3 * i2[ab[3 + m][0]] * i2[ab[3 + m][1]]);
    for (int m = 0; m < 6; ++m) P.l3d[m] = (float)(p.L3 * i2[ab[m][0]] * i2[ab[m][1]]);
    return P;
}

int alloc_or_fail(void** ptr, size_t bytes) {
    cudaError_t e = cudaMalloc(ptr, bytes);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        set_error(std::string("cudaMalloc(") + std::to_string(bytes) + "): " + cudaGetErrorString(e));
        return LDG_ERR_NOMEM;
    }
    return LDG_OK;
}

template <bool L2, bool L3, bool N, bool R>
void launch_direct(const qsr_handle* h, const float* in, float* out, const QsrConst& P) {
    dim3 blk(32, 8, 1), grd((P.Nz + 31) / 32, (P.Ny + 7) / 8, P.Nx);
    k_step_direct<L2, L3, N, R><<<grd, blk, 0, h->stream>>>(in, out, h->flags, P);
}

template <bool R>
void dispatch_direct(const qsr_handle* h, const float* in, float* out, const QsrConst& P, bool L2, bool L3, bool N) {
    const int key = (L2 ? 1 : 0) | (L3 ? 2 : 0) | (N ? 4 : 0);
    switch (key) {
        case 0: launch_direct<false, false, false, R>(h, in, out, P); break;
        case 1: launch_direct<true, false, false, R>(h, in, out, P); break;
        case 2: launch_direct<false, true, false, R>(h, in, out, P); break;
        case 3: launch_direct<true, true, false, R>(h, in, out, P); break;
        case 4: launch_direct<false, false, true, R>(h, in, out, P); break;
        case 5: launch_direct<true, false, true, R>(h, in, out, P); break;
        case 6: launch_direct<false, true, true, R>(h, in, out, P); break;
        default: launch_direct<true, true, true, R>(h, in, out, P); break;
    }
}

int grid_blocks(long long n, int threads, int cap) {
    long long b = (n + threads - 1) / threads;
    return (int)std::max(1LL, std::min<long long>(b, cap));
}

// Kernel selection: 1 = tiled (default), 0 = direct. LDG_QSR_KERNEL=direct forces the direct path.
int kernel_choice() {
    const char* e = getenv("LDG_QSR_KERNEL");
    if (e && std::strcmp(e, "direct") == 0) return 0;
    return 1;
}

}  // namespace

namespace {

// Whether a slice metric was asked for on a slice of the grid.
bool observe_defects(const qsr_handle* h, const qsr_observe_args* a) {
    return a->want_defects && a->defects_z_slice >= 0 && a->defects_z_slice < h->p.Nz;
}
bool observe_xi(const qsr_handle* h, const qsr_observe_args* a) {
    return a->want_xi && a->xi_z_slice >= 0 && a->xi_z_slice < h->p.Nz;
}

// Enqueues the observables of the current field on stream `st`; the result goes to `out` (device).
int observe_enqueue(qsr_handle* h, const qsr_observe_args* a, cudaStream_t st, ObsPartial* out) {
    const qsr_params& p = h->p;
    ObsConst O{};
    O.P = make_const(h, a->T, a->S_shell, 1.0);
    O.i2x = 1.0 / (2.0 * p.dx); O.i2y = 1.0 / (2.0 * p.dy); O.i2z = 1.0 / (2.0 * p.dz);
    const double dT = a->T - p.T_star;
    if (p.bulk_modechoice == 1) { O.c2 = (3.0 * p.a * dT) / 2.0; O.c3 = (3.0 * p.b) / 2.0; O.c4 = (9.0 * p.c) / 8.0; }
    else { O.c2 = (3.0 * p.a * dT) / 2.0; O.c3 = (9.0 * p.b) / 2.0; O.c4 = (9.0 * p.c) / 4.0; }
    O.Liso = (p.L1 == 0.0 && p.L2 == 0.0 && p.L3 == 0.0) ? p.kappa : p.L1;
    O.L2 = p.L2; O.L3 = p.L3;
    O.dV = p.dx * p.dy * p.dz;
    O.Weff_half = (h->delta_eff > 0.0) ? 0.5 * (p.W / h->delta_eff) : 0.0;
    O.S_shell = a->S_shell;
    O.cx = 0.5 * (p.Nx - 1.0); O.cy = 0.5 * (p.Ny - 1.0); O.cz = 0.5 * (p.Nz - 1.0);
    // Surface normal ~ (X dx/rx^2, Y dy/ry^2, Z dz/rz^2) in cell units, scaled relative to x.
    const double sx = p.dx / (h->g.rx * h->g.rx);
    O.gx = 1.0;
    O.gy = (p.dy / (h->g.ry * h->g.ry)) / sx;
    O.gz = (p.dz / (h->g.rz * h->g.rz)) / sx;
    O.hx = p.dx; O.hy = p.dy; O.hz = p.dz;
    O.checker_k = std::min(std::max(a->defects_z_slice, 0), p.Nz - 1);
    const bool wd = observe_defects(h, a), wx = observe_xi(h, a);
    O.mode = (wd ? 1 : 0) | (wx ? 2 : 0);
    O.dk = a->defects_z_slice;
    O.xk = a->xi_z_slice;
    O.dthr = a->defects_S_threshold; O.dcut = a->defects_charge_cutoff; O.xthr = a->xi_S_threshold;
    const long long rows = (long long)p.Nx * p.Ny;
    O.volume_blocks = grid_blocks(rows, kObsWarps, kObsVolumeBlocks);
    const int slice = (wd || wx) ? grid_blocks(rows, kObsThreads, kObsSliceBlocks) : 0;
    ObsPartial* result = h->opart + kObsVolumeBlocks + kObsSliceBlocks;
    k_observe<<<O.volume_blocks + slice, kObsThreads, 0, st>>>(h->q[h->cur], h->flags, O, h->opart,
                                                               reinterpret_cast<unsigned*>(result + 1), out ? out : result);
    h->launches++;
    LDG_LAUNCHED("k_observe");
    return LDG_OK;
}

// Fills the observables from the reduced block results.
void observe_finish(const qsr_handle* h, const qsr_observe_args* a, const ObsPartial& R, qsr_observables* o) {
    const qsr_params& p = h->p;
    const double nan = std::numeric_limits<double>::quiet_NaN();
    std::memset(o, 0, sizeof(*o));
    o->bulk = R.v[kBulk]; o->elastic = R.v[kElastic]; o->anchoring = R.v[kAnch];
    o->total = o->bulk + o->elastic + o->anchoring;
    o->radiality_count = (long long)R.n[kRadN];
    o->radiality = R.n[kRadN] > 0 ? R.v[kRad] / (double)R.n[kRadN] : 0.0;
    o->core_count = (long long)R.n[kCoreN];
    o->avg_S = R.n[kCoreN] > 0 ? R.v[kSumS] / (double)R.n[kCoreN] : 0.0;
    o->max_S = R.v[kMaxS];
    o->checker_rel = nan;
    const double all = R.v[kEven] + R.v[kOdd];
    if (o->max_S >= 0.5 && R.n[kEvenN] > 10 && R.n[kOddN] > 10 && R.n[kEvenN] + R.n[kOddN] > 20 && all != 0.0)
        o->checker_rel = std::fabs(R.v[kEven] - R.v[kOdd]) / std::fabs(all);
    o->defect_count = (long long)R.n[kDefects];
    o->defect_plaquettes = (long long)R.n[kPlaq];
    o->defect_density = (observe_defects(h, a) && R.n[kPlaq] > 0) ? (double)R.n[kDefects] / (double)R.n[kPlaq] : nan;
    o->xi_edges = (long long)R.n[kEdges];
    o->xi_grad_proxy = nan;
    if (observe_xi(h, a) && R.n[kEdges] > 0) {
        const double ms = R.v[kXi] / (double)R.n[kEdges];
        const double inv = (ms > 0.0) ? (1.0 / std::sqrt(ms + 1e-30)) : (1.0 / std::sqrt(1e-30));
        o->xi_grad_proxy = std::min(inv, 0.5 * (double)std::min(p.Nx, p.Ny));
    }
    o->max_q_norm = R.v[kMaxQ];
    o->nonfinite_cells = (long long)R.n[kNonfinite];
}

}  // namespace

extern "C" {

int qsr_create(const qsr_params* params, qsr_handle** out) {
    clear_error();
    LDG_REQUIRE(params && out, LDG_ERR_ARG, "qsr_create: null argument");
    const qsr_params& p = *params;
    LDG_REQUIRE(p.Nx >= 3 && p.Ny >= 3 && p.Nz >= 3, LDG_ERR_ARG, "qsr_create: Nx, Ny, Nz must be >= 3");
    LDG_REQUIRE((long long)p.Nx * p.Ny * p.Nz < (1LL << 32), LDG_ERR_ARG, "qsr_create: grid exceeds 2^32 cells");
    LDG_REQUIRE(p.dx > 0 && p.dy > 0 && p.dz > 0, LDG_ERR_ARG, "qsr_create: spacings must be positive");
    LDG_REQUIRE(p.gamma > 0, LDG_ERR_ARG, "qsr_create: gamma must be positive");
    LDG_REQUIRE(p.bulk_modechoice == 1 || p.bulk_modechoice == 2, LDG_ERR_ARG, "qsr_create: bulk_modechoice must be 1 or 2");
    qsr_handle* h = new (std::nothrow) qsr_handle();
    LDG_REQUIRE(h, LDG_ERR_NOMEM, "qsr_create: host allocation failed");
    h->p = p;
    cudaGetDevice(&h->device);
    h->g = make_geometry(p);
    h->sj = (p.Nz + 7) & ~7;  // rows of whole 32-byte sectors
    h->si = (long long)p.Ny * h->sj;
    h->sc = (long long)p.Nx * h->si;
    h->ncells = (long long)p.Nx * p.Ny * p.Nz;

    // Classification in FP64 on the host (QSR.cu:2160-2187 and the device predicates).
    std::vector<uint8_t> fl((size_t)h->sc, 0);
    const Geometry g = h->g;
    const double band = (p.W > 0.0) ? g.shell_half : 0.0;
    long long shell = 0;
#pragma omp parallel for collapse(2) reduction(+ : shell)
    for (int i = 0; i < p.Nx; ++i)
        for (int j = 0; j < p.Ny; ++j)
            for (int k = 0; k < p.Nz; ++k) {
                double sd, r;
                signed_distance(g, i, j, k, sd, r);
                uint8_t f = 0;
                if (std::fabs(sd) <= g.shell_half) { f |= kShell; ++shell; }
                if (sd <= 0.0) f |= kInside;
                if (sd < -2.0 * g.min_spacing) f |= kCore;
                if (sd <= 0.0 && r > 2.0 * g.min_spacing) f |= kRadial;
                fl[(size_t)i * h->si + (size_t)j * h->sj + k] = f;
                (void)band;
            }
    // delta_eff = shell volume / Knud-Thomsen ellipsoid area (QSR.cu:164-185).
    double delta = 2.0 * g.shell_half;
    if (shell > 0) {
        const double pp = 1.6075;
        const double ap = std::pow(g.rx, pp), bp = std::pow(g.ry, pp), cp = std::pow(g.rz, pp);
        const double mean = (ap * bp + ap * cp + bp * cp) / 3.0;
        const double area = (mean > 0.0) ? 4.0 * kPi * std::pow(mean, 1.0 / pp) : std::numeric_limits<double>::quiet_NaN();
        if (area > 0.0) {
            const double t = (double)shell * g.dx * g.dy * g.dz / area;
            if (std::isfinite(t) && t > 0.0) delta = t;
        }
    }
    h->delta_eff = delta;
    h->shell_cells = shell;
    long long evolving = 0;
#pragma omp parallel for collapse(2) reduction(+ : evolving)
    for (int i = 0; i < p.Nx; ++i)
        for (int j = 0; j < p.Ny; ++j)
            for (int k = 0; k < p.Nz; ++k) {
                double sd, r;
                signed_distance(g, i, j, k, sd, r);
                uint8_t& f = fl[(size_t)i * h->si + (size_t)j * h->sj + k];
                const bool sh = (f & kShell) != 0;
                const bool moves = !(p.W == 0.0 && sh) && (sd <= band);
                if (moves) { f |= kMove; ++evolving; }
                if (p.W <= 0.0 && sh) f |= kFixed;
                if (sh && p.W != 0.0 && delta > 0.0) f |= kAnchor;
            }
    h->evolving_cells = evolving;

    int rc;
    const size_t fbytes = (size_t)h->sc * 5 * sizeof(float);
    if ((rc = alloc_or_fail((void**)&h->q[0], fbytes)) || (rc = alloc_or_fail((void**)&h->q[1], fbytes)) ||
        (rc = alloc_or_fail((void**)&h->flags, (size_t)h->sc)) ||
        (rc = alloc_or_fail((void**)&h->opart, kObsBytes)) ||
        (p.compensated && ((rc = alloc_or_fail((void**)&h->lo[0], fbytes)) ||
                           (rc = alloc_or_fail((void**)&h->lo[1], fbytes))))) {
        qsr_destroy(h);
        return rc;
    }
    cudaError_t e = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking);
    // On the handle's stream, as all later work: it is non-blocking, so nothing would order a default-stream
    // operation before that work, and a late one would clear what has been written since.
    if (e == cudaSuccess) e = cudaMemcpyAsync(h->flags, fl.data(), (size_t)h->sc, cudaMemcpyHostToDevice, h->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(h->opart, 0, kObsBytes, h->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(h->q[0], 0, fbytes, h->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(h->q[1], 0, fbytes, h->stream);
    if (e == cudaSuccess && h->lo[0]) e = cudaMemsetAsync(h->lo[0], 0, fbytes, h->stream);
    if (e == cudaSuccess && h->lo[1]) e = cudaMemsetAsync(h->lo[1], 0, fbytes, h->stream);
    if (e != cudaSuccess) {
        set_error(std::string("qsr_create: ") + cudaGetErrorString(e));
        qsr_destroy(h);
        return LDG_ERR_CUDA;
    }
    rc = tiled_plan_build(h->tiled, p.Nx, p.Ny, p.Nz, h->sj, h->si, fl.data(), h->flags, h->q[0], h->q[1],
                          h->sc, p.L2 != 0.0, p.L3 != 0.0, h->stream);
    // an ensemble works on its droplets from a stream of its own
    if (rc == LDG_OK && cudaStreamSynchronize(h->stream) != cudaSuccess) {
        set_error("qsr_create: clearing the fields failed");
        rc = LDG_ERR_CUDA;
    }
    if (rc != LDG_OK) {
        qsr_destroy(h);
        return rc;
    }
    h->active_cells = h->tiled.active_cells;
    h->written_cells = h->tiled.written_cells;
    *out = h;
    return LDG_OK;
}

int qsr_geometry(const qsr_handle* h, qsr_geometry_info* o) {
    clear_error();
    LDG_REQUIRE(h && o, LDG_ERR_ARG, "qsr_geometry: null argument");
    o->center_x = h->g.cx; o->center_y = h->g.cy; o->center_z = h->g.cz;
    o->radius_x = h->g.rx; o->radius_y = h->g.ry; o->radius_z = h->g.rz;
    o->min_spacing = h->g.min_spacing;
    o->shell_half_thickness = h->g.shell_half;
    o->delta_eff = h->delta_eff;
    o->shell_cells = h->shell_cells;
    o->evolving_cells = h->evolving_cells;
    o->active_cells = h->tiled.ok ? h->tiled.active_cells : h->active_cells;
    o->written_cells = h->written_cells;
    o->box_cells = h->ncells;
    return LDG_OK;
}

int qsr_initial_field(const qsr_handle* h, int mode, long long seed, double S0, double noise_amplitude,
                      double* q) {
    clear_error();
    LDG_REQUIRE(h && q, LDG_ERR_ARG, "qsr_initial_field: null argument");
    LDG_REQUIRE(mode >= 0 && mode <= 2, LDG_ERR_ARG, "qsr_initial_field: init_mode must be 0, 1 or 2");
    const qsr_params& p = h->p;
    const Geometry& g = h->g;
    const size_t n = (size_t)h->ncells;
    std::fill(q, q + 5 * n, 0.0);
    std::mt19937 gen = (seed >= 0) ? std::mt19937((std::mt19937::result_type)seed) : std::mt19937(std::random_device{}());
    auto id = [&](int i, int j, int k) { return (size_t)k + (size_t)p.Nz * ((size_t)j + (size_t)p.Ny * (size_t)i); };
    if (mode == 2) {
        if (noise_amplitude <= 0.0) return LDG_OK;
        std::normal_distribution<double> dist(0.0, noise_amplitude);
        for (int i = 0; i < p.Nx; ++i)
            for (int j = 0; j < p.Ny; ++j)
                for (int k = 0; k < p.Nz; ++k) {
                    double sd, r;
                    signed_distance(g, i, j, k, sd, r);
                    if (sd <= 0.0)
                        for (int m = 0; m < 5; ++m) q[5 * id(i, j, k) + m] = dist(gen);
                }
        return LDG_OK;
    }
    std::uniform_real_distribution<double> dist_theta(0.0, kPi);
    std::uniform_real_distribution<double> dist_phi(0.0, 2.0 * kPi);
    for (int i = 0; i < p.Nx; ++i)
        for (int j = 0; j < p.Ny; ++j)
            for (int k = 0; k < p.Nz; ++k) {
                double sd, r;
                signed_distance(g, i, j, k, sd, r);
                if (!(sd <= 0.0)) continue;
                double S = S0;
                if (r < g.core_radius) S *= (r / g.core_radius);
                double nx = 1.0, ny = 0.0, nz = 0.0;
                if (mode == 0) {
                    const double theta = dist_theta(gen);
                    const double phi = dist_phi(gen);
                    nx = std::sin(theta) * std::cos(phi);
                    ny = std::sin(theta) * std::sin(phi);
                    nz = std::cos(theta);
                } else if (r > 1e-30) {
                    nx = (i * g.dx - g.cx) / r;
                    ny = (j * g.dy - g.cy) / r;
                    nz = (k * g.dz - g.cz) / r;
                }
                double* c = q + 5 * id(i, j, k);
                c[0] = S * (nx * nx - 1.0 / 3.0);
                c[1] = S * (nx * ny);
                c[2] = S * (nx * nz);
                c[3] = S * (ny * ny - 1.0 / 3.0);
                c[4] = S * (ny * nz);
            }
    return LDG_OK;
}

static int ensure_stage(qsr_handle* h, size_t doubles) {
    if (h->stage) return LDG_OK;
    (void)doubles;
    return alloc_or_fail((void**)&h->stage, (size_t)h->ncells * 5 * sizeof(double));
}

int qsr_upload(qsr_handle* h, const double* q) {
    clear_error();
    LDG_REQUIRE(h && q, LDG_ERR_ARG, "qsr_upload: null argument");
    DeviceGuard device_guard(h->device);
    int rc = ensure_stage(h, 5);
    if (rc) return rc;
    LDG_CUDA(cudaMemcpyAsync(h->stage, q, (size_t)h->ncells * 5 * sizeof(double), cudaMemcpyHostToDevice, h->stream));
    h->cur = 0;
    k_aos_to_soa<<<grid_blocks(h->ncells, 256, 148 * 16), 256, 0, h->stream>>>(h->stage, h->q[0], h->q[1], h->p.Nx,
                                                                              h->p.Ny, h->p.Nz, h->sj, h->si, h->sc,
                                                                              h->lo[0], h->lo[1]);
    h->launches++;
    LDG_LAUNCHED("k_aos_to_soa");
    LDG_CUDA(cudaStreamSynchronize(h->stream));
    h->uploaded = true;
    return LDG_OK;
}

int qsr_download(qsr_handle* h, double* q) {
    clear_error();
    LDG_REQUIRE(h && q, LDG_ERR_ARG, "qsr_download: null argument");
    DeviceGuard device_guard(h->device);
    int rc = ensure_stage(h, 5);
    if (rc) return rc;
    k_soa_to_aos<<<grid_blocks(h->ncells, 256, 148 * 16), 256, 0, h->stream>>>(h->q[h->cur], h->stage, h->p.Nx,
                                                                              h->p.Ny, h->p.Nz, h->sj, h->si, h->sc,
                                                                              h->lo[h->cur]);
    h->launches++;
    LDG_LAUNCHED("k_soa_to_aos");
    LDG_CUDA(cudaMemcpyAsync(q, h->stage, (size_t)h->ncells * 5 * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    LDG_CUDA(cudaStreamSynchronize(h->stream));
    return tiled_check(h->tiled, h->stream);
}

int qsr_nematic(qsr_handle* h, double* s_n) {
    clear_error();
    LDG_REQUIRE(h && s_n, LDG_ERR_ARG, "qsr_nematic: null argument");
    DeviceGuard device_guard(h->device);
    int rc = ensure_stage(h, 5);
    if (rc) return rc;
    k_nematic_out<<<grid_blocks(h->ncells, 256, 148 * 16), 256, 0, h->stream>>>(h->q[h->cur], h->stage, h->p.Nx,
                                                                               h->p.Ny, h->p.Nz, h->sj, h->si, h->sc);
    h->launches++;
    LDG_LAUNCHED("k_nematic_out");
    LDG_CUDA(cudaMemcpyAsync(s_n, h->stage, (size_t)h->ncells * 4 * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    LDG_CUDA(cudaStreamSynchronize(h->stream));
    return LDG_OK;
}

int qsr_step(qsr_handle* h, int n_steps, const qsr_step_args* a) {
    clear_error();
    LDG_REQUIRE(h && a, LDG_ERR_ARG, "qsr_step: null argument");
    DeviceGuard device_guard(h->device);
    LDG_REQUIRE(n_steps >= 0, LDG_ERR_ARG, "qsr_step: n_steps must be >= 0");
    LDG_REQUIRE(h->uploaded, LDG_ERR_STATE, "qsr_step: no field uploaded");
    LDG_REQUIRE(a->dt > 0.0 && std::isfinite(a->dt), LDG_ERR_ARG, "qsr_step: dt must be positive and finite");
    const qsr_params& p = h->p;
    QsrConst P = make_const(h, a->T, a->S_shell, a->dt);
    P.qcap = (float)a->q_norm_cap;
    P.sigma = (float)a->noise_sigma;
    P.key0 = (uint32_t)a->seed;
    P.key1 = (uint32_t)(a->seed >> 32);
    P.instance = 0;
    const bool noise = a->noise_sigma > 0.0;
    const bool L2 = p.L2 != 0.0, L3 = p.L3 != 0.0;
    // The reference falls back to the explicit update when the stabiliser is inactive (QSR.cu:2721).
    const bool imex = a->semi_implicit && a->L_stab > 0.0 && a->jacobi_iters > 0;
    if (imex) {
        if (!h->sweep.ok) {
            // all of it or nothing: the next call starts again where this one fails
            const size_t bytes = (size_t)h->sc * 5 * sizeof(float);
            float* rhs = nullptr;
            int rc = alloc_or_fail((void**)&rhs, bytes);
            if (rc) return rc;
            if (cudaMemsetAsync(rhs, 0, bytes, h->stream) != cudaSuccess) {
                set_error("qsr_step: clearing the right-hand side failed");
                rc = LDG_ERR_CUDA;
            }
            if (rc == LDG_OK) rc = tiled_encode(&h->rhs_map, rhs, p.Nx, p.Ny, p.Nz, h->sj, h->si, h->sc, false, false);
            if (rc == LDG_OK) rc = tiled_sweep_plan(h->tiled, h->sc, h->sweep, h->stream);
            if (rc) {
                cudaFree(rhs);
                return rc;
            }
            h->rhs = rhs;
        }
        P.alpha = (float)(a->dt * (1.0 / p.gamma) * a->L_stab);
        const double aj = (a->dt / p.gamma) * a->L_stab;  // QSR.cu:2728
        const double denom = 1.0 + 2.0 * aj * (1.0 / (p.dx * p.dx) + 1.0 / (p.dy * p.dy) + 1.0 / (p.dz * p.dz));
        LDG_REQUIRE(denom > 0.0, LDG_ERR_ARG, "qsr_step: non-positive Jacobi denominator");
        P.jdenom_inv = (float)(1.0 / denom);
    }
    const int choice = kernel_choice();
    for (int s = 0; s < n_steps; ++s) {
        P.step = a->step_index + s;
        const float* in = h->q[h->cur];
        float* outb = h->q[1 - h->cur];
        if (!imex) {
            if (choice == 1 && h->tiled.ok) {
                int rc = tiled_step(h->tiled, in, outb, P, L2, L3, noise, false, h->stream, h->lo[h->cur],
                                    h->lo[1 - h->cur]);
                if (rc) return rc;
            } else {
                dispatch_direct<false>(h, in, outb, P, L2, L3, noise);
            }
            h->launches++;
            LDG_LAUNCHED("qsr step kernel");
            h->cur = 1 - h->cur;
        } else {
            if (choice == 1 && h->tiled.ok) {
                int rc = tiled_step(h->tiled, in, h->rhs, P, L2, L3, noise, true, h->stream);
                if (rc) return rc;
            } else {
                dispatch_direct<true>(h, in, h->rhs, P, L2, L3, noise);
            }
            h->launches++;
            LDG_LAUNCHED("k_step_direct(rhs)");
            dim3 blk(32, 8, 1), grd((p.Nz + 31) / 32, (p.Ny + 7) / 8, p.Nx);
            const bool tiled = choice == 1 && h->tiled.ok;
            int c = h->cur;
            for (int it = 0; it < a->jacobi_iters; ++it) {
                const bool last = (it == a->jacobi_iters - 1);
                if (tiled) {
                    int rc = tiled_sweep(h->sweep, h->q[c], h->q[1 - c], h->rhs_map, P, last, h->stream);
                    if (rc) return rc;
                } else if (last) {
                    k_jacobi<true><<<grd, blk, 0, h->stream>>>(h->rhs, h->q[c], h->q[1 - c], h->flags, P);
                } else {
                    k_jacobi<false><<<grd, blk, 0, h->stream>>>(h->rhs, h->q[c], h->q[1 - c], h->flags, P);
                }
                h->launches++;
                LDG_LAUNCHED("k_jacobi");
                c = 1 - c;
            }
            h->cur = c;
        }
    }
    // Compensated storage is kept by the explicit tiled step only; after other updates the
    // field is its high words.
    if (h->lo[0] && n_steps > 0 && (imex || choice != 1 || !h->tiled.ok)) {
        const size_t fbytes = (size_t)h->sc * 5 * sizeof(float);
        LDG_CUDA(cudaMemsetAsync(h->lo[0], 0, fbytes, h->stream));
        LDG_CUDA(cudaMemsetAsync(h->lo[1], 0, fbytes, h->stream));
    }
    return LDG_OK;
}

int qsr_observe(qsr_handle* h, const qsr_observe_args* a, qsr_observables* o) {
    clear_error();
    LDG_REQUIRE(h && a && o, LDG_ERR_ARG, "qsr_observe: null argument");
    DeviceGuard device_guard(h->device);
    ObsPartial R{};
    int rc = observe_enqueue(h, a, h->stream, nullptr);
    if (rc) return rc;
    LDG_CUDA(cudaMemcpyAsync(&R, h->opart + kObsVolumeBlocks + kObsSliceBlocks, sizeof(R), cudaMemcpyDeviceToHost,
                             h->stream));
    if ((rc = tiled_check(h->tiled, h->stream))) return rc;
    observe_finish(h, a, R, o);
    return LDG_OK;
}

int qsr_autotune(qsr_handle* h, const qsr_step_args* a, int trial_steps, int* chosen_chunk) {
    clear_error();
    LDG_REQUIRE(h && a, LDG_ERR_ARG, "qsr_autotune: null argument");
    DeviceGuard device_guard(h->device);
    LDG_REQUIRE(trial_steps >= 1, LDG_ERR_ARG, "qsr_autotune: trial_steps must be >= 1");
    LDG_REQUIRE(h->uploaded, LDG_ERR_STATE, "qsr_autotune: no field uploaded");
    LDG_REQUIRE(h->tiled.ok, LDG_ERR_STATE, "qsr_autotune: no tiled plan");
    LDG_CUDA(cudaStreamSynchronize(h->stream));
    // Back up the current field (and its low words) and the launch count; restore both after.
    const size_t fbytes = (size_t)h->sc * 5 * sizeof(float);
    const int planes = h->lo[0] ? 2 : 1;
    float* backup = nullptr;
    int rc = alloc_or_fail((void**)&backup, fbytes * planes);
    if (rc) return rc;
    const int cur0 = h->cur;
    const long long launches0 = h->launches;
    LDG_CUDA(cudaMemcpyAsync(backup, h->q[cur0], fbytes, cudaMemcpyDeviceToDevice, h->stream));
    if (h->lo[0]) LDG_CUDA(cudaMemcpyAsync(backup + h->sc * 5, h->lo[cur0], fbytes, cudaMemcpyDeviceToDevice, h->stream));
    const int candidates[] = {8, 12, 16, 24, 32, 48, 64};
    int best = candidates[0];
    std::vector<int> tried;  // lengths in use: on a short list several candidates are cut to the same one
    float best_ms = std::numeric_limits<float>::infinity();
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess) {
        set_error("qsr_autotune: event creation failed");
        rc = LDG_ERR_CUDA;
    }
    qsr_step_args t = *a;
    for (int c : candidates) {
        if (rc) break;
        if ((rc = tiled_plan_rechunk(h->tiled, ItemLength{c, false}, h->stream))) break;
        if (std::find(tried.begin(), tried.end(), h->tiled.chunk) != tried.end()) continue;
        tried.push_back(h->tiled.chunk);
        if ((rc = qsr_step(h, 2, &t))) break;
        cudaEventRecord(e0, h->stream);
        if ((rc = qsr_step(h, trial_steps, &t))) break;
        cudaEventRecord(e1, h->stream);
        if (cudaEventSynchronize(e1) != cudaSuccess) {
            set_error("qsr_autotune: trial failed");
            rc = LDG_ERR_CUDA;
            break;
        }
        float ms = 0.0f;
        cudaEventElapsedTime(&ms, e0, e1);
        if (ms < best_ms) { best_ms = ms; best = c; }
    }
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    // restore both ping-pong buffers from the backup (frozen cells are identical in both)
    for (int b = 0; b < 2; ++b) {
        cudaMemcpyAsync(h->q[b], backup, fbytes, cudaMemcpyDeviceToDevice, h->stream);
        if (h->lo[0]) cudaMemcpyAsync(h->lo[b], backup + h->sc * 5, fbytes, cudaMemcpyDeviceToDevice, h->stream);
    }
    cudaStreamSynchronize(h->stream);
    cudaFree(backup);
    h->cur = cur0;
    h->launches = launches0;
    if (rc == LDG_OK) rc = tiled_check(h->tiled, h->stream);
    if (rc) return rc;
    if ((rc = tiled_plan_rechunk(h->tiled, ItemLength{best, false}, h->stream))) return rc;
    if (chosen_chunk) *chosen_chunk = best;
    return LDG_OK;
}

int qsr_sync(qsr_handle* h) {
    clear_error();
    LDG_REQUIRE(h, LDG_ERR_ARG, "qsr_sync: null handle");
    DeviceGuard device_guard(h->device);
    LDG_CUDA(cudaStreamSynchronize(h->stream));
    return tiled_check(h->tiled, h->stream);
}

void* qsr_stream(qsr_handle* h) { return h ? (void*)h->stream : nullptr; }

long long qsr_launch_count(const qsr_handle* h) { return h ? h->launches : 0; }

int qsr_destroy(qsr_handle* h) {
    if (!h) return LDG_OK;
    DeviceGuard device_guard(h->device);
    if (h->stream) cudaStreamSynchronize(h->stream);
    cudaFree(h->q[0]); cudaFree(h->q[1]); cudaFree(h->lo[0]); cudaFree(h->lo[1]); cudaFree(h->rhs); cudaFree(h->flags);
    if (!h->stage_shared) cudaFree(h->stage);
    cudaFree(h->opart);
    tiled_sweep_free(h->sweep);
    tiled_plan_free(h->tiled);
    if (h->stream) cudaStreamDestroy(h->stream);
    delete h;
    return LDG_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------------------
// Ensemble of droplets: every instance is a qsr_handle (geometry, classification, buffers,
// tensor maps, observables); one persistent work-stealing launch per step covers the active
// tiles of all instances, and runs of steps are replayed from a captured CUDA graph.
// ---------------------------------------------------------------------------------------
struct ens_handle {
    ens_params p{};
    int device = -1;                       // the GPU the ensemble was created on
    double* stage = nullptr;               // host-boundary staging shared by all droplets
    ObsPartial* d_obs = nullptr;           // results of ens_observe_all, one per droplet
    std::vector<qsr_handle*> inst;
    std::vector<ens_instance> desc;
    std::vector<tiled::EnsInstDev> host_inst;
    CUtensorMap* d_tms = nullptr;          // 2 per instance: input buffer q[0] / q[1]
    tiled::EnsInstDev* d_inst = nullptr;
    tiled::TileItem* d_items = nullptr;
    tiled::RowMask* d_masks = nullptr;
    int n_items = 0;
    tiled::EnsCtl* d_ctl = nullptr;
    int* d_err = nullptr;
    int chunk = 0;
    int grid = 0;
    size_t smem = 0;
    bool L2 = false, L3 = false, noise = false;
    long long step = 0;
    long long cells = 0, active = 0, written = 0;
    cudaStream_t stream = nullptr;
    cudaGraphExec_t graph = nullptr;
    int graph_steps = 0;
    long long launches = 0;
};

namespace {

constexpr int kEnsGraphSteps = 32;

using EnsKernel = void (*)(const CUtensorMap*, const tiled::EnsInstDev*, const tiled::TileItem*,
                           const tiled::RowMask*, int, tiled::EnsCtl*, int*);

EnsKernel ens_kernel(bool L2, bool L3, bool N) {
    using namespace tiled;
    const int key = (L2 ? 1 : 0) | (L3 ? 2 : 0) | (N ? 4 : 0);
    switch (key) {
        case 0: return k_step_ensemble<false, false, false>;
        case 1: return k_step_ensemble<true, false, false>;
        case 2: return k_step_ensemble<false, true, false>;
        case 3: return k_step_ensemble<true, true, false>;
        case 4: return k_step_ensemble<false, false, true>;
        case 5: return k_step_ensemble<true, false, true>;
        case 6: return k_step_ensemble<false, true, true>;
        default: return k_step_ensemble<true, true, true>;
    }
}

void ens_drop_graph(ens_handle* h) {
    if (h->graph) cudaGraphExecDestroy(h->graph);
    h->graph = nullptr;
    h->graph_steps = 0;
}

// Work list of all instances for items of that length (instance-major, so CTAs that run together share halo
// planes of one droplet in L2), and the persistent grid size. On failure the ensemble is as before.
int ens_rechunk(ens_handle* h, ItemLength len) {
    std::vector<const TiledPlan*> plans;
    for (const qsr_handle* q : h->inst) plans.push_back(&q->tiled);
    const int chunk = len.exact ? len.planes
                                : tiled_length(plans, len.planes, (h->L2 || h->L3) ? kLoadDeep : kLoadL1, h->L2);
    std::vector<tiled::TileItem> items;
    std::vector<int> first;   // first item of every instance
    long long active = 0;
    int recs = 0;
    for (size_t n = 0; n < h->inst.size(); ++n) {
        long long a = 0;
        int nr = 0;
        first.push_back((int)items.size());
        tiled_device_items(tiled_items(h->inst[n]->tiled, chunk, h->L2, &a), (int)n, recs, items, &nr);
        recs += nr;
        active += a;
    }
    first.push_back((int)items.size());
    const EnsKernel k = ens_kernel(h->L2, h->L3, h->noise);
    LDG_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)h->smem));
    int dev = 0, sms = 0, per_sm = 0;
    LDG_CUDA(cudaGetDevice(&dev));
    LDG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    LDG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, tiled::THREADS, h->smem));
    LDG_REQUIRE(per_sm > 0, LDG_ERR_CUDA, "ensemble: step kernel does not fit on an SM");
    DeviceList now;
    const int rc = tiled_list_make(items, recs, h->stream, now, [&](const DeviceList& d) -> int {
        for (size_t n = 0; n < h->inst.size(); ++n)
            if (int e = tiled_masks(h->inst[n]->tiled, d.items + first[n], first[n + 1] - first[n], h->L2, d.masks,
                                    h->stream))
                return e;
        return LDG_OK;
    });
    if (rc) return rc;
    ens_drop_graph(h);  // it launches the old list
    DeviceList old{h->d_items, h->d_masks};
    tiled_list_free(old);
    h->d_items = now.items;
    h->d_masks = now.masks;
    h->n_items = (int)items.size();
    h->active = active;
    h->chunk = chunk;
    h->grid = std::max(1, std::min(sms * per_sm, h->n_items));
    return LDG_OK;
}

int ens_launch(ens_handle* h) {
    const EnsKernel k = ens_kernel(h->L2, h->L3, h->noise);
    LDG_CUDA(launch_pdl(k, dim3((unsigned)h->grid), tiled::THREADS, h->smem, h->stream, h->d_tms, h->d_inst, h->d_items, h->d_masks,
                        h->n_items, h->d_ctl, h->d_err));
    return LDG_OK;
}

// Captures kEnsGraphSteps launches of the step kernel into a CUDA graph and uploads it, so the
// first ens_step that replays it pays no instantiation cost. Capturing runs no kernel.
int ens_build_graph(ens_handle* h) {
    ens_drop_graph(h);
    if (h->n_items == 0) return LDG_OK;
    cudaGraph_t g = nullptr;
    LDG_CUDA(cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal));
    int rc = LDG_OK;
    for (int s = 0; s < kEnsGraphSteps && rc == LDG_OK; ++s) rc = ens_launch(h);
    cudaError_t e = cudaStreamEndCapture(h->stream, &g);
    if (rc) {
        if (g) cudaGraphDestroy(g);
        return rc;
    }
    if (e == cudaSuccess) e = cudaGraphInstantiate(&h->graph, g, 0);
    if (g) cudaGraphDestroy(g);
    if (e == cudaSuccess) e = cudaGraphUpload(h->graph, h->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
    if (e != cudaSuccess) {
        ens_drop_graph(h);
        set_error(std::string("ensemble: graph capture failed: ") + cudaGetErrorString(e));
        return LDG_ERR_CUDA;
    }
    h->graph_steps = kEnsGraphSteps;
    return LDG_OK;
}

// Reads and clears the ensemble's device error word.
int ens_check(ens_handle* h) {
    int e = 0;
    LDG_CUDA(cudaMemcpyAsync(&e, h->d_err, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
    LDG_CUDA(cudaStreamSynchronize(h->stream));
    if (e != 0) {
        LDG_CUDA(cudaMemsetAsync(h->d_err, 0, sizeof(int), h->stream));
        LDG_CUDA(cudaStreamSynchronize(h->stream));
        set_error("ensemble step: a bounded shared-memory pipeline wait gave up");
        return LDG_ERR_TIMEOUT;
    }
    return LDG_OK;
}

// Makes every instance's current buffer the input of the ensemble's next step.
void ens_sync_cur(ens_handle* h) {
    for (qsr_handle* q : h->inst) q->cur = (int)(h->step & 1);
}

// Observables of a droplet at the ensemble's current step: its protocol temperature, its shell
// order, slices Nz/2, thresholds 0.1 / 0.25.
qsr_observe_args ens_default_observe_args(const ens_handle* h, int instance) {
    qsr_observe_args a{};
    const tiled::EnsInstDev& D = h->host_inst[instance];
    a.T = tiled::ens_temperature(D, h->step);
    const double A = D.a3 * (a.T - D.T_star);
    a.S_shell = D.custom_shell ? D.S_custom : std::max(0.0, tiled::ens_S_eq(A, D.B, D.C));
    const int Nz = h->inst[instance]->p.Nz;
    a.defects_z_slice = Nz / 2;
    a.xi_z_slice = Nz / 2;
    a.defects_S_threshold = 0.1;
    a.defects_charge_cutoff = 0.25;
    a.xi_S_threshold = 0.1;
    a.want_defects = 1;
    a.want_xi = 1;
    return a;
}

int ens_set_step(ens_handle* h, long long step) {
    tiled::EnsCtl c{0, 0u, step};
    LDG_CUDA(cudaMemcpyAsync(h->d_ctl, &c, sizeof(c), cudaMemcpyHostToDevice, h->stream));
    LDG_CUDA(cudaStreamSynchronize(h->stream));
    h->step = step;
    ens_sync_cur(h);
    return LDG_OK;
}

}  // namespace

extern "C" {

int ens_destroy(ens_handle* h);

int ens_create(const ens_params* params, int n_instances, const ens_instance* instances, ens_handle** out) {
    clear_error();
    LDG_REQUIRE(params && instances && out, LDG_ERR_ARG, "ens_create: null argument");
    LDG_REQUIRE(n_instances >= 1, LDG_ERR_ARG, "ens_create: need at least one instance");
    const ens_params& p = *params;
    LDG_REQUIRE(p.dt > 0.0 && std::isfinite(p.dt), LDG_ERR_ARG, "ens_create: dt must be positive and finite");
    LDG_REQUIRE(p.protocol == 1 || p.protocol == 2, LDG_ERR_ARG, "ens_create: protocol must be 1 (step) or 2 (ramp)");
    for (int n = 0; n < n_instances; ++n) {
        LDG_REQUIRE(instances[n].N >= 3 && (instances[n].Ny == 0 || instances[n].Ny >= 3) &&
                        (instances[n].Nz == 0 || instances[n].Nz >= 3),
                    LDG_ERR_ARG, "ens_create: instance grid extents must be >= 3");
        LDG_REQUIRE(instances[n].pre_equil_iters >= 0 && instances[n].ramp_iters >= 0, LDG_ERR_ARG,
                    "ens_create: negative protocol length");
        LDG_REQUIRE(instances[n].noise_sigma >= 0.0, LDG_ERR_ARG, "ens_create: negative noise amplitude");
    }
    ens_handle* h = new (std::nothrow) ens_handle();
    LDG_REQUIRE(h, LDG_ERR_NOMEM, "ens_create: host allocation failed");
    h->p = p;
    cudaGetDevice(&h->device);
    h->desc.assign(instances, instances + n_instances);
    h->L2 = p.L2 != 0.0;
    h->L3 = p.L3 != 0.0;
    for (int n = 0; n < n_instances; ++n) {
        const ens_instance& d = instances[n];
        h->noise = h->noise || d.noise_sigma > 0.0;
        if (d.own_material) {
            h->L2 = h->L2 || d.L2 != 0.0;
            h->L3 = h->L3 || d.L3 != 0.0;
        }
    }
    int rc = LDG_OK;
    for (int n = 0; n < n_instances && rc == LDG_OK; ++n) {
        const ens_instance& d = instances[n];
        qsr_params q{};
        q.Nx = d.N;
        q.Ny = d.Ny > 0 ? d.Ny : d.N;
        q.Nz = d.Nz > 0 ? d.Nz : d.N;
        q.dx = p.dx; q.dy = p.dy; q.dz = p.dz;
        q.a = p.a; q.b = p.b; q.c = p.c; q.T_star = p.T_star; q.bulk_modechoice = p.bulk_modechoice;
        q.kappa = p.kappa; q.L1 = p.L1; q.L2 = p.L2; q.L3 = p.L3; q.W = p.W; q.gamma = p.gamma;
        q.droplet_radius_cells = d.droplet_radius_cells;
        if (d.own_material) {
            q.W = d.W; q.L2 = d.L2; q.L3 = d.L3;
        }
        qsr_handle* qh = nullptr;
        rc = qsr_create(&q, &qh);
        if (rc == LDG_OK) h->inst.push_back(qh);
    }
    if (rc != LDG_OK) {
        const std::string msg = ldg_last_error();
        ens_destroy(h);
        set_error(msg);
        return rc;
    }
    // One FP64 staging buffer for the host boundary of every droplet (calls are sequential and
    // each synchronises before returning), allocated here rather than on first use.
    {
        long long maxc = 0;
        for (qsr_handle* q : h->inst) maxc = std::max(maxc, q->ncells);
        rc = alloc_or_fail((void**)&h->stage, (size_t)maxc * 5 * sizeof(double));
        if (rc) {
            ens_destroy(h);
            return rc;
        }
        for (qsr_handle* q : h->inst) {
            q->stage = h->stage;
            q->stage_shared = true;
        }
    }
    // Per-instance descriptors: the static step constants plus the protocol.
    const double a3 = 3.0 * p.a;
    const double B = (p.bulk_modechoice == 1) ? (9.0 * p.b) / 2.0 : (27.0 * p.b) / 2.0;
    const double Cc = (p.bulk_modechoice == 1) ? (9.0 * p.c) / 2.0 : 9.0 * p.c;
    std::vector<CUtensorMap> tms(2 * (size_t)n_instances);
    h->host_inst.resize(n_instances);
    for (int n = 0; n < n_instances; ++n) {
        qsr_handle* qh = h->inst[n];
        const ens_instance& d = instances[n];
        tiled::EnsInstDev& D = h->host_inst[n];
        D.P = make_const(qh, d.T_high, 0.0, p.dt);
        D.P.qcap = (float)p.q_norm_cap;
        D.P.sigma = (float)d.noise_sigma;
        D.P.key0 = (uint32_t)d.seed;
        D.P.key1 = (uint32_t)(d.seed >> 32);
        D.P.instance = 0;
        D.q[0] = qh->q[0];
        D.q[1] = qh->q[1];
        D.T_high = d.T_high; D.T_low = d.T_low;
        D.pre = d.pre_equil_iters; D.ramp = d.ramp_iters;
        D.protocol = p.protocol;
        D.custom_shell = p.boundary_custom ? 1 : 0;
        D.S_custom = p.boundary_S;
        D.a3 = a3; D.T_star = p.T_star; D.B = B; D.C = Cc;
        // the ensemble's kernel reads every droplet with the same halo
        for (int b = 0; b < 2 && rc == LDG_OK; ++b)
            rc = tiled_encode(&tms[2 * n + b], qh->q[b], qh->p.Nx, qh->p.Ny, qh->p.Nz, qh->sj, qh->si, qh->sc, h->L2);
        h->cells += qh->ncells;
        h->active += qh->active_cells;
        h->written += qh->written_cells;
    }
    using namespace tiled;
    if (rc != LDG_OK) {
        const std::string msg = ldg_last_error();
        ens_destroy(h);
        set_error(msg);
        return rc;
    }
    h->smem = h->L2 ? tile_smem_bytes<true>() : tile_smem_bytes<false>();
    cudaError_t e = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking);
    if ((rc = alloc_or_fail((void**)&h->d_tms, tms.size() * sizeof(CUtensorMap))) ||
        (rc = alloc_or_fail((void**)&h->d_inst, h->host_inst.size() * sizeof(EnsInstDev))) ||
        (rc = alloc_or_fail((void**)&h->d_ctl, sizeof(EnsCtl))) || (rc = alloc_or_fail((void**)&h->d_err, sizeof(int))) ||
        e != cudaSuccess) {
        if (e != cudaSuccess) {
            set_error(std::string("ens_create: ") + cudaGetErrorString(e));
            rc = LDG_ERR_CUDA;
        }
        ens_destroy(h);
        return rc;
    }
    e = cudaMemcpyAsync(h->d_tms, tms.data(), tms.size() * sizeof(CUtensorMap), cudaMemcpyHostToDevice, h->stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(h->d_inst, h->host_inst.data(), h->host_inst.size() * sizeof(EnsInstDev),
                            cudaMemcpyHostToDevice, h->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(h->d_err, 0, sizeof(int), h->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
    if (e != cudaSuccess) {
        set_error(std::string("ens_create: ") + cudaGetErrorString(e));
        ens_destroy(h);
        return LDG_ERR_CUDA;
    }
    if ((rc = ens_rechunk(h, tiled_default_length())) || (rc = ens_set_step(h, 0)) || (rc = ens_build_graph(h))) {
        const std::string msg = ldg_last_error();
        ens_destroy(h);
        set_error(msg);
        return rc;
    }
    *out = h;
    return LDG_OK;
}

int ens_initial_fields(ens_handle* h, int init_mode, double S0, double noise_amplitude) {
    clear_error();
    LDG_REQUIRE(h, LDG_ERR_ARG, "ens_initial_fields: null handle");
    DeviceGuard device_guard(h->device);
    LDG_CUDA(cudaStreamSynchronize(h->stream));
    std::vector<double> buf;
    for (size_t n = 0; n < h->inst.size(); ++n) {
        qsr_handle* qh = h->inst[n];
        buf.resize((size_t)qh->ncells * 5);
        int rc = qsr_initial_field(qh, init_mode, (long long)h->desc[n].seed, S0, noise_amplitude, buf.data());
        if (rc == LDG_OK) rc = qsr_upload(qh, buf.data());
        if (rc) return rc;
    }
    ens_sync_cur(h);
    return LDG_OK;
}

int ens_upload(ens_handle* h, int instance, const double* q) {
    clear_error();
    LDG_REQUIRE(h && q, LDG_ERR_ARG, "ens_upload: null argument");
    DeviceGuard device_guard(h->device);
    LDG_REQUIRE(instance >= 0 && instance < (int)h->inst.size(), LDG_ERR_ARG, "ens_upload: instance out of range");
    LDG_CUDA(cudaStreamSynchronize(h->stream));
    // qsr_upload fills both ping-pong buffers, so either parity of the step index reads it.
    const int rc = qsr_upload(h->inst[instance], q);
    ens_sync_cur(h);
    return rc;
}

int ens_download(ens_handle* h, int instance, double* q) {
    clear_error();
    LDG_REQUIRE(h && q, LDG_ERR_ARG, "ens_download: null argument");
    DeviceGuard device_guard(h->device);
    LDG_REQUIRE(instance >= 0 && instance < (int)h->inst.size(), LDG_ERR_ARG, "ens_download: instance out of range");
    int rc = ens_check(h);
    if (rc) return rc;
    ens_sync_cur(h);
    return qsr_download(h->inst[instance], q);
}

int ens_nematic(ens_handle* h, int instance, double* s_n) {
    clear_error();
    LDG_REQUIRE(h && s_n, LDG_ERR_ARG, "ens_nematic: null argument");
    DeviceGuard device_guard(h->device);
    LDG_REQUIRE(instance >= 0 && instance < (int)h->inst.size(), LDG_ERR_ARG, "ens_nematic: instance out of range");
    int rc = ens_check(h);
    if (rc) return rc;
    ens_sync_cur(h);
    return qsr_nematic(h->inst[instance], s_n);
}

int ens_step(ens_handle* h, int n_steps) {
    clear_error();
    LDG_REQUIRE(h, LDG_ERR_ARG, "ens_step: null handle");
    DeviceGuard device_guard(h->device);
    LDG_REQUIRE(n_steps >= 0, LDG_ERR_ARG, "ens_step: n_steps must be >= 0");
    for (qsr_handle* q : h->inst) LDG_REQUIRE(q->uploaded, LDG_ERR_STATE, "ens_step: an instance has no field");
    if (h->n_items == 0) {
        h->step += n_steps;
        return ens_set_step(h, h->step);
    }
    int left = n_steps;
    while (left >= kEnsGraphSteps) {
        if (!h->graph) {
            const int rc = ens_build_graph(h);
            if (rc) return rc;
        }
        LDG_CUDA(cudaGraphLaunch(h->graph, h->stream));
        h->launches += h->graph_steps;
        left -= h->graph_steps;
    }
    for (int s = 0; s < left; ++s) {
        int rc = ens_launch(h);
        if (rc) return rc;
        h->launches++;
    }
    h->step += n_steps;
    ens_sync_cur(h);
    return LDG_OK;
}

int ens_observe(ens_handle* h, int instance, const qsr_observe_args* args, qsr_observables* out) {
    clear_error();
    LDG_REQUIRE(h && out, LDG_ERR_ARG, "ens_observe: null argument");
    DeviceGuard device_guard(h->device);
    LDG_REQUIRE(instance >= 0 && instance < (int)h->inst.size(), LDG_ERR_ARG, "ens_observe: instance out of range");
    int rc = ens_check(h);
    if (rc) return rc;
    ens_sync_cur(h);
    const qsr_observe_args a = args ? *args : ens_default_observe_args(h, instance);
    return qsr_observe(h->inst[instance], &a, out);
}

int ens_observe_all(ens_handle* h, const qsr_observe_args* args, qsr_observables* out) {
    clear_error();
    LDG_REQUIRE(h && out, LDG_ERR_ARG, "ens_observe_all: null argument");
    DeviceGuard device_guard(h->device);
    int rc = ens_check(h);
    if (rc) return rc;
    ens_sync_cur(h);
    const size_t n = h->inst.size();
    // Every droplet's reductions on the ensemble's stream, after its steps; one copy of all results.
    if (!h->d_obs && (rc = alloc_or_fail((void**)&h->d_obs, n * sizeof(ObsPartial)))) return rc;
    std::vector<ObsPartial> R(n);
    std::vector<qsr_observe_args> a(n);
    for (size_t i = 0; i < n; ++i) {
        a[i] = args ? args[i] : ens_default_observe_args(h, (int)i);
        if ((rc = observe_enqueue(h->inst[i], &a[i], h->stream, h->d_obs + i))) return rc;
    }
    LDG_CUDA(cudaMemcpyAsync(R.data(), h->d_obs, n * sizeof(ObsPartial), cudaMemcpyDeviceToHost, h->stream));
    LDG_CUDA(cudaStreamSynchronize(h->stream));
    for (size_t i = 0; i < n; ++i) observe_finish(h->inst[i], &a[i], R[i], &out[i]);
    return LDG_OK;
}

long long ens_step_index(const ens_handle* h) { return h ? h->step : -1; }

int ens_geometry(const ens_handle* h, int instance, qsr_geometry_info* out) {
    clear_error();
    LDG_REQUIRE(h && out, LDG_ERR_ARG, "ens_geometry: null argument");
    LDG_REQUIRE(instance >= 0 && instance < (int)h->inst.size(), LDG_ERR_ARG, "ens_geometry: instance out of range");
    return qsr_geometry(h->inst[instance], out);
}

int ens_autotune(ens_handle* h, int trial_steps, int* chosen_chunk) {
    clear_error();
    LDG_REQUIRE(h, LDG_ERR_ARG, "ens_autotune: null handle");
    DeviceGuard device_guard(h->device);
    LDG_REQUIRE(trial_steps >= 1, LDG_ERR_ARG, "ens_autotune: trial_steps must be >= 1");
    for (qsr_handle* q : h->inst) LDG_REQUIRE(q->uploaded, LDG_ERR_STATE, "ens_autotune: an instance has no field");
    LDG_CUDA(cudaStreamSynchronize(h->stream));
    // Back up the current field of every instance (the other buffer differs only in cells
    // the next step rewrites).
    const long long step0 = h->step;
    const int w = (int)(step0 & 1);
    std::vector<float*> backup(h->inst.size(), nullptr);
    int rc = LDG_OK;
    for (size_t n = 0; n < h->inst.size() && rc == LDG_OK; ++n) {
        const size_t bytes = (size_t)h->inst[n]->sc * 5 * sizeof(float);
        rc = alloc_or_fail((void**)&backup[n], bytes);
        if (rc == LDG_OK && cudaMemcpyAsync(backup[n], h->inst[n]->q[w], bytes, cudaMemcpyDeviceToDevice, h->stream) !=
                                cudaSuccess) {
            set_error("ens_autotune: backup copy failed");
            rc = LDG_ERR_CUDA;
        }
    }
    const int candidates[] = {8, 12, 16, 24, 32, 48, 64};
    int best = candidates[0];
    std::vector<int> tried;  // lengths in use: on a short list several candidates are cut to the same one
    float best_ms = std::numeric_limits<float>::infinity();
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (rc == LDG_OK && (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess)) {
        set_error("ens_autotune: event creation failed");
        rc = LDG_ERR_CUDA;
    }
    for (int c : candidates) {
        if (rc != LDG_OK) break;
        if ((rc = ens_rechunk(h, ItemLength{c, false}))) break;
        if (std::find(tried.begin(), tried.end(), h->chunk) != tried.end()) continue;
        tried.push_back(h->chunk);
        for (int s = 0; s < 2 && rc == LDG_OK; ++s) rc = ens_launch(h);
        if (rc) break;
        cudaEventRecord(e0, h->stream);
        for (int s = 0; s < trial_steps && rc == LDG_OK; ++s) rc = ens_launch(h);
        if (rc) break;
        cudaEventRecord(e1, h->stream);
        if (cudaEventSynchronize(e1) != cudaSuccess) {
            set_error("ens_autotune: trial failed");
            rc = LDG_ERR_CUDA;
            break;
        }
        h->launches += 2 + trial_steps;
        float ms = 0.0f;
        cudaEventElapsedTime(&ms, e0, e1);
        if (ms < best_ms) { best_ms = ms; best = c; }
        if ((rc = ens_check(h))) break;
    }
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    // Restore the fields into both buffers and the step index, whatever happened above.
    for (size_t n = 0; n < h->inst.size(); ++n) {
        if (!backup[n]) continue;
        const size_t bytes = (size_t)h->inst[n]->sc * 5 * sizeof(float);
        cudaMemcpyAsync(h->inst[n]->q[0], backup[n], bytes, cudaMemcpyDeviceToDevice, h->stream);
        cudaMemcpyAsync(h->inst[n]->q[1], backup[n], bytes, cudaMemcpyDeviceToDevice, h->stream);
    }
    cudaStreamSynchronize(h->stream);
    for (float* b : backup) cudaFree(b);
    {
        const std::string msg = ldg_last_error();
        const int e = ens_set_step(h, step0);
        if (rc != LDG_OK) set_error(msg);
        if (rc != LDG_OK || (rc = e)) return rc;
    }
    if ((rc = ens_rechunk(h, ItemLength{best, false}))) return rc;
    if ((rc = ens_build_graph(h))) return rc;
    if (chosen_chunk) *chosen_chunk = best;
    return LDG_OK;
}

long long ens_cells(const ens_handle* h) { return h ? h->cells : 0; }
long long ens_active_cells(const ens_handle* h) { return h ? h->active : 0; }
long long ens_written_cells(const ens_handle* h) { return h ? h->written : 0; }
void* ens_stream(ens_handle* h) { return h ? (void*)h->stream : nullptr; }
long long ens_launch_count(const ens_handle* h) {
    if (!h) return 0;
    long long n = h->launches;
    for (const qsr_handle* q : h->inst) n += q->launches;
    return n;
}

int ens_destroy(ens_handle* h) {
    if (!h) return LDG_OK;
    DeviceGuard device_guard(h->device);
    if (h->stream) cudaStreamSynchronize(h->stream);
    ens_drop_graph(h);
    for (qsr_handle* q : h->inst) qsr_destroy(q);
    cudaFree(h->stage);
    cudaFree(h->d_obs);
    cudaFree(h->d_tms); cudaFree(h->d_inst); cudaFree(h->d_items); cudaFree(h->d_masks); cudaFree(h->d_ctl); cudaFree(h->d_err);
    if (h->stream) cudaStreamDestroy(h->stream);
    delete h;
    return LDG_OK;
}

}  // extern "C"
