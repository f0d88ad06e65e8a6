// Shared device code of the B200 LdG solver: field layout, per-cell physics written
// against a neighbour accessor, the counter-based noise generator and the FP64 nematic
// eigen-solver used by the reductions.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace ldg {

// Per-cell classification bits, computed once on the host in FP64 (qsr.cu) from the
// reference predicates (QSR.cu:100-111, 697-709, 851-867, 994-1002, 2288-2300).
enum : uint8_t {
    kMove = 1,     // the update touches the cell: !(W == 0 && shell) && sd <= band
    kFixed = 2,    // strong anchoring: W <= 0 && shell, rewritten to Q0 after the update
    kAnchor = 4,   // weak anchoring penalty: shell && W != 0 && delta_eff > 0
    kShell = 8,    // |sd| <= shell half thickness
    kInside = 16,  // sd <= 0
    kCore = 32,    // sd < -2 min_spacing (avg_S, max_S, checker)
    kRadial = 64,  // inside && |r| > 2 min_spacing (radiality)
};

// Constants of one confined-solver step, passed by value to the kernels. The field is
// FP32 SoA: component c of cell (i, j, k) lives at q[c*sc + i*si + j*sj + k].
struct QsrConst {
    int Nx, Ny, Nz;
    int sj;          // row pitch (>= Nz, multiple of 8)
    long long si;    // plane pitch = Ny*sj
    long long sc;    // component pitch = Nx*si
    float ix2, iy2, iz2;        // 1/d^2
    float i2x, i2y, i2z;        // 1/(2d)
    float ix, iy, iz;           // 1/d
    float i4xy, i4xz, i4yz;     // 1/(4 da db)
    float cQ, cQ2, cQ3;         // bulk force coefficients (QSR.cu:385-397)
    float Liso;                 // kappa if L1 = L2 = L3 = 0, else L1 (QSR.cu:420-438)
    float L2, L3;
    float Weff, S_shell;        // W/delta_eff and the shell order
    float mob_dt;               // dt/gamma
    float qcap;                 // Frobenius cap (0 = off)
    float ci, cj, ck;           // droplet centre in cell units, (N-1)/2
    float gnx, gny, gnz;        // d/r^2 per axis: surface normal ~ (X gnx, Y gny, Z gnz)
    float sigma;                // Langevin amplitude per component (0 = off)
    uint32_t key0, key1;        // Philox key (seed)
    uint32_t instance;          // ensemble instance id (noise counter word)
    long long step;             // global step index (noise counter words)
    // semi-implicit (IMEX) Helmholtz-Jacobi
    float alpha;                // (dt/gamma) L_stab
    float jdenom_inv;           // 1/(1 + 2 alpha sum 1/d^2)
    // products of the constants above, folded on the host so the interior stencils need one
    // fused multiply-add per term
    float lap_c;                // -2 (1/dx^2 + 1/dy^2 + 1/dz^2): centre weight of the Laplacian
    float L2i2x, L2i2y, L2i2z;  // L2/(2d)
    float l3m[6];               // (L3/2) / (4 da db) for M_ab from undivided central differences (xx yy zz xy xz yz)
    float l2w[6];               // L2 / (4 da db) for d_a D_b from undivided second differences (xx yy zz xy xz yz)
    float lx, ly, lz;           // Liso/da^2: pure second differences of the L1 term
    float l3s[3];               // L3/da^2: pure second differences of the L3 contraction
    float l3c[3];               // L3/(2 da db): mixed second differences of the L3 contraction (xy xz yz)
    float l3d[6];               // L3/(4 da db): products of first differences in the L3 terms (xx yy zz xy xz yz)
};

// ---------------------------------------------------------------------------------------
// Philox4x32 (Salmon, Moraes, Dror, Shaw, "Parallel random numbers: as easy as 1, 2, 3",
// SC'11) and Box-Muller normals.
// ---------------------------------------------------------------------------------------
// Rounds of the noise generator. The paper reports Philox4x32 with 7 rounds passing TestU01's
// BigCrush (10 is its default safety margin); every noise draw here uses 7.
constexpr int kNoiseRounds = 7;

template <int kRounds>
__device__ __forceinline__ void philox4x32(uint32_t c[4], uint32_t k0, uint32_t k1) {
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
        const uint32_t hi0 = __umulhi(0xD2511F53u, c[0]);
        const uint32_t lo0 = 0xD2511F53u * c[0];
        const uint32_t hi1 = __umulhi(0xCD9E8D57u, c[2]);
        const uint32_t lo1 = 0xCD9E8D57u * c[2];
        const uint32_t n0 = hi1 ^ c[1] ^ k0;
        const uint32_t n2 = hi0 ^ c[3] ^ k1;
        c[0] = n0; c[1] = lo1; c[2] = n2; c[3] = lo0;
        k0 += 0x9E3779B9u; k1 += 0xBB67AE85u;
    }
}

// Uniform (x + 1) 2^-21 in (0, 1] from a 21-bit integer x given as x << 2 in bits 2..22 (other bits
// zero): as the mantissa of a float in [1, 2) it is 1 + x 2^-21, and adding 2^-21 - 1 is exact (the
// result has at most 22 significant bits). Integer and FMA pipes only: a conversion would take the
// same pipe as the logarithms, roots and sines of the draw.
__device__ __forceinline__ float u21(uint32_t x4) {
    return __uint_as_float(0x3F800000u | x4) + (1.0f / 2097152.0f - 1.0f);
}
// Hardware approximations without the subnormal handling of the default forms: every argument of the
// draw is normal (u >= 2^-21, t >= 1e-30), where both give the same value.
__device__ __forceinline__ float lg2_ftz(float x) {
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rsqrt_ftz(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Five standard normals for (cell, instance, step) from one Philox4x32-7 block: the four
// 32-bit words give six disjoint 21-bit fields (the low 21 bits of each word, and the high
// 11 bits of words 0|1 and 2|3 joined), i.e. three Box-Muller pairs; the sixth normal is
// not needed. Counter = (cell, instance, step low word, step high word).
// The radius sqrt(-2 ln u) takes ln u from the hardware base-2 logarithm (absolute error at most
// 2^-22 for u in [0.5, 1], 2 ulp below): a normal is off by at most 2e-4 in absolute terms (only
// when |z| < 0.002, i.e. u within 2e-6 of 1) and by less than 1e-5 relative when |z| > 0.05.
__device__ __forceinline__ void normals5(uint32_t cell, uint32_t instance, long long step, uint32_t k0, uint32_t k1,
                                         float g[5]) {
    uint32_t c[4] = {cell, instance, (uint32_t)step, (uint32_t)((unsigned long long)step >> 32)};
    philox4x32<kNoiseRounds>(c, k0, k1);
    constexpr uint32_t M21 = ((1u << 21) - 1u) << 2;  // the fields are formed shifted left by two (u21)
    const uint32_t f0 = (c[0] << 2) & M21, f1 = (c[1] << 2) & M21, f2 = (c[2] << 2) & M21, f3 = (c[3] << 2) & M21;
    const uint32_t f4 = ((c[0] >> 9) & 0x7FF000u) | ((c[1] >> 20) & 0xFFCu);  // 11 + 10 bits
    const uint32_t f5 = ((c[2] >> 9) & 0x7FF000u) | ((c[3] >> 20) & 0xFFCu);
    // angle 2 pi u taken as pi + t with t = 2 pi u - pi in (-pi, pi], where the fast hardware
    // sine/cosine is accurate to ~4e-7: cos(2 pi u) = -cos t, sin(2 pi u) = -sin t
    constexpr float kTwoPi = 6.28318530717958647692f, kPi = 3.14159265358979323846f;
    constexpr float kM2Ln2 = -1.38629436111989061883f;  // -2 ln 2
    // radius sqrt(-2 ln u) = t * rsqrt(t), t = -2 ln 2 log2(u) (the guard keeps t = 0, u = 1, at zero)
    auto radius = [](float u) {
        const float t = kM2Ln2 * lg2_ftz(u);
        return t * rsqrt_ftz(fmaxf(t, 1e-30f));
    };
    float s, co;
    float r = radius(u21(f0));
    __sincosf(fmaf(kTwoPi, u21(f1), -kPi), &s, &co);
    g[0] = -r * co;
    g[1] = -r * s;
    r = radius(u21(f2));
    __sincosf(fmaf(kTwoPi, u21(f3), -kPi), &s, &co);
    g[2] = -r * co;
    g[3] = -r * s;
    r = radius(u21(f4));
    g[4] = -r * __cosf(fmaf(kTwoPi, u21(f5), -kPi));
}

// ---------------------------------------------------------------------------------------
// Stencil physics. `A(c, di, dj, dk)` returns component c (0..4, 5 = Qzz) of the cell at
// offset (di, dj, dk); the face logic below never asks for a cell outside the grid.
// ---------------------------------------------------------------------------------------

// Second derivative along one axis with the reference's shifted stencil at the faces
// (QSR.cu:296-320).
// kFaces = false is the interior form: the caller guarantees 0 < pos < n - 1 for every
// position the stencil is evaluated at, so the face branches are compiled out.
template <int AX, bool kFaces = true, class Acc>
__device__ __forceinline__ float d2_face(const Acc& A, int c, float cv, int pos, int n, float inv) {
    auto at = [&](int s) { return AX == 0 ? A(c, s, 0, 0) : (AX == 1 ? A(c, 0, s, 0) : A(c, 0, 0, s)); };
    if (!kFaces || (pos > 0 && pos < n - 1)) return (at(1) - cv * 2.0f + at(-1)) * inv;
    if (pos == 0) return (at(2) - at(1) * 2.0f + cv) * inv;
    return (cv - at(-1) * 2.0f + at(-2)) * inv;
}

// First derivative along one axis at offset (oi, oj, ok), one-sided first order at the faces
// (QSR.cu:245-273). `pos` is the absolute coordinate of the offset cell along AX.
template <int AX, bool kFaces = true, class Acc>
__device__ __forceinline__ float d1_face(const Acc& A, int c, int oi, int oj, int ok, int pos, int n, float i2, float i1) {
    auto at = [&](int s) {
        return AX == 0 ? A(c, oi + s, oj, ok) : (AX == 1 ? A(c, oi, oj + s, ok) : A(c, oi, oj, ok + s));
    };
    if (!kFaces || (pos > 0 && pos < n - 1)) return (at(1) - at(-1)) * i2;
    if (pos == 0) return (at(1) - at(0)) * i1;
    return (at(0) - at(-1)) * i1;
}

// Column divergence D_j = d_k Q_kj at offset (oi, oj, ok) of cell (i, j, k) (QSR.cu:325-371).
template <bool kFaces = true, class Acc>
__device__ __forceinline__ void dcol_at(const Acc& A, const QsrConst& P, int i, int j, int k, int oi, int oj, int ok,
                                        float D[3]) {
    const int pi = i + oi, pj = j + oj, pk = k + ok;
    D[0] = d1_face<0, kFaces>(A, 0, oi, oj, ok, pi, P.Nx, P.i2x, P.ix) +
           d1_face<1, kFaces>(A, 1, oi, oj, ok, pj, P.Ny, P.i2y, P.iy) +
           d1_face<2, kFaces>(A, 2, oi, oj, ok, pk, P.Nz, P.i2z, P.iz);
    D[1] = d1_face<0, kFaces>(A, 1, oi, oj, ok, pi, P.Nx, P.i2x, P.ix) +
           d1_face<1, kFaces>(A, 3, oi, oj, ok, pj, P.Ny, P.i2y, P.iy) +
           d1_face<2, kFaces>(A, 4, oi, oj, ok, pk, P.Nz, P.i2z, P.iz);
    D[2] = d1_face<0, kFaces>(A, 2, oi, oj, ok, pi, P.Nx, P.i2x, P.ix) +
           d1_face<1, kFaces>(A, 4, oi, oj, ok, pj, P.Ny, P.i2y, P.iy) +
           d1_face<2, kFaces>(A, 5, oi, oj, ok, pk, P.Nz, P.i2z, P.iz);
}

// Bulk molecular field entries xx yy zz xy xz yz (QSR.cu:399-417).
__device__ __forceinline__ void bulk_field(const float q[5], float cQ, float cQ2, float cQ3, float h[6]) {
    const float Qxx = q[0], Qxy = q[1], Qxz = q[2], Qyy = q[3], Qyz = q[4];
    const float Qzz = -Qxx - Qyy;
    const float trQ2 = Qxx * Qxx + Qyy * Qyy + Qzz * Qzz + 2.0f * (Qxy * Qxy + Qxz * Qxz + Qyz * Qyz);
    const float q2xx = Qxx * Qxx + Qxy * Qxy + Qxz * Qxz;
    const float q2xy = Qxx * Qxy + Qxy * Qyy + Qxz * Qyz;
    const float q2xz = Qxx * Qxz + Qxy * Qyz + Qxz * Qzz;
    const float q2yy = Qxy * Qxy + Qyy * Qyy + Qyz * Qyz;
    const float q2yz = Qxy * Qxz + Qyy * Qyz + Qyz * Qzz;
    const float q2zz = Qxz * Qxz + Qyz * Qyz + Qzz * Qzz;
    const float t3 = trQ2 * (1.0f / 3.0f);  // FP32 path: reciprocal multiply (one rounding)
    // cQ Q - cQ2 (Q^2 - tr/3) + cQ3 tr(Q^2) Q with the two linear terms joined: (cQ + cQ3 tr) Q
    const float cg = fmaf(cQ3, trQ2, cQ);
    h[0] = fmaf(-cQ2, q2xx - t3, cg * Qxx);
    h[1] = fmaf(-cQ2, q2yy - t3, cg * Qyy);
    h[2] = fmaf(-cQ2, q2zz - t3, cg * Qzz);
    h[3] = fmaf(-cQ2, q2xy, cg * Qxy);
    h[4] = fmaf(-cQ2, q2xz, cg * Qxz);
    h[5] = fmaf(-cQ2, q2yz, cg * Qyz);
}

// Droplet surface normal at cell (i, j, k) (QSR.cu:130-142), in FP32 from cell units.
__device__ __forceinline__ void surface_q0(const QsrConst& P, int i, int j, int k, float Q0[5]) {
    const float gx = ((float)i - P.ci) * P.gnx, gy = ((float)j - P.cj) * P.gny, gz = ((float)k - P.ck) * P.gnz;
    const float g2 = gx * gx + gy * gy + gz * gz;
    float nx = 1.0f, ny = 0.0f, nz = 0.0f;
    if (g2 > 0.0f) {  // unit normal by one reciprocal square root (2 ulp) instead of three divisions
        const float inv = rsqrtf(g2);
        nx = gx * inv; ny = gy * inv; nz = gz * inv;
    }
    const float S = P.S_shell;
    Q0[0] = S * (nx * nx - 1.0f / 3.0f);
    Q0[1] = S * (nx * ny);
    Q0[2] = S * (nx * nz);
    Q0[3] = S * (ny * ny - 1.0f / 3.0f);
    Q0[4] = S * (ny * nz);
}

// Chemical potential of cell (i, j, k): bulk + elastic (iso | L1, L2) projected traceless,
// then L3 on interior cells re-projected, then the weak-anchoring penalty
// (QSR.cu:373-472, 474-621, 623-652). `lap` returns the Laplacian (IMEX uses it).
// DAcc(c, di, dj, dk) returns the column divergence D_c at a face-neighbour offset.
// kFaces = false: the caller guarantees the cell and all stencil positions are interior.
template <bool kL2, bool kL3, bool kFaces = true, class Acc, class DAcc>
__device__ __forceinline__ void chem_potential(const Acc& A, const DAcc& DA, const QsrConst& P, int i, int j, int k,
                                               const float q[5], bool anchor, float mu[5], float lap[5]) {
#pragma unroll
    for (int c = 0; c < 5; ++c) {
        if (!kFaces) {
            // interior: sum_a (Q[+1] + Q[-1]) / da^2 - 2 Q sum_a 1/da^2
            const float sx = A(c, 1, 0, 0) + A(c, -1, 0, 0);
            const float sy = A(c, 0, 1, 0) + A(c, 0, -1, 0);
            const float sz = A(c, 0, 0, 1) + A(c, 0, 0, -1);
            lap[c] = fmaf(P.ix2, sx, fmaf(P.iy2, sy, fmaf(P.iz2, sz, P.lap_c * q[c])));
        } else {
            const float d2x = d2_face<0, kFaces>(A, c, q[c], i, P.Nx, P.ix2);
            const float d2y = d2_face<1, kFaces>(A, c, q[c], j, P.Ny, P.iy2);
            const float d2z = d2_face<2, kFaces>(A, c, q[c], k, P.Nz, P.iz2);
            lap[c] = d2x + d2y + d2z;
        }
    }
    float h[6];
    bulk_field(q, P.cQ, P.cQ2, P.cQ3, h);
    const float lzz = -lap[0] - lap[3];
    h[0] -= P.Liso * lap[0];
    h[1] -= P.Liso * lap[3];
    h[2] -= P.Liso * lzz;
    h[3] -= P.Liso * lap[1];
    h[4] -= P.Liso * lap[2];
    h[5] -= P.Liso * lap[4];
    if (kL2) {
        // h -= L2 d_a D_b, d_a central with one-sided faces (QSR.cu:436-460). sub() applies one
        // term as a fused multiply-add with L2/(2 da) (central) or L2/da = 2 L2/(2 da) (one-sided).
        auto sub = [&](float& hv, int comp, int ax) {
            const int pos = ax == 0 ? i : (ax == 1 ? j : k);
            const int n = ax == 0 ? P.Nx : (ax == 1 ? P.Ny : P.Nz);
            const float c2 = ax == 0 ? P.L2i2x : (ax == 1 ? P.L2i2y : P.L2i2z);
            auto at = [&](int s) {
                return ax == 0 ? DA(comp, s, 0, 0) : (ax == 1 ? DA(comp, 0, s, 0) : DA(comp, 0, 0, s));
            };
            if (!kFaces || (pos > 0 && pos < n - 1)) hv = fmaf(-c2, at(1) - at(-1), hv);
            else if (pos == 0) hv = fmaf(-2.0f * c2, at(1) - at(0), hv);
            else hv = fmaf(-2.0f * c2, at(0) - at(-1), hv);
        };
        sub(h[0], 0, 0);
        sub(h[1], 1, 1);
        sub(h[2], 2, 2);
        sub(h[3], 1, 0);
        sub(h[3], 0, 1);
        sub(h[4], 2, 0);
        sub(h[4], 0, 2);
        sub(h[5], 2, 1);
        sub(h[5], 1, 2);
    }
    float corr = (h[0] + h[1] + h[2]) * (1.0f / 3.0f);
    mu[0] = h[0] - corr;
    mu[1] = h[3];
    mu[2] = h[4];
    mu[3] = h[1] - corr;
    mu[4] = h[5];
    if (kL3) {
        const bool interior =
            !kFaces || (i > 0 && i < P.Nx - 1 && j > 0 && j < P.Ny - 1 && k > 0 && k < P.Nz - 1);
        if (interior) {
            float hx[6] = {mu[0], mu[3], -(mu[0] + mu[3]), mu[1], mu[2], mu[4]};
            // undivided central differences Q[+1] - Q[-1]; the 1/(2 da) factors are folded into
            // the M_ab weights (P.l3m) and into the divergence below
            float d[6][3];
#pragma unroll
            for (int c = 0; c < 5; ++c) {
                d[c][0] = A(c, 1, 0, 0) - A(c, -1, 0, 0);
                d[c][1] = A(c, 0, 1, 0) - A(c, 0, -1, 0);
                d[c][2] = A(c, 0, 0, 1) - A(c, 0, 0, -1);
            }
#pragma unroll
            for (int a = 0; a < 3; ++a) d[5][a] = -(d[0][a] + d[3][a]);
            auto M = [&](int a, int b) {
                return d[0][a] * d[0][b] + d[3][a] * d[3][b] + d[5][a] * d[5][b] +
                       2.0f * (d[1][a] * d[1][b] + d[2][a] * d[2][b] + d[4][a] * d[4][b]);
            };
            hx[0] = fmaf(P.l3m[0], M(0, 0), hx[0]);
            hx[1] = fmaf(P.l3m[1], M(1, 1), hx[1]);
            hx[2] = fmaf(P.l3m[2], M(2, 2), hx[2]);
            hx[3] = fmaf(P.l3m[3], M(0, 1), hx[3]);
            hx[4] = fmaf(P.l3m[4], M(0, 2), hx[4]);
            hx[5] = fmaf(P.l3m[5], M(1, 2), hx[5]);
            const float Qxx = q[0], Qxy = q[1], Qxz = q[2], Qyy = q[3], Qyz = q[4], Qzz = -q[0] - q[3];
            // D_a / (2 da): pairs with the undivided differences in D . grad Q_c
            const float Dc0 = DA(0, 0, 0, 0) * P.i2x, Dc1 = DA(1, 0, 0, 0) * P.i2y, Dc2 = DA(2, 0, 0, 0) * P.i2z;
            // B(Q_c) = D . grad Q_c + Q_ab d_a d_b Q_c (QSR.cu:580-603), with the Q_ab / (stencil
            // denominator) weights formed once for all five components.
            const float wxx = Qxx * P.ix2, wyy = Qyy * P.iy2, wzz = Qzz * P.iz2;
            const float wxy = 2.0f * Qxy * P.i4xy, wxz = 2.0f * Qxz * P.i4xz, wyz = 2.0f * Qyz * P.i4yz;
            auto Bc = [&](int c) {
                const float Qc2 = 2.0f * (c == 5 ? Qzz : q[c]);
                const float sxx = (A(c, 1, 0, 0) + A(c, -1, 0, 0)) - Qc2;
                const float syy = (A(c, 0, 1, 0) + A(c, 0, -1, 0)) - Qc2;
                const float szz = (A(c, 0, 0, 1) + A(c, 0, 0, -1)) - Qc2;
                const float sxy = (A(c, 1, 1, 0) - A(c, 1, -1, 0)) - (A(c, -1, 1, 0) - A(c, -1, -1, 0));
                const float sxz = (A(c, 1, 0, 1) - A(c, 1, 0, -1)) - (A(c, -1, 0, 1) - A(c, -1, 0, -1));
                const float syz = (A(c, 0, 1, 1) - A(c, 0, 1, -1)) - (A(c, 0, -1, 1) - A(c, 0, -1, -1));
                const float contract = wxx * sxx + wyy * syy + wzz * szz + wxy * sxy + wxz * sxz + wyz * syz;
                return fmaf(Dc0, d[c][0], fmaf(Dc1, d[c][1], fmaf(Dc2, d[c][2], contract)));
            };
            const float Bxx = Bc(0), Byy = Bc(3), Bzz = -(Bxx + Byy);
            const float Bxy = Bc(1), Bxz = Bc(2), Byz = Bc(4);
            hx[0] -= P.L3 * Bxx;
            hx[1] -= P.L3 * Byy;
            hx[2] -= P.L3 * Bzz;
            hx[3] -= P.L3 * Bxy;
            hx[4] -= P.L3 * Bxz;
            hx[5] -= P.L3 * Byz;
            corr = (hx[0] + hx[1] + hx[2]) * (1.0f / 3.0f);
            mu[0] = hx[0] - corr;
            mu[3] = hx[1] - corr;
            mu[1] = hx[3];
            mu[2] = hx[4];
            mu[4] = hx[5];
        }
    }
    if (anchor) {
        float Q0[5];
        surface_q0(P, i, j, k, Q0);
#pragma unroll
        for (int c = 0; c < 5; ++c) mu[c] += P.Weff * (q[c] - Q0[c]);
    }
}

// ---------------------------------------------------------------------------------------
// Two cells at once: F2 holds one value of two different cells, and every operation on it is
// one packed instruction (FFMA2 / FADD2 / FMUL2) for both cells. The routines below are written
// on a value type F, which is F2 (two cells) or float (one cell).
// ---------------------------------------------------------------------------------------
struct F2 {
    float2 v;
};
__device__ __forceinline__ F2 mk2(float a, float b) { return F2{make_float2(a, b)}; }
__device__ __forceinline__ F2 operator+(F2 a, F2 b) { return F2{__fadd2_rn(a.v, b.v)}; }
__device__ __forceinline__ F2 operator-(F2 a, F2 b) { return F2{__ffma2_rn(b.v, make_float2(-1.0f, -1.0f), a.v)}; }
__device__ __forceinline__ F2 operator*(F2 a, F2 b) { return F2{__fmul2_rn(a.v, b.v)}; }
__device__ __forceinline__ F2 operator*(float s, F2 b) { return F2{__fmul2_rn(make_float2(s, s), b.v)}; }
__device__ __forceinline__ F2 operator-(F2 a) { return F2{__fmul2_rn(a.v, make_float2(-1.0f, -1.0f))}; }
__device__ __forceinline__ F2 vfma(F2 a, F2 b, F2 c) { return F2{__ffma2_rn(a.v, b.v, c.v)}; }
__device__ __forceinline__ F2 vfma(float a, F2 b, F2 c) { return F2{__ffma2_rn(make_float2(a, a), b.v, c.v)}; }
__device__ __forceinline__ float vfma(float a, float b, float c) { return fmaf(a, b, c); }
template <class F>
__device__ __forceinline__ F vset(float a);
template <>
__device__ __forceinline__ F2 vset<F2>(float a) { return mk2(a, a); }
template <>
__device__ __forceinline__ float vset<float>(float a) { return a; }

// Bulk molecular field of the five stored components (xx, xy, xz, yy, yz). It is traceless as
// written (tr(Q^2 - I tr Q^2 / 3) = 0 and Qzz = -(Qxx + Qyy)), so the zz entry is never formed;
// with Qzz eliminated the off-diagonal entries of Q^2 are two products each. The diagonal entries of
// Q^2 - I tr Q^2 / 3 are formed from their own products, (q2xx - 2 u) / 3 and (q2yy - 2 w) / 3, before they meet
// cQ2: taking q2xx and tr Q^2 / 3 to cQ2 apart needs four operations less and rounded 1.25 to 1.3 times as much as
// the six-entry form above at S = 0.5; this one rounds 0.78 times as much.
// Coefficients of the bulk field as values of F: a packed operation takes a pair in registers or
// in the kernel's parameters, and a scalar would have to be copied into both halves at every use.
template <class F>
struct BulkC {
    F cQ, cQ3x2, m3, cQ2, mcQ2;  // cQ, 2 cQ3, -cQ2/3, cQ2, -cQ2
};
template <class F>
__device__ __forceinline__ void bulk_field5(const F q[5], const BulkC<F>& K, F h[5]) {
    const F Qxx = q[0], Qxy = q[1], Qxz = q[2], Qyy = q[3], Qyz = q[4];
    const F s = Qxx + Qyy;  // -Qzz
    const F q2xx = vfma(Qxx, Qxx, vfma(Qxy, Qxy, Qxz * Qxz));
    const F q2yy = vfma(Qyy, Qyy, vfma(Qxy, Qxy, Qyz * Qyz));
    const F u = vfma(Qyy, s, Qyz * Qyz), w = vfma(Qxx, s, Qxz * Qxz);  // tr(Q^2) / 2 less q2xx, less q2yy
    const F cg = vfma(K.cQ3x2, q2xx + u, K.cQ);                        // cQ + cQ3 tr(Q^2)
    const F m1 = K.mcQ2 * Qxy, m2 = K.mcQ2 * Qxz;
    h[0] = vfma(K.m3, vfma(-2.0f, u, q2xx), cg * Qxx);
    h[3] = vfma(K.m3, vfma(-2.0f, w, q2yy), cg * Qyy);
    h[1] = vfma(vfma(K.mcQ2, s, cg), Qxy, m2 * Qyz);    // (Q^2)_xy = Qxy (Qxx + Qyy) + Qxz Qyz
    h[2] = vfma(vfma(K.cQ2, Qyy, cg), Qxz, m1 * Qyz);   // (Q^2)_xz = Qxy Qyz - Qxz Qyy
    h[4] = vfma(vfma(K.cQ2, Qxx, cg), Qyz, m1 * Qxz);   // (Q^2)_yz = Qxy Qxz - Qyz Qxx
}

// What one component contributes to the stencil terms of a cell: undivided first differences
// Q[+1] - Q[-1], sums Q[+1] + Q[-1] (interior) or whole second differences (face stencils), mixed
// second differences of the four corners, and the L2 term's wide second differences, again as sums
// Q[+2] + Q[-2] (interior) or whole (face stencils).
template <class F>
struct Sten {
    F d[3], s[3], mxy, mxz, myz, wx, wy, wz;
};

// Chemical potential (bulk, L1, L2, L3) of one or two cells; S(c, o) fills the stencil of stored
// component c (0 xx, 1 xy, 2 xz, 3 yy, 4 yz). The FMA pipe and the issue slots bound it, so it is
// arranged to need few operations rather than to follow the reference term by term:
//  * the L1 Laplacian and the L3 contraction Q_ab d_a d_b Q_c use the same second differences, so
//    they share one weight per axis, Liso/da^2 + L3 Q_aa/da^2, formed once for all components;
//  * bulk, L1 and L3 D.grad + contraction terms are traceless, so only the L2 term and the
//    (L3/2) M_ab term (kept apart in ax, ay, az) need the traceless projection, and no zz entry
//    of the others is formed (the reference projects after the L1/L2 terms and again after L3,
//    QSR.cu:462-469 and 611-619; the projection is linear);
//  * M_ab is summed over the five stored components: dQ_zz = -(dQ_xx + dQ_yy) turns the three
//    diagonal products into two;
//  * the centre terms -2 Q of the L1 and L3 sums are collected per entry;
//  * the many small terms of L2, M_ab and D.grad are summed apart and meet the bulk and L1 terms once: added one by
//    one, and with the centre terms of the wide differences collected too, they rounded 1.1 to 1.3 times as much
//    as the term-by-term form (chem_potential) does, this way 0.75 to 0.99 times, for 1 to 2 % of a step with all
//    terms (256^3, R = 120: 144.9 -> 146.6 us).
// The L2 term d_a D_b is sum_k S_ak(Q_kb) / (4 da dk): the wide second difference for k = a, four
// corners for k != a. With kFace the stencils hold the reference's one-sided forms (QSR.cu:245-371)
// in the same undivided units and l3on is 0 for a cell on a face (no L3 term there, QSR.cu:474-621).
// lap is formed for the IMEX right-hand side only.
template <bool kL2, bool kL3, bool kLap, bool kFace, class F, class St>
__device__ __forceinline__ void chem_core(const St& S, const QsrConst& P, const F q[5], F l3on, F mu[5], F lap[5]) {
    F* h = mu;
    const BulkC<F> K{vset<F>(P.cQ), vset<F>(2.0f * P.cQ3), vset<F>(-1.0f / 3.0f * P.cQ2), vset<F>(P.cQ2),
                     vset<F>(-P.cQ2)};
    bulk_field5<F>(q, K, h);
    const float cxx = P.l2w[0], cyy = P.l2w[1], czz = P.l2w[2], cxy = P.l2w[3], cxz = P.l2w[4], cyz = P.l2w[5];
    F gx = vset<F>(P.lx), gy = vset<F>(P.ly), gz = vset<F>(P.lz);
    F gxy{}, gxz{}, gyz{};
    if (kL3) {
        const F q0 = kFace ? l3on * q[0] : q[0], q3 = kFace ? l3on * q[3] : q[3];
        gx = vfma(P.l3s[0], q0, gx);
        gy = vfma(P.l3s[1], q3, gy);
        gz = vfma(-P.l3s[2], q0 + q3, gz);
        gxy = P.l3c[0] * q[1];
        gxz = P.l3c[1] * q[2];
        gyz = P.l3c[2] * q[4];
        if (kFace) { gxy = l3on * gxy; gxz = l3on * gxz; gyz = l3on * gyz; }
    }
    F g0{};
    if (!kFace) g0 = -2.0f * (gx + gy + gz);
    // The L2 and M_ab terms (xx, yy, zz apart, for the projection) and then D.grad, to be added to the others at the end.
    F ax = vset<F>(0.0f), ay = ax, az = ax, b[5] = {ax, ax, ax, ax, ax};
    F d[5][3];
#pragma unroll
    for (int c = 0; c < 5; ++c) {
        Sten<F> o;
        S(c, o);
#pragma unroll
        for (int a = 0; a < 3; ++a) d[c][a] = o.d[a];
        F e = vfma(gx, o.s[0], vfma(gy, o.s[1], gz * o.s[2]));
        if (!kFace) e = vfma(g0, q[c], e);
        if (kLap) {
            lap[c] = vfma(P.ix2, o.s[0], vfma(P.iy2, o.s[1], P.iz2 * o.s[2]));
            if (!kFace) lap[c] = vfma(P.lap_c, q[c], lap[c]);
        }
        if (kL3) e = vfma(gxy, o.mxy, vfma(gxz, o.mxz, vfma(gyz, o.myz, e)));
        if (kL2 && !kFace) {
            if (c == 0 || c == 1 || c == 2) o.wx = vfma(-2.0f, q[c], o.wx);
            if (c == 1 || c == 3 || c == 4) o.wy = vfma(-2.0f, q[c], o.wy);
            if (c != 1) o.wz = vfma(-2.0f, q[c], o.wz);
        }
        if (kL2) {
            if (c == 0) {  // xx
                ax = vfma(-cxx, o.wx, ax);
                az = vfma(czz, o.wz, az);
                b[1] = vfma(-cxy, o.mxy, b[1]);
                b[4] = vfma(cyz, o.myz, b[4]);
            } else if (c == 3) {  // yy
                ay = vfma(-cyy, o.wy, ay);
                az = vfma(czz, o.wz, az);
                b[1] = vfma(-cxy, o.mxy, b[1]);
                b[2] = vfma(cxz, o.mxz, b[2]);
            } else if (c == 1) {  // xy
                ax = vfma(-cxy, o.mxy, ax);
                ay = vfma(-cxy, o.mxy, ay);
                b[1] = vfma(-cxx, o.wx, vfma(-cyy, o.wy, b[1]));
                b[2] = vfma(-cyz, o.myz, b[2]);
                b[4] = vfma(-cxz, o.mxz, b[4]);
            } else if (c == 2) {  // xz
                ax = vfma(-cxz, o.mxz, ax);
                az = vfma(-cxz, o.mxz, az);
                b[1] = vfma(-cyz, o.myz, b[1]);
                b[2] = vfma(-cxx, o.wx, vfma(-czz, o.wz, b[2]));
                b[4] = vfma(-cxy, o.mxy, b[4]);
            } else {  // yz
                ay = vfma(-cyz, o.myz, ay);
                az = vfma(-cyz, o.myz, az);
                b[1] = vfma(-cxz, o.mxz, b[1]);
                b[2] = vfma(-cxy, o.mxy, b[2]);
                b[4] = vfma(-cyy, o.wy, vfma(-czz, o.wz, b[4]));
            }
        }
        h[c] = h[c] - e;
    }
    if (kL3) {
        // the face form drops the whole term through its first differences (each term has two)
        if (kFace) {
#pragma unroll
            for (int c = 0; c < 5; ++c)
#pragma unroll
                for (int a = 0; a < 3; ++a) d[c][a] = l3on * d[c][a];
        }
        // (L3/2) M_ab, M_ab = dQ_kl/da dQ_kl/db over all nine entries
        F ex[3], ey[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            ex[a] = vfma(0.5f, d[3][a], d[0][a]);
            ey[a] = vfma(0.5f, d[0][a], d[3][a]);
        }
        auto M = [&](int a, int b) {  // M_ab / 2 (undivided)
            return vfma(d[0][a], ex[b], vfma(d[3][a], ey[b], vfma(d[1][a], d[1][b], vfma(d[2][a], d[2][b],
                        d[4][a] * d[4][b]))));
        };
        ax = vfma(P.l3d[0], M(0, 0), ax);
        ay = vfma(P.l3d[1], M(1, 1), ay);
        az = vfma(P.l3d[2], M(2, 2), az);
        b[1] = vfma(P.l3d[3], M(0, 1), b[1]);
        b[2] = vfma(P.l3d[4], M(0, 2), b[2]);
        b[4] = vfma(P.l3d[5], M(1, 2), b[4]);
        // -L3 D_a / (2 da) with the centre divergence D_x = d_x Q_xx + d_y Q_xy + d_z Q_xz, ... (QSR.cu:325-371)
        const F Dx = vfma(-P.l3d[0], d[0][0], vfma(-P.l3d[3], d[1][1], -P.l3d[4] * d[2][2]));
        const F Dy = vfma(-P.l3d[3], d[1][0], vfma(-P.l3d[1], d[3][1], -P.l3d[5] * d[4][2]));
        const F Dz = vfma(-P.l3d[4], d[2][0], vfma(-P.l3d[5], d[4][1], P.l3d[2] * (d[0][2] + d[3][2])));
#pragma unroll
        for (int c = 0; c < 5; ++c) b[c] = vfma(Dx, d[c][0], vfma(Dy, d[c][1], vfma(Dz, d[c][2], b[c])));
    }
    if (kL2 || kL3) {
        const F corr = (1.0f / 3.0f) * (ax + ay + az);
        b[0] = b[0] + (ax - corr);
        b[3] = b[3] + (ay - corr);
#pragma unroll
        for (int c = 0; c < 5; ++c) h[c] = h[c] + b[c];
    }
}

// Interior stencil of two cells, rows j and j + 1 of one column. V(c, di, dj, dk) returns component
// c at that offset from row j (so dj runs over -2 .. 3). Differences along j are formed per row: the
// two rows overlap (row j is a neighbour of row j + 1), and a packed operand would have to be
// assembled from them with register moves.
template <bool kL2, bool kL3, class Val>
struct InteriorPair {
    const Val& V;
    __device__ __forceinline__ void operator()(int c, Sten<F2>& o) const {
        auto pair = [&](int di, int dk) { return mk2(V(c, di, 0, dk), V(c, di, 1, dk)); };
        auto dj = [&](int di, int dk) {  // Q(j + 1) - Q(j - 1) of both rows
            return mk2(V(c, di, 1, dk) - V(c, di, -1, dk), V(c, di, 2, dk) - V(c, di, 0, dk));
        };
        const F2 px = pair(1, 0), mx = pair(-1, 0), pz = pair(0, 1), mz = pair(0, -1);
        o.s[0] = px + mx;
        o.s[1] = mk2(V(c, 0, 1, 0) + V(c, 0, -1, 0), V(c, 0, 2, 0) + V(c, 0, 0, 0));
        o.s[2] = pz + mz;
        o.d[0] = px - mx;
        o.d[1] = dj(0, 0);
        o.d[2] = pz - mz;
        if (kL2 || kL3) {
            o.mxy = dj(1, 0) - dj(-1, 0);
            o.mxz = (pair(1, 1) - pair(1, -1)) - (pair(-1, 1) - pair(-1, -1));
            o.myz = dj(0, 1) - dj(0, -1);
        }
        if (kL2) {
            if (c == 0 || c == 1 || c == 2) o.wx = pair(2, 0) + pair(-2, 0);
            if (c == 1 || c == 3 || c == 4)
                o.wy = mk2(V(c, 0, 2, 0) + V(c, 0, -2, 0), V(c, 0, 3, 0) + V(c, 0, -1, 0));
            if (c != 1) o.wz = pair(0, 2) + pair(0, -2);
        }
    }
};

// The reference's stencils next to a grid face along one axis, as offsets from a cell at position
// `pos` of n: first differences are one-sided at the faces (QSR.cu:245-273), which is the central
// form with its neighbours clamped to the grid and twice the weight (r, relative to 1/(2 d)); second
// differences are the inner neighbour's (QSR.cu:296-320); the derivative of the divergence takes
// the clamped first difference of clamped first differences.
struct FaceAxis {
    int hi, lo, s;           // clamped neighbours; shift of the second difference's centre
    int hh, hl, lh, ll;      // the clamped neighbours' own neighbours
    float r, rh, rl;         // weights of the first differences at the cell and at its neighbours
    __device__ __forceinline__ FaceAxis(int pos, int n) {
        const int h = min(pos + 1, n - 1), l = max(pos - 1, 0);
        hi = h - pos;
        lo = l - pos;
        s = min(max(pos, 1), n - 2) - pos;
        hh = min(h + 1, n - 1) - pos;
        hl = max(h - 1, 0) - pos;
        lh = min(l + 1, n - 1) - pos;
        ll = max(l - 1, 0) - pos;
        r = (pos == 0 || pos == n - 1) ? 2.0f : 1.0f;
        rh = (h == n - 1) ? 2.0f : 1.0f;
        rl = (l == 0) ? 2.0f : 1.0f;
    }
};

// Stencil of one cell of the grid with the face forms along every axis (equal to the interior one
// away from the faces). V(c, di, dj, dk) takes runtime offsets.
template <bool kL2, bool kL3, class Val>
struct FaceOne {
    const Val& V;
    const FaceAxis &x, &y, &z;
    __device__ __forceinline__ void operator()(int c, Sten<float>& o) const {
        o.d[0] = V(c, x.hi, 0, 0) - V(c, x.lo, 0, 0);
        o.d[1] = V(c, 0, y.hi, 0) - V(c, 0, y.lo, 0);
        o.d[2] = V(c, 0, 0, z.hi) - V(c, 0, 0, z.lo);
        o.s[0] = (V(c, x.s + 1, 0, 0) + V(c, x.s - 1, 0, 0)) - 2.0f * V(c, x.s, 0, 0);
        o.s[1] = (V(c, 0, y.s + 1, 0) + V(c, 0, y.s - 1, 0)) - 2.0f * V(c, 0, y.s, 0);
        o.s[2] = (V(c, 0, 0, z.s + 1) + V(c, 0, 0, z.s - 1)) - 2.0f * V(c, 0, 0, z.s);
        if (kL2 || kL3) {
            o.mxy = (x.r * y.r) * ((V(c, x.hi, y.hi, 0) - V(c, x.hi, y.lo, 0)) - (V(c, x.lo, y.hi, 0) - V(c, x.lo, y.lo, 0)));
            o.mxz = (x.r * z.r) * ((V(c, x.hi, 0, z.hi) - V(c, x.hi, 0, z.lo)) - (V(c, x.lo, 0, z.hi) - V(c, x.lo, 0, z.lo)));
            o.myz = (y.r * z.r) * ((V(c, 0, y.hi, z.hi) - V(c, 0, y.hi, z.lo)) - (V(c, 0, y.lo, z.hi) - V(c, 0, y.lo, z.lo)));
        }
        if (kL2) {
            if (c == 0 || c == 1 || c == 2)
                o.wx = x.r * (x.rh * (V(c, x.hh, 0, 0) - V(c, x.hl, 0, 0)) - x.rl * (V(c, x.lh, 0, 0) - V(c, x.ll, 0, 0)));
            if (c == 1 || c == 3 || c == 4)
                o.wy = y.r * (y.rh * (V(c, 0, y.hh, 0) - V(c, 0, y.hl, 0)) - y.rl * (V(c, 0, y.lh, 0) - V(c, 0, y.ll, 0)));
            if (c != 1)
                o.wz = z.r * (z.rh * (V(c, 0, 0, z.hh) - V(c, 0, 0, z.hl)) - z.rl * (V(c, 0, 0, z.lh) - V(c, 0, 0, z.ll)));
        }
    }
};

// Frobenius-norm cap of the explicit update (QSR.cu:719-731).
__device__ __forceinline__ void cap_norm(float qcap, float out[5]) {
    const float zz = -out[0] - out[3];
    const float tr = out[0] * out[0] + out[3] * out[3] + zz * zz +
                     2.0f * (out[1] * out[1] + out[2] * out[2] + out[4] * out[4]);
    const float qn = sqrtf(tr > 0.0f ? tr : 0.0f);
    if (qn > qcap && qn > 0.0f) {
        const float s = qcap / qn;
#pragma unroll
        for (int c = 0; c < 5; ++c) out[c] *= s;
    }
}

// Explicit update with compensated storage: a cell holds hi + lo (two FP32 words). The
// increment -(dt/gamma) mu (+ noise) is added to hi exactly (Knuth's TwoSum) and the rounding
// error carried in lo, so the stored value keeps about 48 significant bits over any number of
// steps while the stencil arithmetic stays FP32. On return out = new hi, lo = new lo.
__device__ __forceinline__ void euler_update_comp(const QsrConst& P, const float q[5], float lo[5], const float mu[5],
                                                  uint32_t cell, bool noise, float out[5]) {
    float d[5];
#pragma unroll
    for (int c = 0; c < 5; ++c) d[c] = -mu[c] * P.mob_dt;
    if (noise) {
        float g[5];
        normals5(cell, P.instance, P.step, P.key0, P.key1, g);
#pragma unroll
        for (int c = 0; c < 5; ++c) d[c] += P.sigma * g[c];
    }
#pragma unroll
    for (int c = 0; c < 5; ++c) {
        const float s = __fadd_rn(q[c], d[c]);
        const float bp = __fsub_rn(s, q[c]);
        const float e = __fadd_rn(__fsub_rn(q[c], __fsub_rn(s, bp)), __fsub_rn(d[c], bp));
        const float t = __fadd_rn(e, lo[c]);
        const float h = __fadd_rn(s, t);
        lo[c] = __fsub_rn(t, __fsub_rn(h, s));
        out[c] = h;
    }
    if (P.qcap > 0.0f) {
        const float zz = -out[0] - out[3];
        const float tr = out[0] * out[0] + out[3] * out[3] + zz * zz +
                         2.0f * (out[1] * out[1] + out[2] * out[2] + out[4] * out[4]);
        const float qn = sqrtf(tr > 0.0f ? tr : 0.0f);
        if (qn > P.qcap && qn > 0.0f) {
            const float sc = P.qcap / qn;
#pragma unroll
            for (int c = 0; c < 5; ++c) { out[c] *= sc; lo[c] *= sc; }
        }
    }
}

// Explicit Euler update with optional Langevin noise and Frobenius cap (QSR.cu:711-731).
__device__ __forceinline__ void euler_update(const QsrConst& P, const float q[5], const float mu[5], uint32_t cell,
                                             bool noise, float out[5]) {
#pragma unroll
    for (int c = 0; c < 5; ++c) out[c] = q[c] - mu[c] * P.mob_dt;
    if (noise) {
        float g[5];
        normals5(cell, P.instance, P.step, P.key0, P.key1, g);
#pragma unroll
        for (int c = 0; c < 5; ++c) out[c] += P.sigma * g[c];
    }
    if (P.qcap > 0.0f) cap_norm(P.qcap, out);
}

// ---------------------------------------------------------------------------------------
// FP64 nematic eigen-solver (QSR.cu:191-243): shifted power iteration for the largest
// eigenvalue, S = 1.5 lambda, director gauge nz >= 0.
// The reference takes 15 steps n <- M n / |M n| of M = Q + alpha I. Its intermediate norms only scale
// the vector, so the direction after them is that of M^15 n0 = M^8 M^4 M^2 M n0, by three squarings of
// a symmetric matrix and four products with one norm at the end: about 150 operations instead of 15
// roots and 45 divisions. M is taken relative to alpha, so its powers stay in range. The
// reference's early stop (|M n| < 1e-13) can only come at the first step: alpha bounds the row sums of
// Q, so M is positive semidefinite and |M n| does not fall from one step to the next.
// Where that stop comes, or where the start vector lies almost at right angles to the largest eigenvector, the 15
// normalised steps themselves are taken. The row sums of a negative uniaxial order along (1, 1, 1), or of a negative Q_xy
// alone, are the eigenvector to -alpha, which M shrinks by 1e-12 / alpha: the steps hold on to it, while of M^15 n0
// only rounding is left (NaN, or another eigenvector). |M^15 n0|^2 < 1e-6 |n0|^2 decides: M^15 does not shrink
// the largest eigenvector's share of n0, so every start vector with more than 1e-3 of it stays on the fast way.
// ---------------------------------------------------------------------------------------
struct Nematic { double S, nx, ny, nz; };

struct Sym3 { double xx, xy, xz, yy, yz, zz; };
__device__ __forceinline__ Sym3 square(const Sym3& m) {
    return Sym3{fma(m.xx, m.xx, fma(m.xy, m.xy, m.xz * m.xz)), fma(m.xx, m.xy, fma(m.xy, m.yy, m.xz * m.yz)),
                fma(m.xx, m.xz, fma(m.xy, m.yz, m.xz * m.zz)), fma(m.xy, m.xy, fma(m.yy, m.yy, m.yz * m.yz)),
                fma(m.xy, m.xz, fma(m.yy, m.yz, m.yz * m.zz)), fma(m.xz, m.xz, fma(m.yz, m.yz, m.zz * m.zz))};
}
__device__ __forceinline__ void apply(const Sym3& m, double v[3]) {
    const double x = v[0], y = v[1], z = v[2];
    v[0] = fma(m.xx, x, fma(m.xy, y, m.xz * z));
    v[1] = fma(m.xy, x, fma(m.yy, y, m.yz * z));
    v[2] = fma(m.xz, x, fma(m.yz, y, m.zz * z));
}

// The 15 normalised steps (QSR.cu:203-224). Out of line, and from the tensor alone: cells take it rarely, and the
// callers' registers decide how many blocks share an SM.
inline __device__ __noinline__ double3 nematic_steps(double Qxx, double Qxy, double Qxz, double Qyy, double Qyz,
                                                     double alpha) {
    const double Qzz = -Qxx - Qyy;
    double nx = Qxx + Qxy + Qxz, ny = Qxy + Qyy + Qyz, nz = Qxz + Qyz - Qxx - Qyy;
    const double n0 = sqrt(nx * nx + ny * ny + nz * nz);
    if (n0 > 1e-12) { nx /= n0; ny /= n0; nz /= n0; }
    else { nx = 0.0; ny = 0.0; nz = 1.0; }
    for (int it = 0; it < 15; ++it) {
        const double ax = Qxx * nx + Qxy * ny + Qxz * nz + alpha * nx;
        const double ay = Qxy * nx + Qyy * ny + Qyz * nz + alpha * ny;
        const double az = Qxz * nx + Qyz * ny + Qzz * nz + alpha * nz;
        const double nn = sqrt(ax * ax + ay * ay + az * az);
        if (nn < 1e-13) break;
        nx = ax / nn; ny = ay / nn; nz = az / nn;
    }
    return make_double3(nx, ny, nz);
}

__device__ __forceinline__ Nematic nematic64(const double q[5], double iso_cut, Nematic iso) {
    const double Qxx = q[0], Qxy = q[1], Qxz = q[2], Qyy = q[3], Qyz = q[4];
    const double Qzz = -Qxx - Qyy;
    if (fabs(Qxx) < iso_cut && fabs(Qxy) < iso_cut && fabs(Qxz) < iso_cut && fabs(Qyy) < iso_cut &&
        fabs(Qyz) < iso_cut)
        return iso;
    double n[3] = {Qxx + Qxy + Qxz, Qxy + Qyy + Qyz, Qxz + Qyz - Qxx - Qyy};
    double n2 = n[0] * n[0] + n[1] * n[1] + n[2] * n[2];
    if (!(n2 > 1e-24)) { n[0] = 0.0; n[1] = 0.0; n[2] = 1.0; n2 = 1.0; }
    const double r1 = fabs(Qxx) + fabs(Qxy) + fabs(Qxz);
    const double r2 = fabs(Qxy) + fabs(Qyy) + fabs(Qyz);
    const double r3 = fabs(Qxz) + fabs(Qyz) + fabs(Qzz);
    const double alpha = fmax(r1, fmax(r2, r3)) + 1e-12;
    const double ia = 1.0 / alpha;
    Sym3 m{fma(Qxx, ia, 1.0), Qxy * ia, Qxz * ia, fma(Qyy, ia, 1.0), Qyz * ia, fma(Qzz, ia, 1.0)};
    apply(m, n);
    const double v1 = n[0] * n[0] + n[1] * n[1] + n[2] * n[2];
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        m = square(m);
        apply(m, n);
    }
    const double v2 = n[0] * n[0] + n[1] * n[1] + n[2] * n[2];
    double inv = 1.0 / sqrt(v2);
    if (v2 < 1e-6 * n2 || v1 * (alpha * alpha) < 1e-26 * n2) {
        const double3 v = nematic_steps(Qxx, Qxy, Qxz, Qyy, Qyz, alpha);
        n[0] = v.x; n[1] = v.y; n[2] = v.z;
        inv = 1.0;
    }
    const double nx = n[0] * inv, ny = n[1] * inv, nz = n[2] * inv;
    const double lam = nx * (Qxx * nx + Qxy * ny + Qxz * nz) + ny * (Qxy * nx + Qyy * ny + Qyz * nz) +
                       nz * (Qxz * nx + Qyz * ny + Qzz * nz);
    Nematic r{1.5 * lam, nx, ny, nz};
    if (nz < -1e-10) { r.nx = -nx; r.ny = -ny; r.nz = -nz; }
    return r;
}

// Programmatic dependent launch (launch_pdl): a kernel is put on the SMs while its predecessor in the
// stream drains, sets itself up, and waits in pdl_wait until the predecessor's writes are complete;
// pdl_trigger then lets its own successor be put in place. Every access to data that an earlier
// kernel writes comes after pdl_wait, and is an ordinary load: the data changes during the kernel's
// lifetime, so neither __ldg nor a const __restrict__ pointer may be used for it (their read-only loads
// may be taken before the wait).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Warp and block reductions (fixed order: deterministic for a fixed launch shape).
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ unsigned long long warp_sum(unsigned long long v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
    return v;
}

}  // namespace ldg
