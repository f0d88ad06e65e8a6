// Periodic bulk LdG solver (KZM_bulk_ldg drop-in): device kernels and the kzm_* C ABI.
//
// Device layout: FP32 SoA, x fastest (the reference's flatten order, KZM_bulk_ldg.cu:161-169). Each
// row carries its periodic neighbours: columns x = -1 and x = Nx hold copies of x = Nx - 1 and x = 0,
// and each plane has the rows y = -1 and y = Ny, all written by whoever writes the site. A tile with
// its halo is then one rectangle of memory for any Nx and Ny, which a single TMA box fetches; z wraps
// by the plane index. One fused kernel per step: periodic 7-point Laplacian, bulk field, traceless
// projection, Euler, Philox Langevin noise, optional cap.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <limits>
#include <mutex>
#include <new>
#include <string>

#include "ldg_api_common.h"
#include "ldg_common.cuh"
#include "sm100_ptx.cuh"

using namespace ldg;

namespace {

constexpr double kPi = 3.14159265358979323846;

struct KzmConst {
    int Nx, Ny, Nz;
    int sy;          // row pitch (x fastest); arrays start at site (0, 0, 0), kPadX columns and one row in
    long long sz;    // plane pitch
    long long sc;    // component pitch
    float ix2, iy2, iz2;
    float lap_c;     // -2 (1/dx^2 + 1/dy^2 + 1/dz^2): centre weight of the Laplacian
    // both halves equal, for the packed arithmetic: -kappa/da^2, -kappa lap_c, -dt/gamma and the bulk
    // coefficients
    F2 mkx, mky, mkz, mk0, mmob;
    BulkC<F2> K;
    float A, B, C, kappa, mob_dt, qcap, sigma;
    uint32_t key0, key1;
    long long step;
};

// Columns before x = 0, and the multiple of floats of a row: 32 bytes, so that the rows a warp stores
// (x0 a multiple of 32) are whole sectors. Rows that cut sectors held the step back more than anything
// else: the same loads and stores without arithmetic take 164 us a step at 256^3 with rows starting
// 16 bytes into a sector and 110 us with whole sectors (a plain copy of the field takes 112 us).
constexpr int kPadX = 8;
constexpr int kHaloX = 4;  // columns of a TMA box before x0 (the box start stays on 16 bytes)

// Copies of a site on a face of the box in the periodic halo (five values at stride sc).
__device__ __forceinline__ void store_halo(float* __restrict__ out, const KzmConst& P, int x, int y, long long id,
                                           const float v[5]) {
    if (x == 0 || x == P.Nx - 1) {
        const long long o = id + (x == 0 ? P.Nx : -P.Nx);
#pragma unroll
        for (int m = 0; m < 5; ++m) out[m * P.sc + o] = v[m];
    }
    if (y == 0 || y == P.Ny - 1) {
        const long long o = id + (long long)(y == 0 ? P.Ny : -P.Ny) * P.sy;
#pragma unroll
        for (int m = 0; m < 5; ++m) out[m * P.sc + o] = v[m];
    }
}
// Writes a site and its halo copies.
__device__ __forceinline__ void store_site(float* __restrict__ out, const KzmConst& P, int x, int y, long long id,
                                           const float v[5]) {
#pragma unroll
    for (int m = 0; m < 5; ++m) out[m * P.sc + id] = v[m];
    store_halo(out, P, x, y, id, v);
}

// One periodic step: block (32, 8) over (x, y), grid z over planes (KZM_bulk_ldg.cu:351-469).
template <bool kNoise>
__global__ void __launch_bounds__(256) k_kzm_step(const float* __restrict__ q, float* __restrict__ out, KzmConst P) {
    const int x = blockIdx.x * 32 + threadIdx.x;
    const int y = blockIdx.y * 8 + threadIdx.y;
    const int z = blockIdx.z;
    if (x >= P.Nx || y >= P.Ny) return;
    const int xp = (x + 1 == P.Nx) ? 0 : x + 1, xm = (x == 0) ? P.Nx - 1 : x - 1;
    const int yp = (y + 1 == P.Ny) ? 0 : y + 1, ym = (y == 0) ? P.Ny - 1 : y - 1;
    const int zp = (z + 1 == P.Nz) ? 0 : z + 1, zm = (z == 0) ? P.Nz - 1 : z - 1;
    const long long row = (long long)z * P.sz + (long long)y * P.sy;
    const long long id = row + x;
    const long long oxp = row + xp, oxm = row + xm;
    const long long oyp = (long long)z * P.sz + (long long)yp * P.sy + x;
    const long long oym = (long long)z * P.sz + (long long)ym * P.sy + x;
    const long long ozp = (long long)zp * P.sz + (long long)y * P.sy + x;
    const long long ozm = (long long)zm * P.sz + (long long)y * P.sy + x;
    float c[5], lap[5];
#pragma unroll
    for (int m = 0; m < 5; ++m) {
        const float* b = q + m * P.sc;
        c[m] = __ldg(b + id);
        lap[m] = fmaf(P.ix2, __ldg(b + oxp) + __ldg(b + oxm),
                      fmaf(P.iy2, __ldg(b + oyp) + __ldg(b + oym),
                           fmaf(P.iz2, __ldg(b + ozp) + __ldg(b + ozm), P.lap_c * c[m])));
    }
    float h[6];
    bulk_field(c, P.A, P.B, P.C, h);
    h[0] -= P.kappa * lap[0];
    h[1] -= P.kappa * lap[3];
    h[2] += P.kappa * (lap[0] + lap[3]);
    h[3] -= P.kappa * lap[1];
    h[4] -= P.kappa * lap[2];
    h[5] -= P.kappa * lap[4];
    const float corr = (h[0] + h[1] + h[2]) * (1.0f / 3.0f);
    float u[5] = {c[0] - P.mob_dt * (h[0] - corr), c[1] - P.mob_dt * h[3], c[2] - P.mob_dt * h[4],
                  c[3] - P.mob_dt * (h[1] - corr), c[4] - P.mob_dt * h[5]};
    if (kNoise) {
        float g[5];
        const uint32_t cell = (uint32_t)(x + P.Nx * (y + P.Ny * z));
        normals5(cell, 0u, P.step, P.key0, P.key1, g);
#pragma unroll
        for (int m = 0; m < 5; ++m) u[m] += P.sigma * g[m];
    }
    if (P.qcap > 0.0f) {
        const float zz = -u[0] - u[3];
        const float tr = u[0] * u[0] + u[3] * u[3] + zz * zz + 2.0f * (u[1] * u[1] + u[2] * u[2] + u[4] * u[4]);
        const float qn = sqrtf(fmaxf(tr, 0.0f));
        if (qn > P.qcap && qn > 0.0f) {
            const float s = P.qcap / qn;
#pragma unroll
            for (int m = 0; m < 5; ++m) u[m] *= s;
        }
    }
    store_site(out, P, x, y, id, u);
}

// The step over (32 x 8) column tiles marching along z over a chunk of planes: 128 threads, each
// updating two sites (rows 2w and 2w + 1 of warp w) as one packed FP32 instruction stream (FFMA2 /
// FADD2 / FMUL2); the noise draw, the cap and the stores are per site. A plane of the tile with its
// halo (40 columns from x0 - 4, 10 rows, 5 components) is one TMA box in a ring of KNQ slots. A site's
// centre column is carried in registers (z - 1, z; z + 1 is read when its plane arrives), so a
// plane is read for its neighbours at its own step only, can be refilled right after it, and costs
// eight shared loads per component and pair instead of fourteen. The warps march independently: the
// last one done with a plane issues the load that reuses its slot.
// With noise it is bound by issue slots (234 instructions a site, 101 of them the draw, at 70 % issue
// efficiency); without, by HBM and the wait for planes (256^3: 4.4 TB/s of the 6.1 that the same loads and stores
// reach without arithmetic).
constexpr int KTX = 32, KTY = 8;
constexpr int KTHREADS = KTX * KTY / 2, KWARPS = KTHREADS / 32;
constexpr int KROW = KTX + 2 * kHaloX;        // floats per ring row: x0 - 4 .. x0 + 35
constexpr int KROWS = KTY + 2;
constexpr int KCSTR = KROW * KROWS;           // floats per component plane
constexpr int KSLOT = (5 * KCSTR + 31) / 32 * 32;  // floats per slot (128-byte aligned)
constexpr uint32_t KBYTES = 5 * KCSTR * 4;
constexpr int KNQ = 5;                        // slots: planes z and z + 1 in use, three in flight
constexpr int KCTAS = 5;                      // CTAs per SM
constexpr size_t kRingBytes = (size_t)KNQ * KSLOT * 4 + KNQ * 8 + KNQ * 4 + 4;

__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* tm, int c0, int c1, int c2, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
        "[%6];" ::"r"(sm100::smem_u32(dst)),
        "l"(tm), "r"(c0), "r"(c1), "r"(c2), "r"(0), "r"(sm100::smem_u32(bar))
        : "memory");
}

template <bool kNoise>
__global__ void __launch_bounds__(KTHREADS, KCTAS)
    k_kzm_step_ring(const __grid_constant__ CUtensorMap tm, float* __restrict__ out, KzmConst P, int planes,
                    int* __restrict__ err) {
    extern __shared__ __align__(128) unsigned char smem[];
    float* ring = reinterpret_cast<float*>(smem);
    uint64_t* bar = reinterpret_cast<uint64_t*>(ring + KNQ * KSLOT);
    unsigned* freed = reinterpret_cast<unsigned*>(bar + KNQ);
    int* s_abort = reinterpret_cast<int*>(freed + KNQ);
    const int tid = threadIdx.x, tx = tid & 31, w = tid >> 5;
    const int x0 = blockIdx.x * KTX, y0 = blockIdx.y * KTY, z0 = blockIdx.z * planes;
    const int z1 = min(z0 + planes, P.Nz);
    if (tid == 0) {
        for (int s = 0; s < KNQ; ++s) {
            sm100::mbar_init(&bar[s], 1);
            freed[s] = 0;
        }
        sm100::fence_mbar_init();
        *s_abort = 0;
    }
    __syncthreads();
    pdl_wait();
    pdl_trigger();
    // Plane p of this chunk (z0 - 1 <= p <= z1) in slot (p - z0 + 1) % KNQ.
    auto issue = [&](int p, int sl) {
        if (p > z1) return;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        sm100::mbar_expect_tx(&bar[sl], KBYTES);
        const int zw = p < 0 ? p + P.Nz : (p >= P.Nz ? p - P.Nz : p);
        tma_load_4d(ring + sl * KSLOT, &tm, x0 + kPadX - kHaloX, y0, zw, &bar[sl]);
    };
    if (tid == 0)
        for (int s = 0; s < KNQ; ++s) issue(z0 - 1 + s, s);
    bool ok = true;
    uint32_t par = 0;  // parity of the next wait on every slot
    auto wait_slot = [&](int sl) {
        const uint32_t ph = (par >> sl) & 1u;
        par ^= 1u << sl;
        if (sm100::mbar_try_wait(&bar[sl], ph)) return;
        const long long t0 = clock64();
        while (!sm100::mbar_try_wait(&bar[sl], ph))
            if (*(volatile int*)s_abort || clock64() - t0 > 4000000000ll) {  // about 2 s
                atomicExch(err, LDG_ERR_TIMEOUT);
                *(volatile int*)s_abort = 1;
                ok = false;
                return;
            }
    };
    // This warp is done with plane p: the last warp refills its slot with plane p + KNQ.
    auto done = [&](int p, int sl) {
        __syncwarp();
        if (tx == 0) {
            unsigned old;
            asm volatile("atom.acq_rel.cta.shared::cta.add.u32 %0, [%1], 1;"
                         : "=r"(old)
                         : "r"(sm100::smem_u32(&freed[sl]))
                         : "memory");
            if (old % (unsigned)KWARPS == (unsigned)KWARPS - 1u) issue(p + KNQ, sl);
        }
    };
    const int x = x0 + tx, y = y0 + 2 * w;
    const bool v0 = x < P.Nx && y < P.Ny, v1 = x < P.Nx && y + 1 < P.Ny;
    const int s_c = (2 * w + 1) * KROW + tx + kHaloX;
    const bool edge = x == 0 || x == P.Nx - 1 || y == 0 || y >= P.Ny - 2;
    float* o = out + (long long)z0 * P.sz + (long long)y * P.sy + x;
    uint32_t cell = (uint32_t)x + (uint32_t)P.Nx * ((uint32_t)y + (uint32_t)P.Ny * (uint32_t)z0);
    const uint32_t cells_z = (uint32_t)P.Nx * (uint32_t)P.Ny;
    F2 cm[5], c[5];
    wait_slot(0);
#pragma unroll
    for (int m = 0; m < 5; ++m) cm[m] = mk2(ring[m * KCSTR + s_c], ring[m * KCSTR + s_c + KROW]);
    done(z0 - 1, 0);
    wait_slot(1);
#pragma unroll
    for (int m = 0; m < 5; ++m) c[m] = mk2(ring[KSLOT + m * KCSTR + s_c], ring[KSLOT + m * KCSTR + s_c + KROW]);
    int sl = 1, sn = 2 % KNQ;  // slots of planes z and z + 1
    int waited = z0 + 1;       // planes below this one were waited for
    for (int z = z0; z < z1; ++z, o += P.sz, cell += cells_z) {
        wait_slot(sn);
        waited = z + 2;
        if (!__all_sync(0xffffffffu, ok)) break;  // the whole warp stops or none of it
        const float* pc = ring + sl * KSLOT + s_c;
        const float* pn = ring + sn * KSLOT + s_c;
        F2 h[5], u[5];
        bulk_field5<F2>(c, P.K, h);
#pragma unroll
        for (int m = 0; m < 5; ++m) {
            const float* s = pc + m * KCSTR;
            const F2 cp = mk2(pn[m * KCSTR], pn[m * KCSTR + KROW]);
            const F2 sx = mk2(s[1], s[KROW + 1]) + mk2(s[-1], s[KROW - 1]);
            // row y + 1 of the first site is the second site, and the other way round
            const F2 sy = mk2(c[m].v.y + s[-KROW], s[2 * KROW] + c[m].v.x);
            const F2 e = vfma(P.mkx, sx, vfma(P.mky, sy, vfma(P.mkz, cp + cm[m], vfma(P.mk0, c[m], h[m]))));
            u[m] = vfma(P.mmob, e, c[m]);
            cm[m] = c[m];
            c[m] = cp;
        }
        done(z, sl);
        if (v0) {
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                if (r && !v1) continue;
                float v[5];
#pragma unroll
                for (int m = 0; m < 5; ++m) v[m] = r ? u[m].v.y : u[m].v.x;
                if (kNoise) {
                    float g[5];
                    normals5(cell + (r ? (uint32_t)P.Nx : 0u), 0u, P.step, P.key0, P.key1, g);
#pragma unroll
                    for (int m = 0; m < 5; ++m) v[m] = fmaf(P.sigma, g[m], v[m]);
                }
                if (P.qcap > 0.0f) cap_norm(P.qcap, v);
                float* d = r ? o + P.sy : o;
#pragma unroll
                for (int m = 0; m < 5; ++m) d[m * P.sc] = v[m];
                if (edge) store_halo(d, P, x, y + r, 0, v);
            }
        }
        sl = sn;
        sn = sn + 1 == KNQ ? 0 : sn + 1;
    }
    if (!ok)  // after an abort: copies that may be in flight, for a bounded time
        for (int p = waited; p <= z1; ++p) {
            const int s = (p - z0 + 1) % KNQ;
            const long long t0 = clock64();
            while (!sm100::mbar_try_wait(&bar[s], (par >> s) & 1u) && clock64() - t0 < 40000000ll) {
            }
            par ^= 1u << s;
        }
}

__global__ void k_kzm_from_aos(const double* __restrict__ aos, float* __restrict__ a, KzmConst P) {
    const long long n = (long long)P.Nx * P.Ny * P.Nz;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        const int x = (int)(t % P.Nx);
        const long long r = t / P.Nx;
        const int y = (int)(r % P.Ny);
        const int z = (int)(r / P.Ny);
        const long long id = (long long)z * P.sz + (long long)y * P.sy + x;
        float v[5];
#pragma unroll
        for (int m = 0; m < 5; ++m) v[m] = (float)aos[5 * t + m];
        store_site(a, P, x, y, id, v);
    }
}

__global__ void k_kzm_to_aos(const float* __restrict__ a, double* __restrict__ aos, KzmConst P) {
    const long long n = (long long)P.Nx * P.Ny * P.Nz;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        const int x = (int)(t % P.Nx);
        const long long r = t / P.Nx;
        const int y = (int)(r % P.Ny);
        const int z = (int)(r / P.Ny);
        const long long id = (long long)z * P.sz + (long long)y * P.sy + x;
#pragma unroll
        for (int m = 0; m < 5; ++m) aos[5 * t + m] = (double)a[m * P.sc + id];
    }
}

struct KzmPartial {
    double bulk, elastic, qint, gint, S_sum, S_max, line;
    unsigned long long used, defects;
};

constexpr int kThreads = 256;
constexpr int kBlocks = 148 * 8;

template <class T>
__device__ __forceinline__ T bsum(T v, T* sh) {
    v = warp_sum(v);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) sh[w] = v;
    __syncthreads();
    T r = 0;
    if (threadIdx.x == 0)
        for (int x = 0; x < (int)(blockDim.x >> 5); ++x) r += sh[x];
    return r;
}

__device__ __forceinline__ double bmax(double v, double* sh) {
    v = warp_max(v);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) sh[w] = v;
    __syncthreads();
    double r = 0.0;
    if (threadIdx.x == 0)
        for (int x = 0; x < (int)(blockDim.x >> 5); ++x) r = fmax(r, sh[x]);
    return r;
}

struct KzmObsConst {
    KzmConst P;
    double A, B, C, kappa, cv, ix, iy, iz;
};

// Pass 1 (KZM_bulk_ldg.cu:564-632): bulk and forward-difference elastic energy, |Q|^2 and
// |grad Q|^2 integrals, nematic (S, n) per site into an FP64 scratch field. kAos: the field is the
// caller's own (reference layout, AoS FP64, x fastest), else the solver's FP32 arrays. A warp takes a
// row of sites at a time.
template <bool kAos, class T>
__global__ void __launch_bounds__(kThreads) k_kzm_obs_sites(const T* __restrict__ q, KzmObsConst O,
                                                            double4* __restrict__ nf, KzmPartial* __restrict__ part) {
    const KzmConst& P = O.P;
    KzmPartial a{};
    const int lane = threadIdx.x & 31;
    const long long rows = (long long)P.Ny * P.Nz, warps = (long long)gridDim.x * (kThreads / 32);
    for (long long r = (long long)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5); r < rows; r += warps) {
        const int z = (int)(r / P.Ny), y = (int)(r - (long long)z * P.Ny);
        const int yp = y + 1 == P.Ny ? 0 : y + 1, zp = z + 1 == P.Nz ? 0 : z + 1;
        auto row = [&](int yy, int zz) {
            return kAos ? q + 5 * (long long)P.Nx * (yy + (long long)P.Ny * zz) : q + (long long)zz * P.sz + (long long)yy * P.sy;
        };
        const T *q0 = row(y, z), *qy = row(yp, z), *qz = row(y, zp);
        const int step = kAos ? 5 : 1;
        const long long comp = kAos ? 1 : P.sc;
        for (int x = lane; x < P.Nx; x += 32) {
            const long long ox = (long long)step * x, op = (long long)step * (x + 1 == P.Nx ? 0 : x + 1);
            double c[5], d[6][3];
#pragma unroll
            for (int m = 0; m < 5; ++m) {
                c[m] = (double)q0[m * comp + ox];
                d[m][0] = ((double)q0[m * comp + op] - c[m]) * O.ix;
                d[m][1] = ((double)qy[m * comp + ox] - c[m]) * O.iy;
                d[m][2] = ((double)qz[m * comp + ox] - c[m]) * O.iz;
            }
#pragma unroll
            for (int w = 0; w < 3; ++w) d[5][w] = -(d[0][w] + d[3][w]);
            const double Qxx = c[0], Qxy = c[1], Qxz = c[2], Qyy = c[3], Qyz = c[4], Qzz = -Qxx - Qyy;
            const double q2xx = Qxx * Qxx + Qxy * Qxy + Qxz * Qxz;
            const double q2xy = Qxx * Qxy + Qxy * Qyy + Qxz * Qyz;
            const double q2xz = Qxx * Qxz + Qxy * Qyz + Qxz * Qzz;
            const double q2yy = Qxy * Qxy + Qyy * Qyy + Qyz * Qyz;
            const double q2yz = Qxy * Qxz + Qyy * Qyz + Qyz * Qzz;
            const double q2zz = Qxz * Qxz + Qyz * Qyz + Qzz * Qzz;
            const double trQ2 = Qxx * Qxx + Qyy * Qyy + Qzz * Qzz + 2.0 * (Qxy * Qxy + Qxz * Qxz + Qyz * Qyz);
            const double trQ3 = Qxx * q2xx + Qxy * q2xy + Qxz * q2xz + Qxy * q2xy + Qyy * q2yy + Qyz * q2yz +
                                Qxz * q2xz + Qyz * q2yz + Qzz * q2zz;
            a.bulk += ((O.A / 2.0) * trQ2 - (O.B / 3.0) * trQ3 + (O.C / 4.0) * trQ2 * trQ2) * O.cv;
            double g2 = 0.0;
#pragma unroll
            for (int m = 0; m < 6; ++m) {
                const double s = d[m][0] * d[m][0] + d[m][1] * d[m][1] + d[m][2] * d[m][2];
                g2 += (m == 1 || m == 2 || m == 4) ? 2.0 * s : s;
            }
            a.gint += g2 * O.cv;
            a.qint += trQ2 * O.cv;
            const Nematic f = nematic64(c, 1e-12, Nematic{0.0, 1.0, 0.0, 0.0});
            nf[r * P.Nx + x] = make_double4(f.S, f.nx, f.ny, f.nz);
            a.S_sum += f.S;
            a.S_max = fmax(a.S_max, f.S);
        }
    }
    a.elastic = 0.5 * O.kappa * a.gint;
    __shared__ double shd[kThreads / 32];
    KzmPartial res{};
    res.bulk = bsum(a.bulk, shd);
    res.elastic = bsum(a.elastic, shd);
    res.qint = bsum(a.qint, shd);
    res.gint = bsum(a.gint, shd);
    res.S_sum = bsum(a.S_sum, shd);
    res.S_max = bmax(a.S_max, shd);
    if (threadIdx.x == 0) part[blockIdx.x] = res;
}

__device__ __forceinline__ double wrap_pi_loop(double d) {
    // wrap_to_pi of KZM_bulk_ldg.cu:471-479.
    while (d <= -kPi) d += 2.0 * kPi;
    while (d > kPi) d -= 2.0 * kPi;
    return d;
}

__device__ __forceinline__ bool project_plane(const double4& f, int plane, double& u, double& v) {
    // project_to_plane (KZM_bulk_ldg.cu:481-499).
    if (plane == 0) { u = f.y; v = f.z; }
    else if (plane == 1) { u = f.z; v = f.w; }
    else { u = f.y; v = f.w; }
    const double nrm = sqrt(u * u + v * v);
    if (!(nrm > 1e-8)) return false;
    u /= nrm;
    v /= nrm;
    return true;
}

// plaquette_charge (KZM_bulk_ldg.cu:501-541): 0 unused, 1 used, 2 defect.
__device__ __forceinline__ int plaquette(const double4& a, const double4& b, const double4& c, const double4& d,
                                         int plane, double thr, double cut) {
    if (!(isfinite(a.x) && isfinite(b.x) && isfinite(c.x) && isfinite(d.x))) return 0;
    if (!(a.x > thr && b.x > thr && c.x > thr && d.x > thr)) return 0;
    double ua, va, ub, vb, uc, vc, ud, vd;
    if (!project_plane(a, plane, ua, va) || !project_plane(b, plane, ub, vb) || !project_plane(c, plane, uc, vc) ||
        !project_plane(d, plane, ud, vd))
        return 0;
    const double pa = 2.0 * atan2(va, ua), pb = 2.0 * atan2(vb, ub), pc = 2.0 * atan2(vc, uc), pd = 2.0 * atan2(vd, ud);
    const double dsum = wrap_pi_loop(pb - pa) + wrap_pi_loop(pc - pb) + wrap_pi_loop(pd - pc) + wrap_pi_loop(pa - pd);
    const double s = 0.5 * (dsum / (2.0 * kPi));
    return (fabs(s) > cut) ? 2 : 1;
}

// The same from sign tests. The doubled angle of a projected director (u, v) is that of
// D = (u^2 - v^2, 2 u v); around a plaquette the wrapped angle differences add up to 2 pi m with a whole
// number m, and m counts the edges that pass the angle pi: an edge from the upper half plane (angle
// in [0, pi]) to the lower one passes it upwards where D_a x D_b > 0, one from the lower to the upper
// downwards where D_a x D_b < 0. So no angle, root or division is needed, and |m| / 2 > cut decides. An edge whose directors
// are parallel or antiparallel to 1e-9, where rounding of the angles would decide, and a cut within
// 1e-9 of 0, 1/2 or 1 take the angles themselves (plaquette above).
struct Doubled {
    double x, y, r;  // D and its length u^2 + v^2
};
__device__ __forceinline__ Doubled doubled(double u, double v) {
    const double uu = u * u, vv = v * v;
    return Doubled{uu - vv, 2.0 * u * v, uu + vv};
}
// Signed passage of the angle pi from a to b, or 2 where the signs do not decide.
__device__ __forceinline__ int passage(const Doubled& a, const Doubled& b) {
    const double cr = a.x * b.y - a.y * b.x;
    const bool ha = a.y >= 0.0, hb = b.y >= 0.0;
    const bool flat = !(fabs(cr) > 1e-9 * (a.r * b.r));
    if (ha == hb && !(flat && !(a.x * b.x + a.y * b.y > 0.0))) return 0;
    if (flat) return 2;
    return ha ? (cr > 0.0 ? 1 : 0) : (cr < 0.0 ? -1 : 0);
}
__device__ __forceinline__ int plaquette_signs(const double4& a, const double4& b, const double4& c, const double4& d,
                                               int plane, double thr, double cut, bool plain_cut) {
    if (!(isfinite(a.x) && isfinite(b.x) && isfinite(c.x) && isfinite(d.x))) return 0;
    if (!(a.x > thr && b.x > thr && c.x > thr && d.x > thr)) return 0;
    auto proj = [plane](const double4& f) {
        return plane == 0 ? doubled(f.y, f.z) : (plane == 1 ? doubled(f.z, f.w) : doubled(f.y, f.w));
    };
    const Doubled A = proj(a), B = proj(b), C = proj(c), E = proj(d);
    const double lo = fmin(fmin(A.r, B.r), fmin(C.r, E.r));
    if (plain_cut && lo > 1.001e-16) {
        const int k0 = passage(A, B), k1 = passage(B, C), k2 = passage(C, E), k3 = passage(E, A);
        if (k0 != 2 && k1 != 2 && k2 != 2 && k3 != 2) return 0.5 * abs(k0 + k1 + k2 + k3) > cut ? 2 : 1;
    }
    return plaquette(a, b, c, d, plane, thr, cut);
}

// Pass 2 (KZM_bulk_ldg.cu:634-689): three plaquette orientations per site, line length. A warp takes a
// row of sites at a time.
__global__ void __launch_bounds__(kThreads) k_kzm_obs_plaq(const double4* __restrict__ nf, KzmObsConst O, double thr,
                                                           double cut, double dx, double dy, double dz,
                                                           KzmPartial* __restrict__ part) {
    const KzmConst& P = O.P;
    KzmPartial a{};
    unsigned used = 0, n0 = 0, n1 = 0, n2 = 0;
    const bool plain_cut = cut > 1e-9 && fabs(cut - 0.5) > 1e-9 && fabs(cut - 1.0) > 1e-9;
    const int lane = threadIdx.x & 31;
    const long long rows = (long long)P.Ny * P.Nz, warps = (long long)gridDim.x * (kThreads / 32);
    for (long long r = (long long)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5); r < rows; r += warps) {
        const int z = (int)(r / P.Ny), y = (int)(r - (long long)z * P.Ny);
        const int yp = y + 1 == P.Ny ? 0 : y + 1, zp = z + 1 == P.Nz ? 0 : z + 1;
        auto row = [&](int yy, int zz) { return nf + (long long)P.Nx * (yy + (long long)P.Ny * zz); };
        const double4 *r00 = row(y, z), *r10 = row(yp, z), *r01 = row(y, zp), *r11 = row(yp, zp);
        for (int x = lane; x < P.Nx; x += 32) {
            const int xp = x + 1 == P.Nx ? 0 : x + 1;
            const double4 f000 = r00[x], f100 = r00[xp], f010 = r10[x], f001 = r01[x];
            const double4 f110 = r10[xp], f101 = r01[xp], f011 = r11[x];
            int res = plaquette_signs(f000, f100, f110, f010, 0, thr, cut, plain_cut);
            used += res != 0;
            n0 += res == 2;
            res = plaquette_signs(f000, f010, f011, f001, 1, thr, cut, plain_cut);
            used += res != 0;
            n1 += res == 2;
            res = plaquette_signs(f000, f100, f101, f001, 2, thr, cut, plain_cut);
            used += res != 0;
            n2 += res == 2;
        }
    }
    a.used = used;
    a.defects = (unsigned long long)n0 + n1 + n2;
    a.line = n0 * dz + n1 * dx + n2 * dy;
    __shared__ double shd[kThreads / 32];
    __shared__ unsigned long long shu[kThreads / 32];
    KzmPartial res{};
    res.line = bsum(a.line, shd);
    res.used = bsum(a.used, shu);
    res.defects = bsum(a.defects, shu);
    if (threadIdx.x == 0) {
        part[blockIdx.x].line = res.line;
        part[blockIdx.x].used = res.used;
        part[blockIdx.x].defects = res.defects;
    }
}

__global__ void __launch_bounds__(kThreads) k_kzm_obs_final(const KzmPartial* __restrict__ part, int n,
                                                            KzmPartial* __restrict__ out) {
    KzmPartial a{};
    for (int b = threadIdx.x; b < n; b += blockDim.x) {
        const KzmPartial& p = part[b];
        a.bulk += p.bulk; a.elastic += p.elastic; a.qint += p.qint; a.gint += p.gint; a.S_sum += p.S_sum;
        a.S_max = fmax(a.S_max, p.S_max); a.line += p.line; a.used += p.used; a.defects += p.defects;
    }
    __shared__ double shd[kThreads / 32];
    __shared__ unsigned long long shu[kThreads / 32];
    KzmPartial r{};
    r.bulk = bsum(a.bulk, shd);
    r.elastic = bsum(a.elastic, shd);
    r.qint = bsum(a.qint, shd);
    r.gint = bsum(a.gint, shd);
    r.S_sum = bsum(a.S_sum, shd);
    r.S_max = bmax(a.S_max, shd);
    r.line = bsum(a.line, shd);
    r.used = bsum(a.used, shu);
    r.defects = bsum(a.defects, shu);
    if (threadIdx.x == 0) *out = r;
}

int alloc_or_fail(void** p, size_t bytes) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        set_error(std::string("cudaMalloc(") + std::to_string(bytes) + "): " + cudaGetErrorString(e));
        return LDG_ERR_NOMEM;
    }
    return LDG_OK;
}

int kzm_encode(CUtensorMap* tm, const float* alloc, const KzmConst& P) {
    static void* const fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        const bool got = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) == cudaSuccess &&
                         q == cudaDriverEntryPointSuccess;
        return got ? f : nullptr;
    }();
    LDG_REQUIRE(fn, LDG_ERR_CUDA, "cuTensorMapEncodeTiled entry point unavailable");
    cuuint64_t dims[4] = {(cuuint64_t)P.sy, (cuuint64_t)P.Ny + 2, (cuuint64_t)P.Nz, 5};
    cuuint64_t strides[3] = {(cuuint64_t)P.sy * 4, (cuuint64_t)P.sz * 4, (cuuint64_t)P.sc * 4};
    cuuint32_t box[4] = {KROW, KROWS, 1, 5}, estr[4] = {1, 1, 1, 1};
    const CUresult r = ((PFN_cuTensorMapEncodeTiled_v12000)fn)(
        tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float*>(alloc), dims, strides, box, estr,
        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("kzm: cuTensorMapEncodeTiled failed: " + std::to_string((int)r));
        return LDG_ERR_CUDA;
    }
    return LDG_OK;
}

// Planes per CTA: the chunk length with the least estimated time. A CTA takes 0.95 us and 0.57 + 0.265 m
// us per plane (with noise) where m CTAs share its SM; full waves of KCTAS per SM, then the rest.
// Measured, us a step with chunks of 2 / 4 / 8 / 16 / 32 planes and of the length chosen (32 planes in every grid before,
// with the kernel of then: 28.7, 40, 208 with noise, 20.5, 29.5, 176 without):
//     64^3  with noise   7.1   6.5   9.2  16.4  30.9   7.1     without   5.7   5.0   7.0  12.2  22.5   5.7
//     128^3             30.9  28.9  29.1  35.5  37.4  28.2              27.1  24.2  24.6  29.3  26.4  25.0
//     256^3            214   192   180   182   188   187               179   156   146   146   151   152
// LDG_KZM_PLANES forces a length.
int kzm_planes(const KzmConst& P) {
    const int lo = (P.Nz + 65534) / 65535;  // the launch grid's z extent is limited
    if (const char* e = getenv("LDG_KZM_PLANES")) return std::min(P.Nz, std::max(lo, atoi(e)));
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const long long tiles = (long long)((P.Nx + KTX - 1) / KTX) * ((P.Ny + KTY - 1) / KTY);
    const long long slots = (long long)sms * KCTAS;
    auto cta = [](int c, int m) { return 0.95 + c * (0.57 + 0.265 * m); };
    int best = lo;
    double best_t = std::numeric_limits<double>::infinity();
    for (int c = lo; c <= std::min(P.Nz, 32); ++c) {
        const long long n = tiles * ((P.Nz + c - 1) / c), rest = n % slots;
        const double t = (double)(n / slots) * cta(c, KCTAS) + (rest ? cta(c, (int)((rest + sms - 1) / sms)) : 0.0);
        if (t < best_t) {
            best_t = t;
            best = c;
        }
    }
    return best;
}

}  // namespace

struct kzm_handle {
    kzm_params p{};
    KzmConst base{};
    long long n = 0;
    float* alloc[2] = {nullptr, nullptr};  // the fields' memory, halo included
    float* q[2] = {nullptr, nullptr};      // site (0, 0, 0) of component 0
    CUtensorMap tmap[2];
    int* err = nullptr;                    // device error word of the bounded waits (after the partials)
    int planes = 1;                        // planes per CTA of the step kernel
    double* stage = nullptr;
    double4* nf = nullptr;
    KzmPartial* part = nullptr;            // kBlocks + 1 partials, then the error word
    int cur = 0;
    bool uploaded = false;
    cudaStream_t stream = nullptr;
    long long launches = 0;
    int device = -1;  // the GPU the handle was created on
};

extern "C" {

int kzm_create(const kzm_params* params, kzm_handle** out) {
    clear_error();
    LDG_REQUIRE(params && out, LDG_ERR_ARG, "kzm_create: null argument");
    const kzm_params& p = *params;
    // Validation of KZM_bulk_ldg.cu:824-841.
    LDG_REQUIRE(p.Nx > 1 && p.Ny > 1 && p.Nz > 1, LDG_ERR_ARG,
                "Nx, Ny, and Nz must all be greater than 1 for the periodic bulk LdG branch");
    LDG_REQUIRE((long long)p.Nx * p.Ny * p.Nz < (1LL << 32), LDG_ERR_ARG, "kzm_create: grid exceeds 2^32 sites");
    LDG_REQUIRE(p.dx > 0 && p.dy > 0 && p.dz > 0, LDG_ERR_ARG, "dx, dy, and dz must be positive");
    LDG_REQUIRE(p.gamma > 0, LDG_ERR_ARG, "gamma must be positive");
    LDG_REQUIRE(p.kappa >= 0, LDG_ERR_ARG, "kappa must be non-negative");
    kzm_handle* h = new (std::nothrow) kzm_handle();
    LDG_REQUIRE(h, LDG_ERR_NOMEM, "kzm_create: host allocation failed");
    h->p = p;
    cudaGetDevice(&h->device);
    KzmConst& P = h->base;
    P.Nx = p.Nx; P.Ny = p.Ny; P.Nz = p.Nz;
    P.sy = kPadX + ((p.Nx + 1 + 7) & ~7);
    P.sz = (long long)(p.Ny + 2) * P.sy;
    P.sc = (long long)p.Nz * P.sz;
    P.ix2 = (float)(1.0 / (p.dx * p.dx)); P.iy2 = (float)(1.0 / (p.dy * p.dy)); P.iz2 = (float)(1.0 / (p.dz * p.dz));
    P.lap_c = (float)(-2.0 * (1.0 / (p.dx * p.dx) + 1.0 / (p.dy * p.dy) + 1.0 / (p.dz * p.dz)));
    P.kappa = (float)p.kappa;
    auto both = [](double v) { return F2{make_float2((float)v, (float)v)}; };
    P.mkx = both(-p.kappa / (p.dx * p.dx)); P.mky = both(-p.kappa / (p.dy * p.dy)); P.mkz = both(-p.kappa / (p.dz * p.dz));
    P.mk0 = both(2.0 * p.kappa * (1.0 / (p.dx * p.dx) + 1.0 / (p.dy * p.dy) + 1.0 / (p.dz * p.dz)));
    P.qcap = (float)p.q_norm_cap;
    h->n = (long long)p.Nx * p.Ny * p.Nz;
    int rc;
    const size_t fb = (size_t)P.sc * 5 * sizeof(float);
    if ((rc = alloc_or_fail((void**)&h->alloc[0], fb)) || (rc = alloc_or_fail((void**)&h->alloc[1], fb)) ||
        (rc = alloc_or_fail((void**)&h->part, (kBlocks + 2) * sizeof(KzmPartial)))) {
        kzm_destroy(h);
        return rc;
    }
    cudaError_t e = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking);
    h->err = reinterpret_cast<int*>(h->part + kBlocks + 1);
    for (int b = 0; b < 2; ++b) {
        // on the handle's stream, as all later work: nothing orders the default stream against it
        if (e == cudaSuccess) e = cudaMemsetAsync(h->alloc[b], 0, fb, h->stream);
        h->q[b] = h->alloc[b] + P.sy + kPadX;
    }
    if (e == cudaSuccess) e = cudaMemsetAsync(h->err, 0, sizeof(int), h->stream);
    if (e != cudaSuccess) {
        set_error(std::string("kzm_create: ") + cudaGetErrorString(e));
        kzm_destroy(h);
        return LDG_ERR_CUDA;
    }
    for (int b = 0; b < 2; ++b)
        if ((rc = kzm_encode(&h->tmap[b], h->alloc[b], P))) {
            kzm_destroy(h);
            return rc;
        }
    h->planes = kzm_planes(P);
    *out = h;
    return LDG_OK;
}

// Reads and clears the device error word (LDG_OK when no bounded wait gave up); synchronises.
static int kzm_check(kzm_handle* h) {
    int e = 0;
    LDG_CUDA(cudaMemcpyAsync(&e, h->err, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
    LDG_CUDA(cudaStreamSynchronize(h->stream));
    if (e == 0) return LDG_OK;
    LDG_CUDA(cudaMemsetAsync(h->err, 0, sizeof(int), h->stream));
    set_error("periodic step: a bounded shared-memory pipeline wait gave up");
    return LDG_ERR_TIMEOUT;
}

static int kzm_stage(kzm_handle* h) {
    if (h->stage) return LDG_OK;
    return alloc_or_fail((void**)&h->stage, (size_t)h->n * 5 * sizeof(double));
}

int kzm_upload(kzm_handle* h, const double* q) {
    clear_error();
    LDG_REQUIRE(h && q, LDG_ERR_ARG, "kzm_upload: null argument");
    DeviceGuard device_guard(h->device);
    int rc = kzm_stage(h);
    if (rc) return rc;
    LDG_CUDA(cudaMemcpyAsync(h->stage, q, (size_t)h->n * 5 * sizeof(double), cudaMemcpyHostToDevice, h->stream));
    h->cur = 0;
    const int blocks = (int)std::min<long long>((h->n + 255) / 256, 148 * 16);
    k_kzm_from_aos<<<blocks, 256, 0, h->stream>>>(h->stage, h->q[0], h->base);
    h->launches++;
    LDG_LAUNCHED("k_kzm_from_aos");
    LDG_CUDA(cudaStreamSynchronize(h->stream));
    h->uploaded = true;
    return LDG_OK;
}

int kzm_download(kzm_handle* h, double* q) {
    clear_error();
    LDG_REQUIRE(h && q, LDG_ERR_ARG, "kzm_download: null argument");
    DeviceGuard device_guard(h->device);
    int rc = kzm_stage(h);
    if (rc) return rc;
    const int blocks = (int)std::min<long long>((h->n + 255) / 256, 148 * 16);
    k_kzm_to_aos<<<blocks, 256, 0, h->stream>>>(h->q[h->cur], h->stage, h->base);
    h->launches++;
    LDG_LAUNCHED("k_kzm_to_aos");
    LDG_CUDA(cudaMemcpyAsync(q, h->stage, (size_t)h->n * 5 * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    return kzm_check(h);
}

int kzm_step(kzm_handle* h, int n_steps, const kzm_step_args* a) {
    clear_error();
    LDG_REQUIRE(h && a, LDG_ERR_ARG, "kzm_step: null argument");
    DeviceGuard device_guard(h->device);
    LDG_REQUIRE(n_steps >= 0, LDG_ERR_ARG, "kzm_step: n_steps must be >= 0");
    LDG_REQUIRE(h->uploaded, LDG_ERR_STATE, "kzm_step: no field uploaded");
    LDG_REQUIRE(a->dt > 0.0, LDG_ERR_ARG, "dt must be positive");
    KzmConst P = h->base;
    P.A = (float)a->A; P.B = (float)a->B; P.C = (float)a->C;
    P.mob_dt = (float)((1.0 / h->p.gamma) * a->dt);
    auto both = [](float v) { return F2{make_float2(v, v)}; };
    P.mmob = both(-P.mob_dt);
    P.K = BulkC<F2>{both(P.A), both(2.0f * P.C), both(-1.0f / 3.0f * P.B), both(P.B), both(-P.B)};
    P.sigma = (float)a->noise_sigma;
    P.key0 = (uint32_t)a->seed;
    P.key1 = (uint32_t)(a->seed >> 32);
    // LDG_KZM_KERNEL=direct selects the one-thread-per-site kernel (comparisons).
    const char* ksel = getenv("LDG_KZM_KERNEL");
    const bool direct = ksel && std::strcmp(ksel, "direct") == 0;
    const bool noise = a->noise_sigma > 0.0;
    const dim3 blk(32, 8, 1), grd((P.Nx + 31) / 32, (P.Ny + 7) / 8, P.Nz);
    const dim3 tgrd((P.Nx + KTX - 1) / KTX, (P.Ny + KTY - 1) / KTY, (P.Nz + h->planes - 1) / h->planes);
    for (int s = 0; s < n_steps; ++s) {
        P.step = a->step_index + s;
        const float* in = h->q[h->cur];
        float* outb = h->q[1 - h->cur];
        if (!direct) {
            LDG_CUDA(launch_pdl(noise ? k_kzm_step_ring<true> : k_kzm_step_ring<false>, tgrd, KTHREADS, kRingBytes,
                                h->stream, h->tmap[h->cur], outb, P, h->planes, h->err));
        } else if (noise) {
            k_kzm_step<true><<<grd, blk, 0, h->stream>>>(in, outb, P);
        } else {
            k_kzm_step<false><<<grd, blk, 0, h->stream>>>(in, outb, P);
        }
        h->launches++;
        LDG_LAUNCHED("k_kzm_step");
        h->cur = 1 - h->cur;
    }
    return LDG_OK;
}

int kzm_observe(kzm_handle* h, double A, double B, double C, kzm_observables* o) {
    clear_error();
    LDG_REQUIRE(h && o, LDG_ERR_ARG, "kzm_observe: null argument");
    DeviceGuard device_guard(h->device);
    if (!h->nf) {
        int rc = alloc_or_fail((void**)&h->nf, (size_t)h->n * sizeof(double4));
        if (rc) return rc;
    }
    const kzm_params& p = h->p;
    KzmObsConst O{};
    O.P = h->base;
    O.A = A; O.B = B; O.C = C; O.kappa = p.kappa;
    O.cv = p.dx * p.dy * p.dz;
    O.ix = 1.0 / p.dx; O.iy = 1.0 / p.dy; O.iz = 1.0 / p.dz;
    k_kzm_obs_sites<false><<<kBlocks, kThreads, 0, h->stream>>>(h->q[h->cur], O, h->nf, h->part);
    k_kzm_obs_plaq<<<kBlocks, kThreads, 0, h->stream>>>(h->nf, O, p.defects_S_threshold, p.defects_charge_cutoff, p.dx,
                                                       p.dy, p.dz, h->part);
    k_kzm_obs_final<<<1, kThreads, 0, h->stream>>>(h->part, kBlocks, h->part + kBlocks);
    h->launches += 3;
    LDG_LAUNCHED("kzm observables");
    KzmPartial R{};
    LDG_CUDA(cudaMemcpyAsync(&R, h->part + kBlocks, sizeof(R), cudaMemcpyDeviceToHost, h->stream));
    if (int rc = kzm_check(h)) return rc;
    const double tv = O.cv * (double)p.Nx * (double)p.Ny * (double)p.Nz;
    const double nan = std::numeric_limits<double>::quiet_NaN();
    o->bulk = R.bulk / tv;
    o->elastic = R.elastic / tv;
    o->total = o->bulk + o->elastic;
    o->avg_S = R.S_sum / (double)h->n;
    o->max_S = R.S_max;
    o->defect_plaquettes_used = (long long)R.used;
    o->nonzero_defect_plaquettes = (long long)R.defects;
    o->defect_density_per_plaquette = R.used > 0 ? (double)R.defects / (double)R.used : nan;
    o->defect_line_density = tv > 0.0 ? R.line / tv : nan;
    o->xi_grad_proxy = (R.gint > 0.0 && R.qint > 0.0) ? std::sqrt(R.qint / R.gint) : nan;
    return LDG_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------------------
// No-allocation observables. Scratch lives in file-scope device arrays of this library:
// the per-site nematic field of at most KZM_NOALLOC_MAX_SITES sites (16 MiB) and one
// partial per reduction block. Every slot a kernel reads is written earlier in the same
// call (all sites of the grid, all kBlocks partials and the final slot), so nothing has to
// start at zero; the arrays keep the last call's contents.
// ---------------------------------------------------------------------------------------
static __device__ __align__(256) double4 g_noalloc_nematic[KZM_NOALLOC_MAX_SITES];
static __device__ __align__(256) KzmPartial g_noalloc_partials[kBlocks + 1];

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mutex;
double4* g_noalloc_nematic_ptr[kMaxDevices] = {};
KzmPartial* g_noalloc_partials_ptr[kMaxDevices] = {};

// Device addresses of the scratch arrays for the current device, looked up once per device.
int noalloc_scratch(double4** nf, KzmPartial** part) {
    int dev = 0;
    LDG_CUDA(cudaGetDevice(&dev));
    LDG_REQUIRE(dev >= 0 && dev < kMaxDevices, LDG_ERR_ARG, "kzm_observe_device_noalloc: device ordinal out of range");
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_nematic_ptr[dev]) {
        void* a = nullptr;
        void* b = nullptr;
        LDG_CUDA(cudaGetSymbolAddress(&a, g_noalloc_nematic));
        LDG_CUDA(cudaGetSymbolAddress(&b, g_noalloc_partials));
        g_noalloc_nematic_ptr[dev] = static_cast<double4*>(a);
        g_noalloc_partials_ptr[dev] = static_cast<KzmPartial*>(b);
    }
    *nf = g_noalloc_nematic_ptr[dev];
    *part = g_noalloc_partials_ptr[dev];
    return LDG_OK;
}
}  // namespace

extern "C" {

int kzm_observe_device_noalloc(const kzm_params* params, const double* q, double A, double B, double C,
                               void* stream, kzm_observables* o) {
    clear_error();
    LDG_REQUIRE(params && q && o, LDG_ERR_ARG, "kzm_observe_device_noalloc: null argument");
    const kzm_params& p = *params;
    LDG_REQUIRE(p.Nx > 1 && p.Ny > 1 && p.Nz > 1, LDG_ERR_ARG,
                "Nx, Ny, and Nz must all be greater than 1 for the periodic bulk LdG branch");
    LDG_REQUIRE(p.dx > 0 && p.dy > 0 && p.dz > 0, LDG_ERR_ARG, "dx, dy, and dz must be positive");
    const long long n = (long long)p.Nx * p.Ny * p.Nz;
    LDG_REQUIRE(n <= KZM_NOALLOC_MAX_SITES, LDG_ERR_ARG,
                "kzm_observe_device_noalloc: " + std::to_string(n) + " sites exceed the no-allocation scratch limit of " +
                    std::to_string(KZM_NOALLOC_MAX_SITES) + " sites (use kzm_observe for larger grids)");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (st) {
        // the scratch address is the current device's: a stream of another device cannot use it
        int cur = 0, sdev = 0;
        LDG_CUDA(cudaGetDevice(&cur));
        LDG_CUDA(cudaStreamGetDevice(st, &sdev));
        LDG_REQUIRE(sdev == cur, LDG_ERR_ARG,
                    "kzm_observe_device_noalloc: the stream belongs to device " + std::to_string(sdev) +
                        ", not to the current device " + std::to_string(cur));
    }
    double4* nf = nullptr;
    KzmPartial* part = nullptr;
    int rc = noalloc_scratch(&nf, &part);
    if (rc) return rc;
    KzmObsConst O{};
    O.P.Nx = p.Nx; O.P.Ny = p.Ny; O.P.Nz = p.Nz;
    O.A = A; O.B = B; O.C = C; O.kappa = p.kappa;
    O.cv = p.dx * p.dy * p.dz;
    O.ix = 1.0 / p.dx; O.iy = 1.0 / p.dy; O.iz = 1.0 / p.dz;
    k_kzm_obs_sites<true><<<kBlocks, kThreads, 0, st>>>(q, O, nf, part);
    k_kzm_obs_plaq<<<kBlocks, kThreads, 0, st>>>(nf, O, p.defects_S_threshold, p.defects_charge_cutoff, p.dx, p.dy,
                                                  p.dz, part);
    k_kzm_obs_final<<<1, kThreads, 0, st>>>(part, kBlocks, part + kBlocks);
    LDG_LAUNCHED("kzm_observe_device_noalloc kernels");
    KzmPartial R{};
    LDG_CUDA(cudaMemcpyAsync(&R, part + kBlocks, sizeof(R), cudaMemcpyDeviceToHost, st));
    LDG_CUDA(cudaStreamSynchronize(st));
    const double tv = O.cv * (double)p.Nx * (double)p.Ny * (double)p.Nz;
    const double nan = std::numeric_limits<double>::quiet_NaN();
    o->bulk = R.bulk / tv;
    o->elastic = R.elastic / tv;
    o->total = o->bulk + o->elastic;
    o->avg_S = R.S_sum / (double)n;
    o->max_S = R.S_max;
    o->defect_plaquettes_used = (long long)R.used;
    o->nonzero_defect_plaquettes = (long long)R.defects;
    o->defect_density_per_plaquette = R.used > 0 ? (double)R.defects / (double)R.used : nan;
    o->defect_line_density = tv > 0.0 ? R.line / tv : nan;
    o->xi_grad_proxy = (R.gint > 0.0 && R.qint > 0.0) ? std::sqrt(R.qint / R.gint) : nan;
    return LDG_OK;
}

void* kzm_stream(kzm_handle* h) { return h ? (void*)h->stream : nullptr; }

long long kzm_launch_count(const kzm_handle* h) { return h ? h->launches : 0; }

int kzm_destroy(kzm_handle* h) {
    if (!h) return LDG_OK;
    DeviceGuard device_guard(h->device);
    if (h->stream) cudaStreamSynchronize(h->stream);
    cudaFree(h->alloc[0]); cudaFree(h->alloc[1]); cudaFree(h->stage); cudaFree(h->nf); cudaFree(h->part);
    if (h->stream) cudaStreamDestroy(h->stream);
    delete h;
    return LDG_OK;
}

}  // extern "C"
