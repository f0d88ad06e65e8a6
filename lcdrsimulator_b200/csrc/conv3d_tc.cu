// BF16 tensor-core (tcgen05) implicit-GEMM 3x3x3 convolutions for the warm-start surrogate.
//
// Activations are NDHWC BF16 (channels innermost), weights [Co][27][Ci] BF16 with the tap
// index t = 9*(dz+1) + 3*(dy+1) + (dx+1). Convolutions are stride 1 with zero padding 1.
//
// Forward (and data gradient, which is the forward of the flipped, transposed weights):
//   GEMM M = 128 output voxels per CTA, N = Co, K = 27 taps x Ci. Each K step is one TMA load
//   of the input box shifted by the tap (the tensor map's zero fill outside the volume is the
//   padding) plus one TMA load of the weights of that tap; both land 128B/64B/32B-swizzled,
//   K-major, exactly as the UMMA descriptors read them. One thread issues tcgen05.mma into a
//   TMEM accumulator of 128 lanes x Co columns; the epilogue reads TMEM with tcgen05.ld and
//   applies bias and leaky ReLU before the BF16 (or FP32) store.
//   Narrow layers on long volumes march along z instead, loading each shifted plane once for the
//   three taps along z that read it.
// Weight gradient:
//   GEMM M = 128 rows of (tap, ci), N = Co, K = voxels, both operands MN-major (channels are
//   contiguous per voxel): the A tile stacks 128/Ci taps of the shifted input, the B tile is
//   the output gradient. K is split over CTAs and reduced with FP32 atomics.
//
// Every mbarrier wait is bounded; on timeout the kernel records LDG_ERR_TIMEOUT, waits
// (bounded) for its loads in flight, releases its TMEM and returns.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <mutex>
#include <string>

#include "ldg_api_common.h"
#include "sm100_ptx.cuh"

using namespace ldg;
using namespace ldg::sm100;

namespace {

constexpr int BM = 128;     // UMMA M
constexpr int STAGES = 4;
// Stages of the weight gradient: three leave room for one more CTA per SM than four, and all the
// CTAs of a launch run at once (32 -> 32 channels, 64^3 x 4: 0.247 ms with four, 0.205 with three).
constexpr int WG_STAGES = 3;
constexpr int kWgFixed = 8;  // a weight-gradient CTA's start and atomics, in K boxes
constexpr int KV = 64;      // voxels per weight-gradient K stage

struct BoxDims {
    int bx, by, bz, bn;     // box extent per dimension, each within the tensor's extent
    int tx, ty, tz, tn;     // boxes per dimension (ceil)
    int rows;               // voxels per box = bx * by * bz * bn (<= the GEMM tile's rows)
};

struct FwdArgs {
    int N, D, H, W, Ci, Co;
    BoxDims b;
    int act;       // 0 identity, 1 leaky ReLU (slope 0.01)
    int out_f32;
    int ksteps;    // 27 * cchunks
    int cs;        // output channels of a CTA: Co / gridDim.y
    uint32_t tmem_cols;
};

struct WgArgs {
    int N, D, H, W, Ci, Co;
    BoxDims b;             // 64-voxel K boxes
    long long nkb;         // number of K boxes
    int kb_per_cta;
    uint32_t tmem_cols;
};

__device__ __forceinline__ void box_origin(const BoxDims& b, long long t, int& x0, int& y0, int& z0, int& n0) {
    const int xi = (int)(t % b.tx); t /= b.tx;
    const int yi = (int)(t % b.ty); t /= b.ty;
    const int zi = (int)(t % b.tz); t /= b.tz;
    x0 = xi * b.bx; y0 = yi * b.by; z0 = zi * b.bz; n0 = (int)t * b.bn;
}

__device__ __forceinline__ float act_apply(float v, int act) { return (act == 1 && v < 0.0f) ? 0.01f * v : v; }

// Bias, activation and store of 16 channels c.. of a voxel, at element o of y.
__device__ __forceinline__ void store16(void* __restrict__ y, const float* __restrict__ bias, float* v, long long o, int c,
                                        int act, int f32) {
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = act_apply(v[i] + (bias ? bias[c + i] : 0.0f), act);
    if (f32) {
        float4* dst = reinterpret_cast<float4*>(static_cast<float*>(y) + o);
#pragma unroll
        for (int q = 0; q < 4; ++q) dst[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
    } else {
        uint32_t p[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * q], v[2 * q + 1]);
            p[q] = *reinterpret_cast<uint32_t*>(&h);
        }
        uint4* dst = reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(y) + o);
        dst[0] = make_uint4(p[0], p[1], p[2], p[3]);
        dst[1] = make_uint4(p[4], p[5], p[6], p[7]);
    }
}

// ---------------------------------------------------------------------------------------
// Forward / data-gradient kernel
// ---------------------------------------------------------------------------------------
template <int CK>
__global__ void __launch_bounds__(128, 1)
    k_conv3d_fwd(const __grid_constant__ CUtensorMap tmx, const __grid_constant__ CUtensorMap tmw, void* __restrict__ y,
                 const float* __restrict__ bias, FwdArgs a, int* __restrict__ err) {
    constexpr uint32_t ROW = CK * 2;             // bytes per smem row (one voxel or one output channel)
    constexpr uint32_t A_BYTES = BM * ROW;
    constexpr uint32_t SWZ = swizzle_code(ROW);
    constexpr uint32_t SBO = 8 * ROW;            // 8-row core-matrix group stride
    const uint32_t B_BYTES = (uint32_t)a.cs * ROW;
    const uint32_t B_STRIDE = (B_BYTES + 1023u) & ~1023u;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* sA = base;
    unsigned char* sB = base + STAGES * A_BYTES;
    uint64_t* full = (uint64_t*)(sB + STAGES * B_STRIDE);
    uint64_t* empty = full + STAGES;
    uint64_t* done = empty + STAGES;
    uint32_t* tslot = (uint32_t*)(done + 1);

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    int x0, y0, z0, n0;
    box_origin(a.b, blockIdx.x, x0, y0, z0, n0);
    const int co0 = (int)blockIdx.y * a.cs;

    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(done, 1);
        fence_mbar_init();
    }
    if (warp == 0) {
        __syncwarp();
        tmem_alloc(tslot, a.tmem_cols);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;

    bool ok = true;
    if (warp == 0) {
        // TMA producer
        int issued = 0, tap = 0, cc = 0, dx = -1, dy = -1, dz = -1;  // tap = 9 (dz + 1) + 3 (dy + 1) + dx + 1
        for (int ks = 0; ks < a.ksteps; ++ks) {
            const int s = ks % STAGES;
            if (ks >= STAGES && !mbar_wait_warp(&empty[s], ((ks / STAGES) - 1) & 1)) {
                atomicExch(err, LDG_ERR_TIMEOUT);
                break;
            }
            if (elect_one()) {
                mbar_expect_tx(&full[s], (uint32_t)a.b.rows * ROW + B_BYTES);
                tma_load_5d(sA + s * A_BYTES, &tmx, cc, x0 + dx, y0 + dy, z0 + dz, n0, &full[s]);
                tma_load_3d(sB + s * B_STRIDE, &tmw, cc, tap, co0, &full[s]);
            }
            __syncwarp();
            issued = ks + 1;
            cc += CK;
            if (cc == a.Ci) {
                cc = 0;
                ++tap;
                if (++dx == 2) {
                    dx = -1;
                    if (++dy == 2) { dy = -1; ++dz; }
                }
            }
        }
        for (int ks = (issued > STAGES ? issued - STAGES : 0); ks < issued; ++ks)
            if (!mbar_wait_warp(&full[ks % STAGES], (ks / STAGES) & 1)) atomicExch(err, LDG_ERR_TIMEOUT);
    } else if (warp == 1) {
        // MMA issuer
        const uint32_t idesc = idesc_bf16(BM, a.cs, false, false);
        for (int ks = 0; ks < a.ksteps; ++ks) {
            const int s = ks % STAGES;
            if (!mbar_wait_warp(&full[s], (ks / STAGES) & 1)) {
                atomicExch(err, LDG_ERR_TIMEOUT);
                break;
            }
            tc_fence_after();
            const uint32_t a0 = smem_u32(sA + s * A_BYTES), b0 = smem_u32(sB + s * B_STRIDE);
            if (elect_one()) {
#pragma unroll
                for (int k = 0; k < CK / 16; ++k)
                    umma_bf16(tmem, smem_desc(a0 + k * 32, 16, SBO, SWZ), smem_desc(b0 + k * 32, 16, SBO, SWZ), idesc,
                              (ks | k) != 0 ? 1u : 0u);
                umma_commit(&empty[s]);
            }
            __syncwarp();
        }
        if (elect_one()) umma_commit(done);
        __syncwarp();
        ok = mbar_wait_warp(done, 0);
    }
    // Epilogue: row m of the accumulator is output voxel m of the box; warp w owns lanes 32w..32w+31.
    // The other lanes of the two working warps stand at a warp barrier until here: polling `done`
    // from them held up the producing and the issuing lane of the same warp at every stage.
    __syncwarp();
    ok = __syncthreads_and(ok) != 0;
    tc_fence_after();
    if (!ok && tid == 0) atomicExch(err, LDG_ERR_TIMEOUT);
    const int m = tid;
    const int xi = m % a.b.bx, yi = (m / a.b.bx) % a.b.by, zi = (m / (a.b.bx * a.b.by)) % a.b.bz;
    const int ni = m / (a.b.bx * a.b.by * a.b.bz);
    const int x = x0 + xi, yy = y0 + yi, z = z0 + zi, n = n0 + ni;
    const bool inside = ok && m < a.b.rows && x < a.W && yy < a.H && z < a.D && n < a.N;
    const long long vox = (((long long)n * a.D + z) * a.H + yy) * a.W + x;
    const uint32_t trow = tmem + ((uint32_t)(warp * 32) << 16);
    for (int c0 = 0; c0 < a.cs; c0 += 16) {
        float v[16];
        tmem_ld16(trow + (uint32_t)c0, v);
        if (!inside) continue;
        store16(y, bias, v, vox * a.Co + co0 + c0, co0 + c0, a.act, a.out_f32);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, a.tmem_cols);
    }
}

// ---------------------------------------------------------------------------------------
// Forward / data gradient of narrow layers: a march along z
// ---------------------------------------------------------------------------------------
// With few channels k_conv3d_fwd is bound by reading each input box 27 times from L2 (64^3 x 4
// volumes, 32 -> 32 channels: 2.3 GB in 0.163 ms). Here a CTA keeps all 27 weight slices in shared
// memory and marches a 128-voxel (x, y) tile along z: each of a plane's nine (dy, dx)-shifted boxes
// is loaded once and multiplied for the three output planes that it belongs to, in three of four
// TMEM accumulators, while four warps store the plane that is complete (0.108 ms). An output takes its
// taps in the order of k_conv3d_fwd (dz outermost), so the results are the same bits.
struct MarchArgs {
    int D, H, W, Co, bx, by, tx, ty;
    int zlen, act, out_f32;
    uint32_t acc_cols, tmem_cols;  // columns of an accumulator, and of the four
};

template <int CK>
__global__ void __launch_bounds__(192, 1)
    k_conv3d_march(const __grid_constant__ CUtensorMap tmx, const __grid_constant__ CUtensorMap tmw, void* __restrict__ y,
                   const float* __restrict__ bias, MarchArgs a, int* __restrict__ err) {
    constexpr int MS = CK == 64 ? 4 : 6;  // stages
    constexpr uint32_t ROW = CK * 2, A_BYTES = BM * ROW, SWZ = swizzle_code(ROW), SBO = 8 * ROW;
    const uint32_t B_BYTES = (uint32_t)a.Co * ROW, B_STRIDE = (B_BYTES + 1023u) & ~1023u;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* sA = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* sB = sA + MS * A_BYTES;
    uint64_t* full = (uint64_t*)(sB + 27 * B_STRIDE);
    uint64_t* empty = full + MS;
    uint64_t* acc_full = empty + MS;    // [4] an accumulator holds its whole output plane
    uint64_t* acc_empty = acc_full + 4; // [4] its plane has been read
    uint64_t* wfull = acc_empty + 4;
    uint64_t* done = wfull + 1;
    uint32_t* tslot = (uint32_t*)(done + 1);

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int x0 = (int)(blockIdx.x % a.tx) * a.bx, y0 = (int)(blockIdx.x / a.tx) * a.by;
    const int n0 = (int)blockIdx.z, z0 = (int)blockIdx.y * a.zlen;
    const int z1 = min(z0 + a.zlen, a.D);  // output planes [z0, z1)
    const int nplanes = z1 - z0 + 2;       // input planes z0 - 1 .. z1 (zeros outside the volume)

    if (tid == 0) {
        for (int s = 0; s < MS; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int s = 0; s < 4; ++s) {
            mbar_init(&acc_full[s], 1);
            mbar_init(&acc_empty[s], 128);
        }
        mbar_init(wfull, 1);
        mbar_init(done, 1);
        fence_mbar_init();
    }
    if (warp == 0) {
        __syncwarp();
        tmem_alloc(tslot, a.tmem_cols);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;

    bool ok = true;
    if (warp == 0) {
        if (elect_one()) {
            mbar_expect_tx(wfull, 27 * B_BYTES);
            for (int t = 0; t < 27; ++t) tma_load_3d(sB + t * B_STRIDE, &tmw, 0, t, 0, wfull);
        }
        __syncwarp();
        int s = 0, issued = 0;
        uint32_t phase = 1;
        for (int p = 0; p < nplanes && ok; ++p)
            for (int t = 0; t < 9; ++t) {
                if (issued >= MS && !(ok = mbar_wait_warp(&empty[s], phase))) break;
                if (elect_one()) {
                    mbar_expect_tx(&full[s], A_BYTES);
                    tma_load_5d(sA + s * A_BYTES, &tmx, 0, x0 + t % 3 - 1, y0 + t / 3 - 1, z0 - 1 + p, n0, &full[s]);
                }
                __syncwarp();
                ++issued;
                if (++s == MS) s = 0, phase ^= 1u;
            }
        // the loads in flight land before the block may end
        for (int k = (issued > MS ? issued - MS : 0); k < issued; ++k)
            if (!mbar_wait_warp(&full[k % MS], (k / MS) & 1)) ok = false;
        if (!mbar_wait_warp(wfull, 0)) ok = false;
    } else if (warp == 1) {
        const uint32_t idesc = idesc_bf16(BM, a.Co, false, false);
        const uint32_t b00 = smem_u32(sB);
        int s = 0;
        uint32_t phase = 0;
        ok = mbar_wait_warp(wfull, 0);
        for (int p = 0; p < nplanes && ok; ++p) {
            // input plane p of the march is dz = +1 of output p - 2, 0 of p - 1, -1 of p
            if (p >= 4 && p < z1 - z0) {
                if (!(ok = mbar_wait_warp(&acc_empty[p & 3], ((p >> 2) - 1) & 1))) break;
                tc_fence_after();
            }
            for (int t = 0; t < 9; ++t) {
                if (!(ok = mbar_wait_warp(&full[s], phase))) break;
                tc_fence_after();
                const uint32_t a0 = smem_u32(sA + s * A_BYTES);
                if (elect_one()) {
#pragma unroll
                    for (int dz = 0; dz < 3; ++dz) {  // dz + 1 of the tap
                        const int o = p - dz;
                        if (o < 0 || o >= z1 - z0) continue;
                        const uint32_t b0 = b00 + (uint32_t)(9 * dz + t) * B_STRIDE, d = tmem + (uint32_t)(o & 3) * a.acc_cols;
#pragma unroll
                        for (int k = 0; k < CK / 16; ++k)
                            umma_bf16(d, smem_desc(a0 + k * 32, 16, SBO, SWZ), smem_desc(b0 + k * 32, 16, SBO, SWZ), idesc,
                                      (dz | t | k) != 0 ? 1u : 0u);
                    }
                    umma_commit(&empty[s]);
                    if (t == 8 && p >= 2) umma_commit(&acc_full[(p - 2) & 3]);
                }
                __syncwarp();
                if (++s == MS) s = 0, phase ^= 1u;
            }
        }
        if (elect_one()) umma_commit(done);
        __syncwarp();
        if (!mbar_wait_warp(done, 0)) ok = false;
    } else {
        // warp w reads the TMEM lanes 32 (w & 3) ..: row m of the tile is voxel (m % bx, m / bx)
        const int m = (warp & 3) * 32 + (tid & 31);
        const int x = x0 + m % a.bx, yy = y0 + m / a.bx;
        const bool inside = x < a.W && yy < a.H;
        for (int o = 0; o < z1 - z0; ++o) {
            if (!(ok = mbar_wait_warp(&acc_full[o & 3], (o >> 2) & 1))) break;
            tc_fence_after();
            const long long vox = (((long long)n0 * a.D + z0 + o) * a.H + yy) * a.W + x;
            const uint32_t trow = tmem + (uint32_t)(o & 3) * a.acc_cols + ((uint32_t)((warp & 3) * 32) << 16);
            for (int c0 = 0; c0 < a.Co; c0 += 16) {
                float v[16];
                __syncwarp();
                tmem_ld16(trow + (uint32_t)c0, v);
                if (inside) store16(y, bias, v, vox * a.Co + c0, c0, a.act, a.out_f32);
            }
            tc_fence_before();
            mbar_arrive(&acc_empty[o & 3]);
        }
    }
    __syncwarp();
    if (!ok) atomicExch(err, LDG_ERR_TIMEOUT);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, a.tmem_cols);
    }
}

// ---------------------------------------------------------------------------------------
// Weight-gradient kernel
// ---------------------------------------------------------------------------------------
template <int ACA, int ACB>
__global__ void __launch_bounds__(128, 1)
    k_conv3d_wgrad(const __grid_constant__ CUtensorMap tmx, const __grid_constant__ CUtensorMap tmdy,
                   float* __restrict__ dw, WgArgs a, int* __restrict__ err) {
    constexpr uint32_t ROWA = ACA * 2, ROWB = ACB * 2;
    constexpr uint32_t ATOM_A = KV * ROWA;            // ACA channels x 64 voxels
    constexpr uint32_t ATOM_B = KV * ROWB;
    constexpr int NATOM_A = BM / ACA;
    constexpr uint32_t A_BYTES = NATOM_A * ATOM_A;    // 16 KB
    constexpr uint32_t SWZA = swizzle_code(ROWA), SWZB = swizzle_code(ROWB);
    constexpr uint32_t SBOA = 8 * ROWA, SBOB = 8 * ROWB;
    const int natom_b = a.Co / ACB;
    const uint32_t B_BYTES = (uint32_t)natom_b * ATOM_B;
    const uint32_t B_STRIDE = (B_BYTES + 1023u) & ~1023u;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* sA = base;
    unsigned char* sB = base + WG_STAGES * A_BYTES;
    uint64_t* full = (uint64_t*)(sB + WG_STAGES * B_STRIDE);
    uint64_t* empty = full + WG_STAGES;
    uint64_t* done = empty + WG_STAGES;
    uint32_t* tslot = (uint32_t*)(done + 1);

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    // Row block of this CTA: 128 rows of (tap, ci).
    const bool wide = a.Ci > BM;                       // Ci = 256: two tiles per tap
    const int tap_base = wide ? (int)(blockIdx.x >> 1) : (int)blockIdx.x * (BM / a.Ci);
    const int ci_base = wide ? (int)(blockIdx.x & 1) * BM : 0;
    const long long kb0 = (long long)blockIdx.y * a.kb_per_cta;
    const long long kb1 = (kb0 + a.kb_per_cta < a.nkb) ? kb0 + a.kb_per_cta : a.nkb;
    const int nsteps = (int)(kb1 > kb0 ? kb1 - kb0 : 0);

    // A atoms of this tile that hold a real tap (rows of taps >= 27 are left unloaded and
    // their accumulator rows are discarded).
    // Channel and tap shift of each atom, worked out once: the one producing thread is a serial
    // chain, and with the divisions inside it the loads of a box were issued more slowly than
    // they arrived (64^3 x 4 volumes, 32 channels: 0.79 ms with the divisions, 0.39 ms
    // without; 0.26 ms with the whole warp in the loop and one elected lane issuing, where operands
    // stay uniform; 0.20 ms with WG_STAGES).
    int natom_a_valid = 0;
    int aci[NATOM_A], adx[NATOM_A], ady[NATOM_A], adz[NATOM_A];
#pragma unroll
    for (int j = 0; j < NATOM_A; ++j) {
        const int row0 = j * ACA;
        const int tap = wide ? tap_base : tap_base + row0 / a.Ci;
        if (tap < 27) natom_a_valid = j + 1;  // taps grow with j
        aci[j] = wide ? ci_base + row0 : row0 % a.Ci;
        adz[j] = tap / 9 - 1, ady[j] = (tap / 3) % 3 - 1, adx[j] = tap % 3 - 1;
    }

    if (tid == 0) {
        for (int s = 0; s < WG_STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(done, 1);
        fence_mbar_init();
    }
    // K rows past the box (volumes smaller than 64 voxels) are never written by the loads and
    // take part in the reduction: zero them once in every stage (a row's 16-byte chunks stay
    // inside the row under the swizzle).
    if (a.b.rows < KV) {
        const uint32_t za = (uint32_t)(KV - a.b.rows) * ROWA, zb = (uint32_t)(KV - a.b.rows) * ROWB;
        for (int s = 0; s < WG_STAGES; ++s) {
            for (int j = 0; j < NATOM_A; ++j) {
                uint4* p = reinterpret_cast<uint4*>(sA + s * A_BYTES + j * ATOM_A + (uint32_t)a.b.rows * ROWA);
                for (uint32_t q = tid; q < za / 16; q += blockDim.x) p[q] = make_uint4(0, 0, 0, 0);
            }
            for (int j = 0; j < natom_b; ++j) {
                uint4* p = reinterpret_cast<uint4*>(sB + s * B_STRIDE + j * ATOM_B + (uint32_t)a.b.rows * ROWB);
                for (uint32_t q = tid; q < zb / 16; q += blockDim.x) p[q] = make_uint4(0, 0, 0, 0);
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 0) {
        __syncwarp();
        tmem_alloc(tslot, a.tmem_cols);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;

    bool ok = true;
    if (warp == 0) {
        int issued = 0, vx, vy, vz, vn;
        box_origin(a.b, kb0, vx, vy, vz, vn);
        int s = 0;
        uint32_t phase = 1;  // of the stage's previous release
        for (int st = 0; st < nsteps; ++st) {
            if (st >= WG_STAGES && !mbar_wait_warp(&empty[s], phase)) {
                atomicExch(err, LDG_ERR_TIMEOUT);
                break;
            }
            if (elect_one()) {
                mbar_expect_tx(&full[s], (uint32_t)(natom_a_valid * ACA + a.Co) * (uint32_t)a.b.rows * 2u);
#pragma unroll
                for (int j = 0; j < NATOM_A; ++j)
                    if (j < natom_a_valid)
                        tma_load_5d(sA + s * A_BYTES + j * ATOM_A, &tmx, aci[j], vx + adx[j], vy + ady[j], vz + adz[j],
                                    vn, &full[s]);
                for (int j = 0; j < natom_b; ++j)
                    tma_load_5d(sB + s * B_STRIDE + j * ATOM_B, &tmdy, j * ACB, vx, vy, vz, vn, &full[s]);
            }
            __syncwarp();
            issued = st + 1;
            if (++s == WG_STAGES) s = 0, phase ^= 1u;
            // next box, x fastest (a division per box here cost more than the box's matrix products)
            if ((vx += a.b.bx) >= a.b.tx * a.b.bx) {
                vx = 0;
                if ((vy += a.b.by) >= a.b.ty * a.b.by) {
                    vy = 0;
                    if ((vz += a.b.bz) >= a.b.tz * a.b.bz) { vz = 0; vn += a.b.bn; }
                }
            }
        }
        for (int st = (issued > WG_STAGES ? issued - WG_STAGES : 0); st < issued; ++st)
            if (!mbar_wait_warp(&full[st % WG_STAGES], (st / WG_STAGES) & 1)) atomicExch(err, LDG_ERR_TIMEOUT);
    } else if (warp == 1) {
        const uint32_t idesc = idesc_bf16(BM, a.Co, true, true);
        int s = 0;
        uint32_t phase = 0;
        for (int st = 0; st < nsteps; ++st) {
            if (!mbar_wait_warp(&full[s], phase)) {
                atomicExch(err, LDG_ERR_TIMEOUT);
                break;
            }
            tc_fence_after();
            const uint32_t a0 = smem_u32(sA + s * A_BYTES), b0 = smem_u32(sB + s * B_STRIDE);
            if (elect_one()) {
#pragma unroll
                for (int k = 0; k < KV / 16; ++k)
                    umma_bf16(tmem, smem_desc(a0 + k * 2 * SBOA, ATOM_A, SBOA, SWZA),
                              smem_desc(b0 + k * 2 * SBOB, ATOM_B, SBOB, SWZB), idesc, (st | k) != 0 ? 1u : 0u);
                umma_commit(&empty[s]);
            }
            __syncwarp();
            if (++s == WG_STAGES) s = 0, phase ^= 1u;
        }
        if (elect_one()) umma_commit(done);
        __syncwarp();
        ok = mbar_wait_warp(done, 0);
    }
    __syncwarp();  // see k_conv3d_fwd
    ok = __syncthreads_and(ok) != 0;
    tc_fence_after();
    if (!ok && tid == 0) atomicExch(err, LDG_ERR_TIMEOUT);
    const int m = tid;
    const int tap = wide ? tap_base : tap_base + m / a.Ci;
    const int ci = wide ? ci_base + m : m % a.Ci;
    const bool valid = ok && nsteps > 0 && tap < 27;
    const uint32_t trow = tmem + ((uint32_t)(warp * 32) << 16);
    for (int c0 = 0; c0 < a.Co; c0 += 16) {
        float v[16];
        tmem_ld16(trow + (uint32_t)c0, v);
        if (!valid) continue;
#pragma unroll
        for (int i = 0; i < 16; ++i) atomicAdd(&dw[((long long)(c0 + i) * 27 + tap) * a.Ci + ci], v[i]);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, a.tmem_cols);
    }
}

// ---------------------------------------------------------------------------------------
// Activation mask of the output gradient and bias gradient, one pass
// ---------------------------------------------------------------------------------------
// g = gy * (y > 0 ? 1 : slope) in gy's type (FP32 or BF16; the slope is rounded to it), rounded
// to BF16; part[block][c] = sum over the block's voxels of g[., c]. Bound by memory: it reads y
// and gy and writes g once, where the same as separate elementwise operations and a reduction
// moved the field eleven times through FP32 temporaries (64^3 x 4, 32 channels: 331 us; 35 us here,
// 201 MB at 5.7 TB/s). A thread keeps eight
// channels, so the sums need no exchange until the block's end; they are kept in FP64.
template <typename T, bool kMask>
__global__ void __launch_bounds__(256)
    k_act_grad(const T* __restrict__ y, const T* __restrict__ gy, __nv_bfloat16* __restrict__ g, double* __restrict__ part,
               long long nvox, int C) {
    extern __shared__ double s_part[];  // [256][8]
    const int lanes = C / 8, per = 256 / lanes, used = per * lanes;  // threads per voxel, voxels per pass
    const int tid = threadIdx.x, c8 = tid % lanes;
    const float slope = sizeof(T) == 2 ? __bfloat162float(__float2bfloat16_rn(0.01f)) : 0.01f;
    double acc[8] = {};
    if (tid < used)
        for (long long v = (long long)blockIdx.x * per + tid / lanes; v < nvox; v += (long long)gridDim.x * per) {
            const long long o = v * C + c8 * 8;
            float a[8], m[8];
            if constexpr (sizeof(T) == 2) {
                const uint4 q = *reinterpret_cast<const uint4*>(gy + o);
                const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    a[2 * i] = __uint_as_float(w[i] << 16), a[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
                if constexpr (kMask) {
                    const uint4 p = *reinterpret_cast<const uint4*>(y + o);
                    const uint32_t u[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        m[2 * i] = __uint_as_float(u[i] << 16), m[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u);
                }
            } else {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float4 q = *reinterpret_cast<const float4*>(gy + o + 4 * h);
                    a[4 * h] = q.x, a[4 * h + 1] = q.y, a[4 * h + 2] = q.z, a[4 * h + 3] = q.w;
                    if constexpr (kMask) {
                        const float4 p = *reinterpret_cast<const float4*>(y + o + 4 * h);
                        m[4 * h] = p.x, m[4 * h + 1] = p.y, m[4 * h + 2] = p.z, m[4 * h + 3] = p.w;
                    }
                }
            }
            uint32_t r[4];
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if constexpr (kMask) a[i] = m[i] > 0.0f ? a[i] : a[i] * slope;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const __nv_bfloat162 h = __floats2bfloat162_rn(a[2 * i], a[2 * i + 1]);
                r[i] = *reinterpret_cast<const uint32_t*>(&h);
                acc[2 * i] += (double)__uint_as_float(r[i] << 16);
                acc[2 * i + 1] += (double)__uint_as_float(r[i] & 0xffff0000u);
            }
            if (g) *reinterpret_cast<uint4*>(g + o) = make_uint4(r[0], r[1], r[2], r[3]);
        }
#pragma unroll
    for (int i = 0; i < 8; ++i) s_part[tid * 8 + i] = acc[i];
    __syncthreads();
    for (int c = tid; c < C; c += 256) {
        double t = 0.0;
        for (int k = 0; k < per; ++k) t += s_part[(k * lanes + c / 8) * 8 + c % 8];
        part[(long long)blockIdx.x * C + c] = t;
    }
}

// db[c] = sum over the blocks of part[block][c]; one block of 32 x 8 threads per 8 channels
__global__ void __launch_bounds__(256) k_act_grad_sum(const double* __restrict__ part, float* __restrict__ db, int blocks, int C) {
    __shared__ double s[256];
    const int c = blockIdx.x * 8 + (threadIdx.x & 7);
    double t = 0.0;
    for (int b = threadIdx.x >> 3; b < blocks; b += 32) t += part[(long long)b * C + c];
    s[threadIdx.x] = t;
    __syncthreads();
    for (int h = 128; h >= 8; h >>= 1) {
        if (threadIdx.x < h) s[threadIdx.x] += s[threadIdx.x + h];
        __syncthreads();
    }
    if (threadIdx.x < 8) db[c] = (float)s[threadIdx.x];
}

int act_grad_blocks(long long nvox, int C) {
    const long long per = 256 / (C / 8);
    return (int)std::max(1LL, std::min<long long>((nvox + 4 * per - 1) / (4 * per), 148 * 8));
}

template <typename T>
int launch_act_grad(long long nvox, int C, const void* y, const void* gy, void* g, float* db, double* ws, cudaStream_t st) {
    const int blocks = act_grad_blocks(nvox, C);
    const size_t smem = 256 * 8 * sizeof(double);
    if (y)
        k_act_grad<T, true><<<blocks, 256, smem, st>>>((const T*)y, (const T*)gy, (__nv_bfloat16*)g, ws, nvox, C);
    else
        k_act_grad<T, false><<<blocks, 256, smem, st>>>(nullptr, (const T*)gy, (__nv_bfloat16*)g, ws, nvox, C);
    LDG_LAUNCHED("k_act_grad");
    k_act_grad_sum<<<C / 8, 256, 0, st>>>(ws, db, blocks, C);
    LDG_LAUNCHED("k_act_grad_sum");
    return LDG_OK;
}

// w[co][t][ci] -> wf[ci][26 - t][co]: the data gradient is the forward convolution of the
// output gradient with these weights. A 32 x 32 tile of (co, ci) of one tap is turned in shared
// memory, so that both sides move whole sectors (element by element the writes were 2 bytes to a
// sector: 18 us at 256 x 256 channels, 4 us now).
__global__ void __launch_bounds__(256)
    k_flip_weights(const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ wf, int Ci, int Co) {
    __shared__ __nv_bfloat16 tile[32][34];
    const int t = blockIdx.x, ci0 = blockIdx.y * 32, co0 = blockIdx.z * 32;
    const int a = threadIdx.x & 31, b = threadIdx.x >> 5;
    for (int r = b; r < 32; r += 8)
        if (co0 + r < Co && ci0 + a < Ci) tile[r][a] = w[((long long)(co0 + r) * 27 + t) * Ci + ci0 + a];
    __syncthreads();
    for (int r = b; r < 32; r += 8)
        if (ci0 + r < Ci && co0 + a < Co) wf[((long long)(ci0 + r) * 27 + 26 - t) * Co + co0 + a] = tile[a][r];
}

// ---------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------
constexpr int kMaxDevices = 64;
int* g_err_dev[kMaxDevices] = {};  // device error word of each GPU (allocated on first use there)
int* g_err = nullptr;              // the current device's word (set by ensure_err)
long long g_launches = 0;
std::mutex g_mu;

int ensure_err() {
    int dev = 0;
    LDG_CUDA(cudaGetDevice(&dev));
    LDG_REQUIRE(dev >= 0 && dev < kMaxDevices, LDG_ERR_ARG, "conv3d: device index out of range");
    if (!g_err_dev[dev]) {
        int* word = nullptr;
        LDG_CUDA(cudaMalloc(&word, sizeof(int)));
        cudaError_t e = cudaMemset(word, 0, sizeof(int));
        if (e == cudaSuccess) e = cudaStreamSynchronize(nullptr);  // callers' streams do not wait for the default one
        if (e != cudaSuccess) cudaFree(word);
        LDG_CUDA(e);
        g_err_dev[dev] = word;
    }
    g_err = g_err_dev[dev];
    return LDG_OK;
}

int pow2_floor(int v) {
    int p = 1;
    while (p * 2 <= v) p *= 2;
    return p;
}

BoxDims make_box(int N, int D, int H, int W, int total) {
    BoxDims b{};
    b.bx = std::min(pow2_floor(W), total);
    b.by = std::min(pow2_floor(H), total / b.bx);
    b.bz = std::min(pow2_floor(D), total / (b.bx * b.by));
    b.bn = std::min(N, total / (b.bx * b.by * b.bz));
    b.rows = b.bx * b.by * b.bz * b.bn;
    b.tx = (W + b.bx - 1) / b.bx;
    b.ty = (H + b.by - 1) / b.by;
    b.tz = (D + b.bz - 1) / b.bz;
    b.tn = (N + b.bn - 1) / b.bn;
    return b;
}

PFN_cuTensorMapEncodeTiled_v12000 encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
    }
    return fn;
}

CUtensorMapSwizzle swizzle_enum(int row_bytes) {
    return row_bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B
                            : (row_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
}

// NDHWC BF16 activation map: dims (C, W, H, D, N), box (cbox, bx, by, bz, bn).
int encode_act(CUtensorMap* tm, const void* p, const sg_conv_shape& s, int C, int cbox, const BoxDims& b) {
    auto enc = encoder();
    LDG_REQUIRE(enc, LDG_ERR_CUDA, "cuTensorMapEncodeTiled entry point unavailable");
    cuuint64_t dims[5] = {(cuuint64_t)C, (cuuint64_t)s.W, (cuuint64_t)s.H, (cuuint64_t)s.D, (cuuint64_t)s.N};
    cuuint64_t strides[4] = {(cuuint64_t)C * 2, (cuuint64_t)C * 2 * s.W, (cuuint64_t)C * 2 * s.W * s.H,
                             (cuuint64_t)C * 2 * s.W * s.H * s.D};
    cuuint32_t box[5] = {(cuuint32_t)cbox, (cuuint32_t)b.bx, (cuuint32_t)b.by, (cuuint32_t)b.bz, (cuuint32_t)b.bn};
    cuuint32_t es[5] = {1, 1, 1, 1, 1};
    CUresult r = enc(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(p), dims, strides, box, es,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_enum(cbox * 2), CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("conv3d: activation tensor map encoding failed: " + std::to_string((int)r));
        return LDG_ERR_CUDA;
    }
    return LDG_OK;
}

// Weight map [Co][27][Ci]: dims (Ci, 27, Co), box (ck, 1, cs).
int encode_w(CUtensorMap* tm, const void* p, int Ci, int Co, int ck, int cs) {
    auto enc = encoder();
    LDG_REQUIRE(enc, LDG_ERR_CUDA, "cuTensorMapEncodeTiled entry point unavailable");
    cuuint64_t dims[3] = {(cuuint64_t)Ci, 27, (cuuint64_t)Co};
    cuuint64_t strides[2] = {(cuuint64_t)Ci * 2, (cuuint64_t)Ci * 2 * 27};
    cuuint32_t box[3] = {(cuuint32_t)ck, 1, (cuuint32_t)cs};
    cuuint32_t es[3] = {1, 1, 1};
    CUresult r = enc(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(p), dims, strides, box, es,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_enum(ck * 2), CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("conv3d: weight tensor map encoding failed: " + std::to_string((int)r));
        return LDG_ERR_CUDA;
    }
    return LDG_OK;
}

bool channels_ok(int c) { return c == 16 || c == 32 || c == 64 || c == 128 || c == 256; }

uint32_t tmem_cols_for(int n) {
    uint32_t c = 32;
    while (c < (uint32_t)n) c *= 2;
    return c;
}

int check_shape(const sg_conv_shape* s, const char* who) {
    LDG_REQUIRE(s, LDG_ERR_ARG, std::string(who) + ": null shape");
    LDG_REQUIRE(s->N >= 1 && s->D >= 1 && s->H >= 1 && s->W >= 1, LDG_ERR_ARG, std::string(who) + ": empty volume");
    LDG_REQUIRE(channels_ok(s->Ci), LDG_ERR_ARG, std::string(who) + ": Ci must be 16, 32, 64, 128 or 256");
    LDG_REQUIRE(s->Co >= 16 && s->Co <= 256 && s->Co % 16 == 0, LDG_ERR_ARG,
                std::string(who) + ": Co must be a multiple of 16 in [16, 256]");
    LDG_REQUIRE((long long)s->N * s->D * s->H * s->W < (1LL << 31), LDG_ERR_ARG, std::string(who) + ": volume too large");
    return LDG_OK;
}

// The march along z where it is the shorter one: the tile is one plane of 128 voxels, the weights
// and the stages fit in shared memory, four accumulators fit in TMEM. Lengths are compared in boxes
// loaded per SM: 27 for each tile of k_conv3d_fwd against nine for each plane of a march, two
// planes more than it stores, and 27 for its weights (a CTA alone on an SM waits more: x 1.3).
template <int CK>
int try_march(const sg_conv_shape& s, const void* x, const void* w, const float* bias, void* y, int act, int f32,
              const BoxDims& b, int sms, cudaStream_t st, bool& taken) {
    taken = false;
    const size_t b_stride = ((size_t)s.Co * CK * 2 + 1023) & ~(size_t)1023;
    constexpr int MS = CK == 64 ? 4 : 6;  // stages
    const size_t smem = 1024 + MS * (size_t)BM * CK * 2 + 27 * b_stride + (2 * MS + 10) * 8 + 16;
    const uint32_t acc = tmem_cols_for(s.Co);
    if (s.Ci != CK || b.bx * b.by != BM || smem > 227 * 1024 || acc * 4 > 512 || s.N > 65535) return LDG_OK;
    const long long cols = (long long)b.tx * b.ty * s.N;
    double best = 27.0 * (double)((cols * s.D + sms - 1) / sms);
    int zlen = 0;
    for (int zs = 1; zs <= s.D && zs <= 65535; ++zs) {
        const int len = (s.D + zs - 1) / zs;
        const long long k = (cols * ((s.D + len - 1) / len) + sms - 1) / sms;
        const double t = ((len + 3) * 9 + 27) * std::max((double)k, 1.3);
        if (t < best) best = t, zlen = len;
    }
    if (!zlen) return LDG_OK;
    MarchArgs a{};
    a.D = s.D; a.H = s.H; a.W = s.W; a.Co = s.Co;
    a.bx = b.bx; a.by = b.by; a.tx = b.tx; a.ty = b.ty;
    a.zlen = zlen; a.act = act; a.out_f32 = f32;
    a.acc_cols = acc; a.tmem_cols = 4 * acc;
    CUtensorMap tmx, tmw;
    int rc = encode_act(&tmx, x, s, CK, CK, b);
    if (rc) return rc;
    if ((rc = encode_w(&tmw, w, CK, s.Co, CK, s.Co))) return rc;
    LDG_CUDA(cudaFuncSetAttribute(k_conv3d_march<CK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const dim3 grid((unsigned)(b.tx * b.ty), (unsigned)((s.D + zlen - 1) / zlen), (unsigned)s.N);
    k_conv3d_march<CK><<<grid, 192, smem, st>>>(tmx, tmw, y, bias, a, g_err);
    LDG_LAUNCHED("k_conv3d_march");
    g_launches++;
    taken = true;
    return LDG_OK;
}

template <int CK>
int launch_fwd(const sg_conv_shape& s, const void* x, const void* w, const float* bias, void* y, int act, int f32,
               cudaStream_t st) {
    FwdArgs a{};
    a.N = s.N; a.D = s.D; a.H = s.H; a.W = s.W; a.Ci = s.Ci; a.Co = s.Co;
    a.b = make_box(s.N, s.D, s.H, s.W, BM);
    a.act = act;
    a.out_f32 = f32;
    a.ksteps = 27 * (s.Ci / CK);
    const long long tiles = (long long)a.b.tx * a.b.ty * a.b.tz * a.b.tn;
    LDG_REQUIRE(tiles < (1LL << 31), LDG_ERR_ARG, "conv3d: too many tiles");
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    bool taken = false;
    int rc = try_march<CK>(s, x, w, bias, y, act, f32, a.b, sms, st, taken);
    if (rc || taken) return rc;
    // Where the tiles leave most SMs idle, a tile's output channels are shared out over CTAs (no
    // fewer than 64 each: every CTA loads the whole input tile). 256 -> 256 channels on 8^3 x 8 has
    // 32 tiles: 42 us undivided, 25 in four.
    int slices = 1;
    while (tiles * slices * 2 <= sms && s.Co % (slices * 32) == 0 && s.Co / (slices * 2) >= 64) slices *= 2;
    a.cs = s.Co / slices;
    a.tmem_cols = tmem_cols_for(a.cs);
    CUtensorMap tmx, tmw;
    rc = encode_act(&tmx, x, s, s.Ci, CK, a.b);
    if (rc) return rc;
    rc = encode_w(&tmw, w, s.Ci, s.Co, CK, a.cs);
    if (rc) return rc;
    const size_t b_stride = ((size_t)a.cs * CK * 2 + 1023) & ~(size_t)1023;
    const size_t smem = 1024 + STAGES * ((size_t)BM * CK * 2 + b_stride) + (2 * STAGES + 1) * 8 + 16;
    LDG_CUDA(cudaFuncSetAttribute(k_conv3d_fwd<CK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k_conv3d_fwd<CK><<<dim3((unsigned)tiles, (unsigned)slices), 128, smem, st>>>(tmx, tmw, y, bias, a, g_err);
    LDG_LAUNCHED("k_conv3d_fwd");
    g_launches++;
    return LDG_OK;
}

template <int ACA, int ACB>
int launch_wgrad(const sg_conv_shape& s, const void* x, const void* dy, float* dw, cudaStream_t st) {
    WgArgs a{};
    a.N = s.N; a.D = s.D; a.H = s.H; a.W = s.W; a.Ci = s.Ci; a.Co = s.Co;
    a.b = make_box(s.N, s.D, s.H, s.W, KV);
    a.nkb = (long long)a.b.tx * a.b.ty * a.b.tz * a.b.tn;
    a.tmem_cols = tmem_cols_for(s.Co);
    const int mtiles = (s.Ci > BM) ? 27 * (s.Ci / BM) : (27 + (BM / s.Ci) - 1) / (BM / s.Ci);
    CUtensorMap tmx, tmdy;
    BoxDims bk = a.b;
    int rc = encode_act(&tmx, x, s, s.Ci, ACA, bk);
    if (rc) return rc;
    rc = encode_act(&tmdy, dy, s, s.Co, ACB, bk);
    if (rc) return rc;
    const size_t b_stride = ((size_t)s.Co * KV * 2 + 1023) & ~(size_t)1023;
    const size_t smem = 1024 + WG_STAGES * ((size_t)BM * KV * 2 + b_stride) + (2 * WG_STAGES + 1) * 8 + 16;
    LDG_CUDA(cudaFuncSetAttribute(k_conv3d_wgrad<ACA, ACB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int dev = 0, sms = 148, per_sm = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    LDG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_conv3d_wgrad<ACA, ACB>, 128, smem));
    const long long slots = (long long)sms * std::max(1, std::min(per_sm, 512 / (int)a.tmem_cols));
    // Split K so the grid covers every SM about twice; at least 8 K boxes per CTA.
    long long splits = std::max(1LL, (2LL * sms + mtiles - 1) / mtiles);
    splits = std::min(splits, std::max(1LL, a.nkb / 8));
    // Small volumes (at most 64 boxes a CTA) are split up to twice as often where that takes
    // fewer or shorter waves: 256 -> 256 channels, 8^3 x 8, is 324 CTAs in 148 places otherwise. A
    // split is never coarser, since a longer accumulation loses precision.
    const long long coarse = splits;
    long long best = -1;
    for (long long c = coarse; c <= 2 * coarse && (c == coarse || (a.nkb + coarse - 1) / coarse <= 64); ++c) {
        const long long boxes = (a.nkb + c - 1) / c, waves = (mtiles * ((a.nkb + boxes - 1) / boxes) + slots - 1) / slots;
        if (best < 0 || waves * (boxes + kWgFixed) < best) best = waves * (boxes + kWgFixed), splits = c;
    }
    a.kb_per_cta = (int)((a.nkb + splits - 1) / splits);
    splits = (a.nkb + a.kb_per_cta - 1) / a.kb_per_cta;
    LDG_CUDA(cudaMemsetAsync(dw, 0, (size_t)s.Co * 27 * s.Ci * sizeof(float), st));
    dim3 grid((unsigned)mtiles, (unsigned)splits);
    k_conv3d_wgrad<ACA, ACB><<<grid, 128, smem, st>>>(tmx, tmdy, dw, a, g_err);
    LDG_LAUNCHED("k_conv3d_wgrad");
    g_launches++;
    return LDG_OK;
}

template <int ACA>
int wgrad_dispatch_b(const sg_conv_shape& s, const void* x, const void* dy, float* dw, cudaStream_t st) {
    if (s.Co == 16) return launch_wgrad<ACA, 16>(s, x, dy, dw, st);
    if (s.Co == 32) return launch_wgrad<ACA, 32>(s, x, dy, dw, st);
    LDG_REQUIRE(s.Co % 64 == 0, LDG_ERR_ARG, "conv3d wgrad: Co must be 16, 32 or a multiple of 64");
    return launch_wgrad<ACA, 64>(s, x, dy, dw, st);
}

}  // namespace

extern "C" {

int sg_conv3d_fwd(const sg_conv_shape* s, const void* x, const void* w, const float* bias, void* y, int act,
                  int y_fp32, void* stream) {
    clear_error();
    int rc = check_shape(s, "sg_conv3d_fwd");
    if (rc) return rc;
    LDG_REQUIRE(x && w && y, LDG_ERR_ARG, "sg_conv3d_fwd: null pointer");
    LDG_REQUIRE(act == 0 || act == 1, LDG_ERR_ARG, "sg_conv3d_fwd: act must be 0 or 1");
    std::lock_guard<std::mutex> lk(g_mu);
    if ((rc = ensure_err())) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    if (s->Ci == 16) return launch_fwd<16>(*s, x, w, bias, y, act, y_fp32, st);
    if (s->Ci == 32) return launch_fwd<32>(*s, x, w, bias, y, act, y_fp32, st);
    return launch_fwd<64>(*s, x, w, bias, y, act, y_fp32, st);
}

int sg_conv3d_wgrad(const sg_conv_shape* s, const void* x, const void* dy, float* dw, void* stream) {
    clear_error();
    int rc = check_shape(s, "sg_conv3d_wgrad");
    if (rc) return rc;
    LDG_REQUIRE(x && dy && dw, LDG_ERR_ARG, "sg_conv3d_wgrad: null pointer");
    std::lock_guard<std::mutex> lk(g_mu);
    if ((rc = ensure_err())) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    if (s->Ci == 16) return wgrad_dispatch_b<16>(*s, x, dy, dw, st);
    if (s->Ci == 32) return wgrad_dispatch_b<32>(*s, x, dy, dw, st);
    return wgrad_dispatch_b<64>(*s, x, dy, dw, st);
}

int sg_conv3d_flip_weights(const sg_conv_shape* s, const void* w, void* wf, void* stream) {
    clear_error();
    LDG_REQUIRE(s && w && wf, LDG_ERR_ARG, "sg_conv3d_flip_weights: null argument");
    LDG_REQUIRE(s->Ci >= 1 && s->Co >= 1 && s->Co <= 65535 * 32 && s->Ci <= 65535 * 32, LDG_ERR_ARG,
                "sg_conv3d_flip_weights: channels out of range");
    const dim3 grid(27, (unsigned)((s->Ci + 31) / 32), (unsigned)((s->Co + 31) / 32));
    k_flip_weights<<<grid, 256, 0, (cudaStream_t)stream>>>(
        static_cast<const __nv_bfloat16*>(w), static_cast<__nv_bfloat16*>(wf), s->Ci, s->Co);
    LDG_LAUNCHED("k_flip_weights");
    std::lock_guard<std::mutex> lk(g_mu);
    g_launches++;
    return LDG_OK;
}

// Doubles of scratch that sg_conv3d_act_grad needs.
long long sg_conv3d_act_grad_ws(long long nvox, int C) {
    return (C >= 16 && C <= 256 && C % 16 == 0 && nvox >= 1) ? (long long)act_grad_blocks(nvox, C) * C : 0;
}

// g = BF16(gy * leaky-ReLU mask of y) (y null: no mask; g null: sums only), db = channel sums of g.
int sg_conv3d_act_grad(long long nvox, int C, const void* y, const void* gy, int fp32, void* g, float* db, double* ws,
                       void* stream) {
    clear_error();
    LDG_REQUIRE(nvox >= 1 && C >= 16 && C <= 256 && C % 16 == 0, LDG_ERR_ARG,
                "sg_conv3d_act_grad: channels must be a multiple of 16 in [16, 256], and the volume not empty");
    LDG_REQUIRE(gy && db && ws, LDG_ERR_ARG, "sg_conv3d_act_grad: null pointer");
    LDG_REQUIRE((((uintptr_t)y | (uintptr_t)gy | (uintptr_t)g) & 15) == 0, LDG_ERR_ARG,
                "sg_conv3d_act_grad: pointers must be 16-byte aligned");
    const int rc = fp32 ? launch_act_grad<float>(nvox, C, y, gy, g, db, ws, (cudaStream_t)stream)
                        : launch_act_grad<__nv_bfloat16>(nvox, C, y, gy, g, db, ws, (cudaStream_t)stream);
    if (rc) return rc;
    std::lock_guard<std::mutex> lk(g_mu);
    g_launches += 2;
    return LDG_OK;
}

// Bytes of scratch that sg_conv3d_bwd needs, 256-byte aligned parts: g, the flipped weights, partial sums.
static size_t bwd_part(size_t b) { return (b + 255) & ~(size_t)255; }
long long sg_conv3d_bwd_ws(const sg_conv_shape* s) {
    if (!s || s->N < 1 || s->D < 1 || s->H < 1 || s->W < 1 || s->Ci < 1 || s->Co < 1) return 0;
    const long long nvox = (long long)s->N * s->D * s->H * s->W;
    return (long long)(bwd_part((size_t)nvox * s->Co * 2) + bwd_part((size_t)s->Ci * 27 * s->Co * 2)) +
           sg_conv3d_act_grad_ws(nvox, s->Co) * (long long)sizeof(double);
}

// All gradients of a layer, from its input x, weights w, output y (null: no activation) and output
// gradient gy, in one call (dx null: not wanted): on small volumes the four separate calls took
// longer to make than their kernels to run.
int sg_conv3d_bwd(const sg_conv_shape* s, const void* x, const void* w, const void* y, const void* gy, int fp32, void* dx,
                  float* dw, float* db, void* ws, void* stream) {
    clear_error();
    int rc = check_shape(s, "sg_conv3d_bwd");
    if (rc) return rc;
    LDG_REQUIRE(x && w && gy && dw && db && ws, LDG_ERR_ARG, "sg_conv3d_bwd: null pointer");
    const long long nvox = (long long)s->N * s->D * s->H * s->W;
    unsigned char* p = static_cast<unsigned char*>(ws);
    void* g = p;
    void* wf = p += bwd_part((size_t)nvox * s->Co * 2);
    double* part = reinterpret_cast<double*>(p + bwd_part((size_t)s->Ci * 27 * s->Co * 2));
    const bool same = !y && !fp32;  // the output gradient as it is
    if ((rc = sg_conv3d_act_grad(nvox, s->Co, y, gy, fp32, same ? nullptr : g, db, part, stream))) return rc;
    const void* go = same ? gy : g;
    if (dx) {
        if ((rc = sg_conv3d_flip_weights(s, w, wf, stream))) return rc;
        sg_conv_shape t = *s;
        t.Ci = s->Co;
        t.Co = s->Ci;
        if ((rc = sg_conv3d_fwd(&t, go, wf, nullptr, dx, 0, 0, stream))) return rc;
    }
    return sg_conv3d_wgrad(s, x, go, dw, stream);
}

// Reads and clears the device error word of the conv kernels (synchronises the stream).
int sg_check(void* stream) {
    clear_error();
    std::lock_guard<std::mutex> lk(g_mu);
    int rc = ensure_err();
    if (rc) return rc;
    int e = 0;
    LDG_CUDA(cudaMemcpyAsync(&e, g_err, sizeof(int), cudaMemcpyDeviceToHost, (cudaStream_t)stream));
    LDG_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
    if (e) {
        LDG_CUDA(cudaMemsetAsync(g_err, 0, sizeof(int), (cudaStream_t)stream));
        LDG_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
        set_error("conv3d: a bounded pipeline wait gave up");
        return LDG_ERR_TIMEOUT;
    }
    return LDG_OK;
}

long long sg_launch_count(void) {
    std::lock_guard<std::mutex> lk(g_mu);
    return g_launches;
}

}  // extern "C"
