// Tiled confined-solver step kernel for sm_100a.
//
// A CTA owns a (TJ x TK) column tile of the (j, k) plane and marches along i over a chunk
// of planes. Each plane of the input field arrives in shared memory through one TMA load
// of a 4-D box (k, j, i, component) covering the tile plus its halo (the k start stays on a 16-byte
// boundary), so every Q value is read from HBM about once. The ring holds the planes that the cells
// of plane i read, plus planes in flight. Interior cells read only Q: the L2 term's derivatives of
// the column divergence are evaluated from Q directly (wide and four-corner second differences,
// which for an interior cell equal the reference's central differences of its central divergence),
// so no divergence field is staged and the warps share nothing but the plane ring. Each warp
// therefore marches on its own: it waits only for the TMA of the planes it reads, and when it
// is done with a plane it arrives on that slot's counter; the warp whose arrival completes the
// count issues the load of the plane that reuses the slot. There is no CTA barrier per plane.
// Rows with cells next to a grid face take the reference's face stencils in the same undivided
// form with neighbours clamped to the grid. Per cell the kernel evaluates the chemical potential and
// the update from shared memory and writes only the cells that change (moving and strongly anchored
// cells): frozen exterior cells hold identical values in both ping-pong buffers. Tiles that contain
// no changing cell are never visited (host-built work list). The same per-tile routine drives a
// persistent, work-stealing ensemble kernel over many droplets.
//
// What bounds it. With L2 and L3 the issue slots: 372 instructions per visited cell at 61 % issue
// efficiency, 170 of them on the FMA pipe, which is busy 48 % of the time. L1 only: the loads and stores (182
// instructions a cell at 55 %, the warps wait for their planes; a 256^3 step with its arithmetic left out
// took 87 of 89 us). A grid of few tiles: the serial march of one item (about 1 us per plane), hence
// tiled_length, and the launch gap, hence the programmatic dependent launches (2 us a step). Per step, one
// work-list length for all before -> now: 256^3, R = 120, with all terms 168 -> 147 us, L1 only (R = 115)
// 101 -> 76 us, 64^3 16.4 -> 5.1 us, 32^3 14.4 -> 3.0 us, 101 x 90 x 117 touching its faces with all terms
// 61.5 -> 17.5 us, with compensated storage 67.6 -> 21.3 us.
//
// mbarrier waits are bounded: on timeout the kernel records LDG_ERR_TIMEOUT in a device
// word, waits (bounded) for its own TMA loads and returns.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <climits>
#include <cmath>
#include <cstdint>
#include <limits>
#include <string>
#include <vector>

#include "ldg_api_common.h"
#include "ldg_common.cuh"

namespace ldg {

namespace tiled {

constexpr int TK = 32;               // tile width along k (one warp per row)
constexpr int TJ = 8;                // tile rows along j
constexpr int THREADS = TK * TJ / 2;  // two cells per thread: rows 2w and 2w + 1 of warp w
constexpr int NWARP = THREADS / 32;
// What the kernels keep of a plane in shared memory. The L2 term reads two cells out (wide second
// differences): two halo rows and the planes i-2 .. i+2. Without it the stencil reaches one cell: one
// halo row and the planes i-1 .. i+1, so a ring has more planes in flight.
// A TMA box starts at column k0 - HK, which must be a multiple of 4 floats (16 bytes). Without L2 the
// tiles start on 8 floats and HK is 4: every row a warp stores is made of whole 32-byte sectors (rows
// are padded to 8 floats). Stores that cut sectors bound the L1-only step: the same loads and stores
// without arithmetic took 164 us with cut and 110 us with whole sectors on a 256^3 box. With L2, a
// plane of 40 columns would let only three blocks share an SM, and that step is bound by
// arithmetic: its tiles start at k0 = 2 (mod 4) with HK = 2 (the first may start at k0 = -2: columns
// outside the grid are zero fill and compute nothing).
// A sweep's slot also holds the tile of the right-hand side.
enum Mode { kStep, kRhs, kSweep, kSweepLast };  // explicit step; IMEX right-hand side; Jacobi sweep, the last one
template <bool kL2, int kMode = kStep>
struct Tile {
    static constexpr bool kHasRhs = kMode >= kSweep;
    static constexpr int H = kL2 ? 2 : 1;             // halo rows and planes read on each side
    static constexpr int HK = kL2 ? 2 : 4;            // halo columns
    static constexpr int RW = TK + 2 * HK;            // floats per shared row
    static constexpr int ROWS = TJ + 2 * H;
    static constexpr int CSTR = RW * ROWS;            // floats per component plane
    static constexpr int PLANE = 5 * CSTR;            // floats per plane (all components)
    static constexpr int RHS = (PLANE + 31) / 32 * 32;            // right-hand side (128-byte aligned)
    static constexpr int MASKS = kHasRhs ? RHS + 5 * TK * TJ : PLANE;
    static constexpr int SLOT = (MASKS + 4 * TJ + 31) / 32 * 32;  // floats per ring slot (128-byte aligned)
    static constexpr uint32_t BYTES = PLANE * 4, RHS_BYTES = kHasRhs ? 5 * TK * TJ * 4 : 0;
    // ring slots: planes i-H .. i+H are read at plane i, the rest are in flight
    static constexpr int NQ = kL2 ? 6 : (kHasRhs ? 4 : 5);
};
// CTAs per SM the register budget is set for.
template <bool kL2, bool kL3, int kMode = kStep>
__host__ __device__ constexpr int ctas() { return kL2 || kL3 || kMode >= kSweep ? 4 : 5; }

// What a warp does with one row of 32 cells of one plane, one bit per cell. They are formed once per
// work list from the cell classes and travel through the ring with their plane (one bulk copy on
// the plane's mbarrier): the classes themselves, one global byte load per cell and plane, had to
// be fetched a plane ahead by every thread, and their latency was exposed at every plane of a march.
struct RowMask {
    uint32_t move, fixed, anchor;  // kMove; kFixed; kMove && kAnchor
    uint32_t face;                 // kMove next to a grid face: the row takes the face stencils
};
constexpr uint32_t MASK_BYTES = TJ * sizeof(RowMask);

// One work item: the tile at (j0, k0) over planes [ib, ie) of droplet `inst`; `rec` is the index of
// its first plane's masks.
struct TileItem {
    int j0, k0, ib, ie, inst, rec, pad0, pad1;
};
constexpr int CHUNK = 12;            // planes per work item of a full work list (tiled_length)
constexpr long long WAIT_CLK = 4000000000ll;  // about 2 s per wait
constexpr long long DRAIN_CLK = 40000000ll;   // about 20 ms per slot after an abort

__device__ __forceinline__ uint32_t su32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* b, uint32_t n) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(su32(b)), "r"(n) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(uint64_t* b, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(su32(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* b) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(su32(b)) : "memory");
}
// One bounded try: the thread may wait in the barrier for a system-dependent time before the
// try returns false. (A suspend-time hint of 1 ms made the two-cell steps 1-2 % slower.)
__device__ __forceinline__ bool mbar_try_wait(uint64_t* b, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(su32(b)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Waits for the phase with the given parity, giving up after WAIT_CLK cycles or when another warp
// of the CTA gave up.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* b, uint32_t parity, const int* abort) {
    if (mbar_try_wait(b, parity)) return true;
    const long long t0 = clock64();
    while (true) {
        if (mbar_try_wait(b, parity)) return true;
        if (*(const volatile int*)abort || clock64() - t0 > WAIT_CLK) return false;
    }
}
// After an abort: waits for a copy that may be in flight, for a bounded time.
__device__ __forceinline__ void drain_bounded(uint64_t* b, uint32_t parity) {
    const long long t0 = clock64();
    while (!mbar_try_wait(b, parity))
        if (clock64() - t0 > DRAIN_CLK) return;
}
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* tm, int c0, int c1, int c2, int c3,
                                            uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
        "[%6];" ::"r"(su32(dst)),
        "l"(tm), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(su32(bar))
        : "memory");
}

// 16-byte shared load that is not merged with an earlier one of the same address.
__device__ __forceinline__ uint4 lds_u4(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
// Untiled bulk copy (16-byte aligned addresses, size a multiple of 16).
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     su32(dst)),
                 "l"(src), "r"(bytes), "r"(su32(bar))
                 : "memory");
}

// Shared-memory Q accessor centred on a cell of plane i; planes i-2..i+2 (i-1..i+1 without the L2 term).
template <bool kL2>
struct SmemQ {
    const float* pl[5];
    int off;
    __device__ __forceinline__ float operator()(int c, int di, int dj, int dk) const {
        return pl[di + 2][off + dj * Tile<kL2>::RW + dk + c * Tile<kL2>::CSTR];
    }
};
// The same with runtime offsets (face cells): the plane is picked from the five by selects.
struct SmemQRt {
    const float* pl[5];
    int off;
    __device__ __forceinline__ float operator()(int c, int di, int dj, int dk) const {
        const float* s = di == 0 ? pl[2] : (di > 0 ? (di == 1 ? pl[3] : pl[4]) : (di == -1 ? pl[1] : pl[0]));
        return s[off + dj * Tile<true>::RW + dk + c * Tile<true>::CSTR];
    }
};
// Face cells without the L2 term read the field itself: the shifted second difference of a cell on
// a face reaches two cells in, one more than the one-cell halo holds. Plain loads (pdl_wait).
struct GlobQRt {
    const float* q;  // component 0 of the cell
    long long sc, si;
    int sj;
    __device__ __forceinline__ float operator()(int c, int di, int dj, int dk) const {
        return q[c * sc + di * si + (long long)dj * sj + dk];
    }
};

// Chemical potential of one cell of a row that has cells next to a grid face. The cell is in the
// grid: every stencil position is clamped to it. One cell at a time: the packed form of both rows
// needs about twice the registers for the runtime offsets and spilled (101 x 90 x 117 box, default
// radius: 23.5 against 21.5 us a step).
template <bool kL2, bool kL3, bool kLap>
__device__ __forceinline__ void chem_face(const SmemQ<kL2>& A, int row, const float* qin, const QsrConst& P, int i, int j,
                                          int k, const float q[5], float mu[5], float lap[5]) {
    const FaceAxis x(i, P.Nx), y(j, P.Ny), z(k, P.Nz);
    const bool inner = i > 0 && i < P.Nx - 1 && j > 0 && j < P.Ny - 1 && k > 0 && k < P.Nz - 1;
    if constexpr (kL2) {
        SmemQRt R;
#pragma unroll
        for (int d = 0; d < 5; ++d) R.pl[d] = A.pl[d];
        R.off = A.off + row * Tile<kL2>::RW;
        const FaceOne<kL2, kL3, SmemQRt> S{R, x, y, z};
        chem_core<kL2, kL3, kLap, true, float>(S, P, q, inner ? 1.0f : 0.0f, mu, lap);
    } else {
        const GlobQRt R{qin + (long long)i * P.si + (long long)j * P.sj + k, P.sc, P.si, P.sj};
        const FaceOne<kL2, kL3, GlobQRt> S{R, x, y, z};
        chem_core<kL2, kL3, kLap, true, float>(S, P, q, inner ? 1.0f : 0.0f, mu, lap);
    }
}

// Shared-memory layout of one CTA of the tiled kernels.
struct TileSmem {
    float* sq;          // NQ slots: a plane of Q (tile + halo, 5 components) and its row masks
    uint64_t* bar;      // NQ mbarriers, one per slot (copy completion)
    unsigned* freed;    // NQ counters of warps done with the slot's plane
    int* s_abort;       // set when a bounded wait gave up
    int* s_item;        // work item broadcast (persistent kernel)
};

template <bool kL2, int kMode = kStep>
__device__ __forceinline__ TileSmem tile_smem(unsigned char* raw) {
    using G = Tile<kL2, kMode>;
    TileSmem S;
    S.sq = reinterpret_cast<float*>(raw);
    S.bar = reinterpret_cast<uint64_t*>(S.sq + G::NQ * G::SLOT);
    S.freed = reinterpret_cast<unsigned*>(S.bar + G::NQ);
    S.s_abort = reinterpret_cast<int*>(S.freed + G::NQ);
    S.s_item = S.s_abort + 1;
    return S;
}
template <bool kL2, int kMode = kStep>
__host__ __device__ constexpr size_t tile_smem_bytes() {
    return (size_t)Tile<kL2, kMode>::NQ * (Tile<kL2, kMode>::SLOT * 4 + 8 + 4) + 16;
}

// A warp's arrival on a slot counter: returns the count before it (acquire-release at CTA
// scope, so the warp's reads of the plane happen before the slot is refilled).
__device__ __forceinline__ unsigned arrive_freed(unsigned* ctr) {
    unsigned old;
    asm volatile("atom.acq_rel.cta.shared::cta.add.u32 %0, [%1], 1;" : "=r"(old) : "r"(su32(ctr)) : "memory");
    return old;
}

// One work item: the (TJ x TK) column tile at (j0, k0) over planes [ib, ie), `masks` the RowMasks of
// its planes. `phase` holds the parity of the next phase of every slot barrier (bit s for slot s),
// so a CTA can run many items in a row; every copy the item issues is waited for by every warp
// before it returns. Returns false when a bounded wait gave up (the CTA must stop). The caller
// synchronises the CTA before and after an item.
// Each thread updates two cells (rows 2w and 2w + 1 of warp w): their chemical potential runs as one
// packed (FFMA2 / FADD2 / FMUL2) instruction stream, and adjacent rows share operands (the centre of
// one is a j-neighbour of the other). kComp: compensated storage (explicit steps only): the low words
// of the input cells are read from lo_in and the new low words written to lo_out.
template <bool kL2, bool kL3, bool kNoise, int kMode, bool kComp = false>
__device__ __forceinline__ bool process_tile(const CUtensorMap* tm, const float* qin,
                                             float* __restrict__ qout, const RowMask* __restrict__ masks, int j0,
                                             int k0, int ib, int ie, const QsrConst& P, const TileSmem& S,
                                             uint32_t& phase, int* __restrict__ err,
                                             const float* lo_in = nullptr, float* __restrict__ lo_out = nullptr,
                                             const CUtensorMap* tm_rhs = nullptr) {
    using G = Tile<kL2, kMode>;
    constexpr int H = G::H, SLOT = G::SLOT, NQ = G::NQ, RW = G::RW;
    constexpr bool kRHS = kMode == kRhs, kJacobi = kMode >= kSweep;
    static_assert(NQ > 2 * H + 1, "the ring holds planes i - H .. i + H and at least one in flight");
    static_assert(!kJacobi || !kL2, "a sweep reaches one cell");
    float* sq = S.sq;
    uint64_t* bar = S.bar;
    const int base = ib - H;  // first plane this item loads; slots and phases count from it
    const int tid = threadIdx.x;
    const int kl = tid & 31, w = tid >> 5;
    // Plane p (p >= base) lives in slot (p - base) % NQ.
    auto slot = [&](int p) { return (uint32_t)(p - base) % (uint32_t)NQ; };
    // Planes outside the grid, and planes past the last one this item reads (ie - 1 + H), complete
    // their phase with a plain arrive (no data). The planes of the item bring their row masks.
    auto issue = [&](int p, uint32_t sl) {
        uint64_t* b = &bar[sl];
        if (p >= 0 && p < P.Nx && p < ie + H) {
            const bool own = p >= ib && p < ie;
            float* dst = sq + sl * SLOT;
            fence_proxy_async();
            mbar_expect_tx(b, G::BYTES + (own ? MASK_BYTES + G::RHS_BYTES : 0u));
            tma_load_4d(dst, tm, k0 - G::HK, j0 - H, p, 0, b);
            if (own) {
                bulk_load(dst + G::MASKS, masks + (size_t)(p - ib) * TJ, MASK_BYTES, b);
                if (kJacobi) tma_load_4d(dst + G::RHS, tm_rhs, k0, j0, p, 0, b);
            }
        } else {
            mbar_arrive(b);
        }
    };
    if (tid == 0)
        for (int p = base; p < base + NQ; ++p) issue(p, slot(p));
    bool ok = true;
    // Waits run in increasing plane order, so each slot's expected parity is tracked by toggling
    // its bit of `par` after every wait on it (no division per plane).
    uint32_t par = phase;
    auto wait_slot = [&](uint32_t sl) {
        if (!mbar_wait_bounded(&bar[sl], (par >> sl) & 1u, S.s_abort)) {
            atomicExch(err, LDG_ERR_TIMEOUT);
            *(volatile int*)S.s_abort = 1;
            ok = false;
        }
        par ^= 1u << sl;
    };
    // Planes [base, ie + NQ - H) are issued: the first NQ here, then plane p + NQ when the last
    // warp is done with plane p (after its plane p + H), for every p <= ie - H - 1.
    const int issued_end = ie + NQ - H;
    const int j = j0 + 2 * w, k = k0 + kl;
    const uint32_t bit = 1u << kl;
    const int off = (2 * w + H) * RW + kl + G::HK;
    long long id = (long long)ib * P.si + (long long)j * P.sj + k;  // row j; row j + 1 is P.sj further
    // Shared-memory planes i-H .. i+H of the current step, rolled forward by one plane per step.
    const float* qpl[5];
#pragma unroll
    for (int d = 2 - H; d <= 2 + H; ++d) qpl[d] = sq + slot(ib + d - 2) * SLOT;
    for (int p = base; p < ib + H; ++p) wait_slot(slot(p));
    int waited_end = ib + H;
    uint32_t s_w = slot(ib + H);  // slot of plane i + H, advanced by one per plane
    for (int i = ib; i < ie; ++i, id += P.si) {
        wait_slot(s_w);
        waited_end = i + H + 1;
        if (!__all_sync(0xffffffffu, ok)) break;  // the whole warp stops or none of it
        // The masks are read again after the chemical potential: eight registers fewer live across it.
        const uint32_t mk = su32(qpl[2] + G::MASKS) + 2 * w * sizeof(RowMask);
        uint4 m0 = lds_u4(mk), m1 = lds_u4(mk + sizeof(RowMask));
        if ((m0.x | m1.x) != 0u || (!kRHS && (m0.y | m1.y) != 0u)) {
            SmemQ<kL2> A;
#pragma unroll
            for (int d = 2 - H; d <= 2 + H; ++d) A.pl[d] = qpl[d];
            A.off = off;
            F2 c[5], mu[5], lap[5];
#pragma unroll
            for (int m = 0; m < 5; ++m) c[m] = mk2(A(m, 0, 0, 0), A(m, 0, 1, 0));
            // the chemical potential, then the new values of both cells (compensated storage keeps the potential)
            if constexpr (kJacobi) {
                // (I - alpha Lap) Q = rhs with the centre term on the left (QSR.cu:786-849); cells on a grid face hold
                const float* rh = qpl[2] + G::RHS + 2 * w * TK + kl;
                const uint32_t up0 = m0.x & ~m0.w & bit, up1 = m1.x & ~m1.w & bit;
#pragma unroll
                for (int m = 0; m < 5; ++m) {
                    const F2 sx = mk2(A(m, 1, 0, 0), A(m, 1, 1, 0)) + mk2(A(m, -1, 0, 0), A(m, -1, 1, 0));
                    const F2 sy = mk2(c[m].v.y + A(m, 0, -1, 0), A(m, 0, 2, 0) + c[m].v.x);
                    const F2 sz = mk2(A(m, 0, 0, 1), A(m, 0, 1, 1)) + mk2(A(m, 0, 0, -1), A(m, 0, 1, -1));
                    const F2 r = mk2(rh[m * TK * TJ], rh[m * TK * TJ + TK]);
                    const F2 v = P.jdenom_inv * vfma(P.alpha, vfma(P.ix2, sx, vfma(P.iy2, sy, P.iz2 * sz)), r);
                    mu[m] = mk2(up0 ? v.v.x : c[m].v.x, up1 ? v.v.y : c[m].v.y);
                }
            } else {
                if ((m0.w | m1.w) == 0u) {
                    const InteriorPair<kL2, kL3, SmemQ<kL2>> St{A};
                    chem_core<kL2, kL3, kRHS, false, F2>(St, P, c, F2{}, mu, lap);
                } else {
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        float cr[5], mr[5], lr[5];
#pragma unroll
                        for (int m = 0; m < 5; ++m) cr[m] = mr[m] = lr[m] = r ? c[m].v.y : c[m].v.x;
                        if ((r ? m1.x : m0.x) & bit) chem_face<kL2, kL3, kRHS>(A, r, qin, P, i, j + r, k, cr, mr, lr);
#pragma unroll
                        for (int m = 0; m < 5; ++m) {
                            (r ? mu[m].v.y : mu[m].v.x) = mr[m];
                            if (kRHS) (r ? lap[m].v.y : lap[m].v.x) = lr[m];
                        }
                    }
                }
                m0 = lds_u4(mk);
                m1 = lds_u4(mk + sizeof(RowMask));
                if ((m0.z | m1.z) != 0u) {  // weak-anchoring penalty (QSR.cu:623-652)
                    float Qa[5], Qb[5];
                    surface_q0(P, i, j, k, Qa);
                    surface_q0(P, i, j + 1, k, Qb);
                    const F2 wf = mk2((m0.z & bit) ? P.Weff : 0.0f, (m1.z & bit) ? P.Weff : 0.0f);
#pragma unroll
                    for (int m = 0; m < 5; ++m) mu[m] = vfma(wf, c[m] - mk2(Qa[m], Qb[m]), mu[m]);
                }
                if (kRHS) {
#pragma unroll
                    for (int m = 0; m < 5; ++m) mu[m] = vfma(-P.alpha, lap[m], vfma(-P.mob_dt, mu[m], c[m]));
                } else if (!kComp) {
#pragma unroll
                    for (int m = 0; m < 5; ++m) mu[m] = vfma(-P.mob_dt, mu[m], c[m]);
                }
            }
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const uint32_t mv = r ? m1.x : m0.x, fx = r ? m1.y : m0.y;
                const bool fixed = !kRHS && (fx & bit), move = (mv & bit) != 0u;
                if (!(fixed || move)) continue;
                const long long ir = id + (r ? P.sj : 0);
                float o[5];
#pragma unroll
                for (int m = 0; m < 5; ++m) o[m] = r ? mu[m].v.y : mu[m].v.x;
                if (kJacobi) {
                    if (kMode == kSweepLast && fixed) surface_q0(P, i, j + r, k, o);
                } else if (fixed) {
                    surface_q0(P, i, j + r, k, o);
                    if (kComp) {
#pragma unroll
                        for (int m = 0; m < 5; ++m) lo_out[m * P.sc + ir] = 0.0f;
                    }
                } else if (kComp) {
                    float lo[5], cr[5], mr[5];
#pragma unroll
                    for (int m = 0; m < 5; ++m) {
                        lo[m] = lo_in[m * P.sc + ir];
                        cr[m] = r ? c[m].v.y : c[m].v.x;
                        mr[m] = r ? mu[m].v.y : mu[m].v.x;
                    }
                    euler_update_comp(P, cr, lo, mr, (uint32_t)(k + P.Nz * (j + r + P.Ny * i)), kNoise, o);
#pragma unroll
                    for (int m = 0; m < 5; ++m) lo_out[m * P.sc + ir] = lo[m];
                } else {
                    if (kNoise) {
                        float g[5];
                        normals5((uint32_t)(k + P.Nz * (j + r + P.Ny * i)), P.instance, P.step, P.key0, P.key1, g);
#pragma unroll
                        for (int m = 0; m < 5; ++m) o[m] = fmaf(P.sigma, g[m], o[m]);
                    }
                    if (!kRHS && P.qcap > 0.0f) cap_norm(P.qcap, o);
                }
#pragma unroll
                for (int m = 0; m < 5; ++m) qout[m * P.sc + ir] = o[m];
            }
        }
        // This warp is done with plane i-H: arrive on its slot; the last warp refills the slot with
        // plane i-H+NQ.
        __syncwarp();
        if (kl == 0) {
            // slot of plane i - H = slot of plane i + H minus 2 H
            const uint32_t sl = s_w >= 2u * H ? s_w - 2 * H : s_w + (NQ - 2 * H);
            if (arrive_freed(&S.freed[sl]) % (unsigned)NWARP == (unsigned)NWARP - 1u) issue(i - H + NQ, sl);
        }
        s_w = (s_w + 1 == (uint32_t)NQ) ? 0u : s_w + 1;  // now the slot of plane i + H + 1
#pragma unroll
        for (int d = 2 - H; d < 2 + H; ++d) qpl[d] = qpl[d + 1];
        qpl[2 + H] = sq + s_w * SLOT;
    }
    // Drain: every copy this item issues lands before the slots are reused or released. After
    // an abort some refills are never issued; those waits give up at once.
    for (int p = waited_end; p < issued_end; ++p) {
        if (ok) {
            wait_slot(slot(p));
        } else {
            const uint32_t sl = slot(p);
            drain_bounded(&bar[sl], (par >> sl) & 1u);
            par ^= 1u << sl;
        }
    }
    // Advance the per-slot phase parities by the number of copies each slot received.
    const int n_issued = issued_end - base;
#pragma unroll
    for (int sl = 0; sl < NQ; ++sl) {
        const int uses = (n_issued > sl) ? (n_issued - sl + NQ - 1) / NQ : 0;
        phase ^= (uint32_t)(uses & 1) << sl;
    }
    return ok;
}

template <bool kL2, int kMode = kStep>
__device__ __forceinline__ void tile_smem_init(const TileSmem& S) {
    if (threadIdx.x == 0) {
        for (int s = 0; s < Tile<kL2, kMode>::NQ; ++s) {
            mbar_init(&S.bar[s], 1);
            S.freed[s] = 0;
        }
        mbar_fence_init();
        *S.s_abort = 0;
    }
    __syncthreads();
}

// Single grid: one work item per CTA.
template <bool kL2, bool kL3, bool kNoise, int kMode, bool kComp = false>
__global__ void __launch_bounds__(THREADS, ctas<kL2, kL3>())
    k_step_tiled(const __grid_constant__ CUtensorMap tm_in, const float* qin, float* __restrict__ qout,
                 const RowMask* __restrict__ masks, const TileItem* __restrict__ items, QsrConst P,
                 int* __restrict__ err, const float* lo_in, float* __restrict__ lo_out) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const TileSmem S = tile_smem<kL2>(smem_raw);
    tile_smem_init<kL2>(S);
    const TileItem e = items[blockIdx.x];
    uint32_t phase = 0;
    pdl_wait();
    pdl_trigger();
    process_tile<kL2, kL3, kNoise, kMode, kComp>(&tm_in, qin, qout, masks + (size_t)e.rec * TJ, e.j0, e.k0, e.ib, e.ie,
                                                 P, S, phase, err, lo_in, lo_out);
}

// One Jacobi sweep of (I - alpha Lap) Q = rhs over the changing cells, the field through the same plane
// ring as the step's (one load per value) and the right-hand side's tile beside it. Bound by HBM: at
// 256^3, R = 120, a sweep takes 105 us (135 with one block per tile plane and its loads from global
// memory) and moves 616 MB, 438 MB of them needed: the rest are the tiles' idle cells and halo planes
// that fell out of L2. Tried and slower or no faster: four sweeps per pass in overlapping patches (2.8 ms
// for 25 against 2.7: 2.7 to 4.3 times the cells), the right-hand side by plain loads a plane ahead
// (3.0 ms), a ring of its own for it (2.7 ms). Every other cell never changes:
// it holds the same value in both ping-pong buffers, so the reference's copy of it (QSR.cu:803-810) is
// already done. The last sweep applies the strong-anchoring rewrite (QSR.cu:851-867).
template <int kMode>
__global__ void __launch_bounds__(THREADS, ctas<false, false, kMode>())
    k_sweep_tiled(const __grid_constant__ CUtensorMap tm_in, const __grid_constant__ CUtensorMap tm_rhs,
                  float* __restrict__ qout, const RowMask* __restrict__ masks, const TileItem* __restrict__ items,
                  QsrConst P, int* __restrict__ err) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const TileSmem S = tile_smem<false, kMode>(smem_raw);
    tile_smem_init<false, kMode>(S);
    const TileItem e = items[blockIdx.x];
    uint32_t phase = 0;
    pdl_wait();
    pdl_trigger();
    process_tile<false, false, false, kMode>(&tm_in, nullptr, qout, masks + (size_t)e.rec * TJ, e.j0, e.k0, e.ib, e.ie,
                                             P, S, phase, err, nullptr, nullptr, &tm_rhs);
}

// Row masks of a work list: one block per item, one warp per tile row, a ballot per plane. `lo` is
// the distance from a face from which the interior stencils hold (2 with the L2 term, else 1).
static __global__ void __launch_bounds__(TK* TJ) k_tile_masks(const TileItem* __restrict__ items,
                                                              const uint8_t* __restrict__ flags, int Nx, int Ny, int Nz,
                                                              int sj, long long si, int lo, RowMask* __restrict__ masks) {
    const TileItem e = items[blockIdx.x];
    const int kl = threadIdx.x & 31, row = threadIdx.x >> 5;
    const int j = e.j0 + row, k = e.k0 + kl;
    const bool in = j < Ny && k >= 0 && k < Nz;
    const bool jk = j >= lo && j <= Ny - 1 - lo && k >= lo && k <= Nz - 1 - lo;
    for (int i = e.ib; i < e.ie; ++i) {
        const uint8_t f = in ? flags[(long long)i * si + (long long)j * sj + k] : 0;
        RowMask m;
        m.move = __ballot_sync(0xffffffffu, f & kMove);
        m.fixed = __ballot_sync(0xffffffffu, f & kFixed);
        m.anchor = __ballot_sync(0xffffffffu, (f & kMove) && (f & kAnchor));
        m.face = __ballot_sync(0xffffffffu, (f & kMove) && !(jk && i >= lo && i <= Nx - 1 - lo));
        if (kl == 0) masks[(size_t)(e.rec + i - e.ib) * TJ + row] = m;
    }
}

// ---------------------------------------------------------------------------------------
// Ensemble: many independent droplets, one persistent work-stealing launch per step.
// ---------------------------------------------------------------------------------------
// Per-instance descriptor. The step index lives on the device (EnsCtl), so the temperature of
// the protocol, the shell order and the noise counter are formed in the kernel and one captured
// CUDA graph can be replayed for any number of steps.
struct EnsInstDev {
    QsrConst P;            // static parts (noise key and stream included); cQ, S_shell, step set per step
    float* q[2];           // ping-pong buffers: input of step s is q[s & 1]
    double T_high, T_low;  // protocol (QSR.cu:2679-2687)
    long long pre, ramp;
    int protocol;          // 1 step, 2 linear ramp
    int custom_shell;      // 1: S_shell = S_custom, 0: equilibrium S_eq(T)
    double S_custom;
    double a3, T_star, B, C;  // A = a3 (T - T_star); B, C of the bulk convention
};

struct EnsCtl {
    int next;            // work-stealing counter (reset by the last CTA of a step)
    unsigned int done;   // CTAs finished in this step
    long long step;      // global step index
};

__host__ __device__ __forceinline__ double ens_temperature(const EnsInstDev& D, long long it) {
    if (it < D.pre) return D.T_high;
    if (D.protocol == 1) return D.T_low;
    const long long t = it - D.pre;
    if (t <= 0) return D.T_high;
    if (t >= D.ramp) return D.T_low;
    return D.T_high + (D.T_low - D.T_high) * ((double)t / (double)D.ramp);
}

// Lower-energy positive root of 2 C S^2 - B S + 3 A = 0 (QSR.cu:1391-1418), FP64.
__host__ __device__ __forceinline__ double ens_S_eq(double A, double B, double C) {
    if (!(C > 0.0)) return 0.0;
    const double disc = B * B - 24.0 * A * C;
    if (!(disc > 0.0)) return 0.0;
    const double sd = sqrt(disc);
    double best_S = 0.0, best_f = 0.0;
    const double roots[2] = {(B - sd) / (4.0 * C), (B + sd) / (4.0 * C)};
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const double S = roots[r];
        if (!(S > 0.0)) continue;
        const double S2 = S * S;
        const double f = (A / 3.0) * S2 - (2.0 * B / 27.0) * (S2 * S) + (C / 9.0) * (S2 * S2);
        if (f < best_f) { best_f = f; best_S = S; }
    }
    return best_S;
}

template <bool kL2, bool kL3, bool kNoise>
__global__ void __launch_bounds__(THREADS, ctas<kL2, kL3>())
    k_step_ensemble(const CUtensorMap* __restrict__ tms, const EnsInstDev* __restrict__ inst,
                    const TileItem* __restrict__ items, const RowMask* __restrict__ masks, int n_items,
                    EnsCtl* __restrict__ ctl, int* __restrict__ err) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const TileSmem S = tile_smem<kL2>(smem_raw);
    tile_smem_init<kL2>(S);
    pdl_wait();
    pdl_trigger();
    // Every CTA reads the step index before any CTA of this launch finishes (the last CTA to
    // finish advances it).
    const long long step = *((volatile long long*)&ctl->step);
    const int which = (int)(step & 1);
    uint32_t phase = 0;
    while (true) {
        if (threadIdx.x == 0) *S.s_item = atomicAdd(&ctl->next, 1);
        __syncthreads();
        const int it = *S.s_item;
        // Uniform across the CTA: the item and the abort flag are read between two barriers.
        const bool stop = (it >= n_items) || (*S.s_abort != 0);
        __syncthreads();
        if (stop) break;
        const TileItem e = items[it];
        const EnsInstDev& D = inst[e.inst];
        QsrConst P = D.P;
        const double T = ens_temperature(D, step);
        const double A = D.a3 * (T - D.T_star);
        P.cQ = (float)A;
        if (!D.custom_shell) {
            const double s = ens_S_eq(A, D.B, D.C);
            P.S_shell = (float)(s > 0.0 ? s : 0.0);
        } else {
            P.S_shell = (float)D.S_custom;
        }
        P.step = step;
        process_tile<kL2, kL3, kNoise, kStep>(tms + 2 * e.inst + which, D.q[which], D.q[1 - which],
                                              masks + (size_t)e.rec * TJ, e.j0, e.k0, e.ib, e.ie, P, S, phase, err);
    }
    if (threadIdx.x == 0) {
        __threadfence();
        const unsigned int d = atomicAdd(&ctl->done, 1u);
        if (d == gridDim.x - 1) {
            ctl->next = 0;
            ctl->done = 0;
            ctl->step = step + 1;
            __threadfence();
        }
    }
}

}  // namespace tiled

// One band of TJ rows of the (j, k) plane: for every plane of [ib, ie) the k range [kmin, kmax]
// of its changing cells (kmin > kmax: none).
struct TiledBand {
    int j0 = 0, rows = 0, ib = 0, ie = 0;
    bool face = false;            // changing cells next to a j face
    std::vector<int> kmin, kmax;
};

enum Load { kLoadL1, kLoadDeep, kLoadSweep };  // L1-only step; step with L2 or L3; Jacobi sweep
struct TiledPlan {
    bool ok = false;
    long long active_cells = 0;   // cells inside visited tiles at the current chunk (read once per step)
    long long written_cells = 0;  // cells written per step (moving + strongly anchored)
    int n_items = 0;
    int chunk = 0;                // planes per work item (the longest item)
    tiled::TileItem* items = nullptr;   // device work list
    tiled::RowMask* masks = nullptr;    // row masks of the items' planes
    const uint8_t* flags = nullptr;     // device cell classes
    int Nx = 0, Ny = 0, sj = 0;
    long long si = 0;
    bool L2 = false;              // the kernels take the L2 term (halo, interior distance)
    Load load = kLoadL1;          // what the kernels do (tiled_length)
    int Nz = 0;
    std::vector<TiledBand> bands; // host: the changing cells' extent per row band and plane
    int* err = nullptr;           // device error word
    CUtensorMap tmap[2];
    const float* bufs[2] = {nullptr, nullptr};
};

// Calls emit(j0, k0, first, last + 1, face, rows) for every work item of chunks of `chunk` planes. `L2` says which kernel
// takes the list, and with it where its tiles may start (Tile): an ensemble's kernel has the L2 term when any of its
// droplets has, so that a droplet's own plan.L2 does not decide. In each row band and plane chunk the k tiles start at the first changing cell (rounded down to the tiles'
// alignment) instead of at multiples of TK, and each tile's plane range is cut to the planes
// whose changing cells reach it: every changing cell lies in exactly one item, and fewer idle lanes
// are visited than with a fixed tile grid. `face`: the item has changing cells next to a grid face.
template <class Emit>
inline void tiled_each_item(const TiledPlan& plan, int chunk, bool L2, Emit emit) {
    using namespace tiled;
    const int lo_d = L2 ? 2 : 1;
    for (const TiledBand& b : plan.bands) {
        for (int ib = b.ib; ib < b.ie; ib += chunk) {
            const int ie = std::min(b.ie, ib + chunk);
            int kmin = INT32_MAX, kmax = -1;
            for (int p = ib; p < ie; ++p)
                if (b.kmin[p - b.ib] <= b.kmax[p - b.ib]) {
                    kmin = std::min(kmin, b.kmin[p - b.ib]);
                    kmax = std::max(kmax, b.kmax[p - b.ib]);
                }
            if (kmax < 0) continue;
            for (int k0 = L2 ? ((kmin - 2) & ~3) + 2 : kmin & ~7; k0 <= kmax; k0 += TK) {
                int first = -1, last = -1;
                bool face = false;
                for (int p = ib; p < ie; ++p) {
                    const int lo = b.kmin[p - b.ib], hi = b.kmax[p - b.ib];
                    if (lo <= hi && lo <= k0 + TK - 1 && hi >= k0) {
                        if (first < 0) first = p;
                        last = p;
                        face = face || p < lo_d || p > plan.Nx - 1 - lo_d || (lo < lo_d && k0 <= lo) ||
                               (hi > plan.Nz - 1 - lo_d && k0 + TK > hi);
                    }
                }
                if (first < 0) continue;
                emit(b.j0, k0, first, last + 1, face || b.face, b.rows);
            }
        }
    }
}

// Planes per work item. `cap` is the longest (the default, or a length the autotuner tries); a list too short to fill
// the GPU at that length is cut further, by this estimate of a step's time in microseconds: with n items on `slots` CTA slots,
//     waves(n) * (kItem + c * kPlane),
// kItem the first planes' way to shared memory, kPlane a plane of a CTA while its SM is shared (L1
// only: 0.95 us alone to 1.75 us with five CTAs; with L2 / L3 2.6 us), waves fractional from the
// fifth on (longest items first evens them out). An item on a face takes twice as long per plane.
// Measured against it, us a step with items of 1 / 2 / 3 / 4 / 6 / 8 / 16 planes and of the length chosen:
//     64^3, R = 28, L1              5.2   5.1   5.4   6.3   7.8   9.4  16.8   5.2
//     128^3, R = 58, L1            18.8  15.6  14.9  15.7  16.8  15.9  20.0  15.7
//     96^3, R = 42, L2 and L3      15.7  15.2  16.2  14.4  19.0  15.6  23.2  15.7
//     256^3, R = 120, L2 and L3   219   170   159   152   147   145   144   147
//     256^3, R = 115, L1          131    95    85    80    77    75    78    76
static int tiled_length(const std::vector<const TiledPlan*>& plans, int cap, Load load, bool L2) {
    static const int sms = [] {
        int dev = 0, n = 0;
        if (cudaGetDevice(&dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
            return 148;
        return n;
    }();
    const int per_sm = load == kLoadL1 ? 5 : 4;
    const double kItem = load == kLoadDeep ? 1.3 : 1.0, face_plane = load == kLoadDeep ? 5.3 : 2.0;
    int best = cap;
    double best_t = std::numeric_limits<double>::infinity();
    for (int c : {cap, 6, 4, 3, 2, 1}) {
        if (c > cap) continue;
        long long n = 0;
        bool faces = false;
        for (const TiledPlan* p : plans)
            tiled_each_item(*p, c, L2, [&](int, int, int, int, bool f, int) {
                ++n;
                faces = faces || f;
            });
        const double full = (double)n / ((double)sms * per_sm);
        const int m = (int)std::min<long long>(per_sm, (n + sms - 1) / sms);
        const double waves = full > 4.0 ? full + 0.5 : std::ceil(full);
        double t = waves * (kItem + c * (load == kLoadDeep ? 2.6 : load == kLoadL1 ? 0.75 + 0.2 * m : 0.6 + 0.35 * m));
        if (faces) t = std::max(t, kItem + c * face_plane + 0.5 * t);
        if (t < best_t) {
            best_t = t;
            best = c;
        }
        if (full > 24.0) break;  // shorter items only add halo planes
    }
    return best;
}

// The work list. Items are ordered longest first (an item on a face counting double): CTAs are
// dispatched in item order, so the short items of the droplet's poles fill the last wave instead of
// trailing it; among items of one length the plane chunk is slowest (CTAs resident together share
// halo planes in L2). *active: the cells of the grid inside the items' tiles (read once per step).
inline std::vector<int4> tiled_items(const TiledPlan& plan, int chunk, bool L2, long long* active) {
    struct Item {
        int4 t;
        int cost;
    };
    std::vector<Item> items;
    long long act = 0;
    tiled_each_item(plan, chunk, L2, [&](int j0, int k0, int first, int end, bool face, int rows) {
        items.push_back(Item{make_int4(j0, k0, first, end), (end - first) * (face ? 2 : 1)});
        act += (long long)rows * (std::min(plan.Nz, k0 + tiled::TK) - std::max(0, k0)) * (end - first);
    });
    std::stable_sort(items.begin(), items.end(), [](const Item& a, const Item& b) {
        if (a.cost != b.cost) return a.cost > b.cost;
        if (a.t.z != b.t.z) return a.t.z < b.t.z;
        if (a.t.x != b.t.x) return a.t.x < b.t.x;
        return a.t.y < b.t.y;
    });
    std::vector<int4> out;
    for (const Item& i : items) out.push_back(i.t);
    if (active) *active = act;
    return out;
}

// Length of the work items asked for: at most `planes` (tiled_length), or exactly.
struct ItemLength {
    int planes;
    bool exact;
};
// LDG_QSR_CHUNK sets the length exactly.
inline ItemLength tiled_default_length() {
    if (const char* e = getenv("LDG_QSR_CHUNK")) return ItemLength{std::min(4096, std::max(1, atoi(e))), true};
    return ItemLength{tiled::CHUNK, false};
}

// Tensor map of a field: boxes of a tile with its halo, or of the tile alone.
static int tiled_encode(CUtensorMap* tm, const float* base, int Nx, int Ny, int Nz, int sj, long long si, long long sc,
                        bool L2, bool halo = true) {
    static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
    if (!encode) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess || !fn) {
            set_error("cuTensorMapEncodeTiled entry point unavailable");
            return LDG_ERR_CUDA;
        }
        encode = (PFN_cuTensorMapEncodeTiled_v12000)fn;
    }
    cuuint64_t dims[4] = {(cuuint64_t)Nz, (cuuint64_t)Ny, (cuuint64_t)Nx, 5};
    cuuint64_t strides[3] = {(cuuint64_t)sj * 4, (cuuint64_t)si * 4, (cuuint64_t)sc * 4};
    using namespace tiled;
    const int w = L2 ? Tile<true>::RW : Tile<false>::RW, r = L2 ? Tile<true>::ROWS : Tile<false>::ROWS;
    cuuint32_t box[4] = {(cuuint32_t)(halo ? w : TK), (cuuint32_t)(halo ? r : TJ), 1, 5};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult res = encode(tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, (void*)base, dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (res != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled failed: " + std::to_string((int)res));
        return LDG_ERR_CUDA;
    }
    return LDG_OK;
}

// Work items and their planes' row masks on the device. `inst` and `rec` are set for droplet `inst`
// whose masks start at record rec0; returns the number of records through *n_rec.
inline void tiled_device_items(const std::vector<int4>& list, int inst, int rec0, std::vector<tiled::TileItem>& out,
                               int* n_rec) {
    int rec = rec0;
    for (const int4& t : list) {
        out.push_back(tiled::TileItem{t.x, t.y, t.z, t.w, inst, rec, 0, 0});
        rec += t.w - t.z;
    }
    *n_rec = rec - rec0;
}
inline int tiled_masks(const TiledPlan& plan, const tiled::TileItem* d_items, int n_items, bool L2,
                       tiled::RowMask* d_masks, cudaStream_t st) {
    if (n_items == 0) return LDG_OK;
    tiled::k_tile_masks<<<n_items, tiled::TK * tiled::TJ, 0, st>>>(d_items, plan.flags, plan.Nx, plan.Ny, plan.Nz, plan.sj,
                                                            plan.si, L2 ? 2 : 1, d_masks);
    LDG_LAUNCHED("k_tile_masks");
    return LDG_OK;
}

// A work list on the device. It is made in full before it takes the place of another, so that a plan keeps a
// list that can be launched where making a new one fails.
struct DeviceList {
    tiled::TileItem* items = nullptr;
    tiled::RowMask* masks = nullptr;
};
inline void tiled_list_free(DeviceList& d) {
    cudaFree(d.items);
    cudaFree(d.masks);
    d = DeviceList{};
}
// Uploads `items` (n_rec planes in all) and forms their masks by `form`, both on `st` and complete on return.
template <class Form>
inline int tiled_list_make(const std::vector<tiled::TileItem>& items, int n_rec, cudaStream_t st, DeviceList& d,
                           Form form) {
    d = DeviceList{};
    if (items.empty()) return LDG_OK;
    auto make = [&]() -> int {
        LDG_CUDA(cudaMalloc(&d.items, items.size() * sizeof(items[0])));
        LDG_CUDA(cudaMalloc(&d.masks, (size_t)n_rec * tiled::MASK_BYTES));
        LDG_CUDA(cudaMemcpyAsync(d.items, items.data(), items.size() * sizeof(items[0]), cudaMemcpyHostToDevice, st));
        const int rc = form(d);
        LDG_CUDA(cudaStreamSynchronize(st));
        return rc;
    };
    const int rc = make();
    if (rc) tiled_list_free(d);
    return rc;
}

// Uploads the work list for items of that length. On failure the plan is as before.
inline int tiled_plan_rechunk(TiledPlan& plan, ItemLength len, cudaStream_t st) {
    const int chunk = len.exact ? len.planes : tiled_length({&plan}, len.planes, plan.load, plan.L2);
    long long active = 0;
    std::vector<tiled::TileItem> items;
    int n_rec = 0;
    tiled_device_items(tiled_items(plan, chunk, plan.L2, &active), 0, 0, items, &n_rec);
    DeviceList now;
    const int rc = tiled_list_make(items, n_rec, st, now, [&](const DeviceList& d) {
        return tiled_masks(plan, d.items, (int)items.size(), plan.L2, d.masks, st);
    });
    if (rc) return rc;
    DeviceList old{plan.items, plan.masks};
    tiled_list_free(old);
    plan.items = now.items;
    plan.masks = now.masks;
    plan.n_items = (int)items.size();
    plan.active_cells = active;
    plan.chunk = chunk;
    return LDG_OK;
}

// Builds the work list from the host classification and encodes the two tensor maps. The device's part runs on `st`, which
// the caller's later work uses or waits for (a default-stream operation has no order against a non-blocking stream).
inline int tiled_plan_build(TiledPlan& plan, int Nx, int Ny, int Nz, int sj, long long si, const uint8_t* fl,
                            const uint8_t* d_flags, const float* buf0, const float* buf1, long long sc, bool L2, bool L3, cudaStream_t st) {
    using namespace tiled;
    plan = TiledPlan{};
    plan.load = (L2 || L3) ? kLoadDeep : kLoadL1;
    plan.Nx = Nx; plan.Ny = Ny; plan.Nz = Nz;
    plan.sj = sj; plan.si = si;
    plan.flags = d_flags;
    plan.L2 = L2;
    const int ntj = (Ny + TJ - 1) / TJ;
    long long written = 0;
    std::vector<TiledBand> bands(ntj);
    for (TiledBand& b : bands) {  // no allocation inside the parallel loop
        b.kmin.assign(Nx, INT32_MAX);
        b.kmax.assign(Nx, -1);
    }
    // the bands are independent; with one thread the creation of a 256^3 solver took 77 ms, 34-61 with sixteen
#pragma omp parallel for reduction(+ : written) schedule(dynamic) if (sc > (1 << 18))
    for (int jt = 0; jt < ntj; ++jt) {
        TiledBand& b = bands[jt];
        b.j0 = jt * TJ;
        b.rows = std::min(Ny, (jt + 1) * TJ) - b.j0;
        int imin = Nx, imax = -1;
        for (int i = 0; i < Nx; ++i)
            for (int j = b.j0; j < b.j0 + b.rows; ++j)
                for (int k = 0; k < Nz; ++k)
                    if (fl[(size_t)i * si + (size_t)j * sj + k] & (kMove | kFixed)) {
                        b.kmin[i] = std::min(b.kmin[i], k);
                        b.kmax[i] = std::max(b.kmax[i], k);
                        imin = std::min(imin, i);
                        imax = std::max(imax, i);
                        ++written;
                    }
        b.face = b.j0 < (L2 ? 2 : 1) || b.j0 + b.rows > Ny - (L2 ? 2 : 1);
        b.ib = imin;
        b.ie = imax + 1;
    }
    for (TiledBand& b : bands) {
        if (b.ie <= b.ib) continue;
        b.kmin.erase(b.kmin.begin() + b.ie, b.kmin.end());
        b.kmin.erase(b.kmin.begin(), b.kmin.begin() + b.ib);
        b.kmax.erase(b.kmax.begin() + b.ie, b.kmax.end());
        b.kmax.erase(b.kmax.begin(), b.kmax.begin() + b.ib);
        plan.bands.push_back(std::move(b));
    }
    plan.written_cells = written;
    int rc = tiled_plan_rechunk(plan, tiled_default_length(), st);
    if (rc) return rc;
    LDG_CUDA(cudaMalloc(&plan.err, sizeof(int)));
    LDG_CUDA(cudaMemsetAsync(plan.err, 0, sizeof(int), st));
    rc = tiled_encode(&plan.tmap[0], buf0, Nx, Ny, Nz, sj, si, sc, L2);
    if (rc) return rc;
    rc = tiled_encode(&plan.tmap[1], buf1, Nx, Ny, Nz, sj, si, sc, L2);
    if (rc) return rc;
    plan.bufs[0] = buf0;
    plan.bufs[1] = buf1;
    plan.ok = true;
    return LDG_OK;
}

// Raises a kernel's shared-memory limit on the current device. The limit belongs to the device: `done` holds one bit for
// each device (of the first 64) that has it, so that it is set once on each.
template <class Kernel>
inline int tiled_smem_limit(Kernel k, size_t smem, std::atomic<unsigned long long>& done) {
    int dev = 0;
    LDG_CUDA(cudaGetDevice(&dev));
    const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
    if (done.load(std::memory_order_relaxed) & bit) return LDG_OK;
    LDG_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    done.fetch_or(bit, std::memory_order_relaxed);
    return LDG_OK;
}

template <bool L2, bool L3, bool N, int R, bool K>
static int tiled_launch_t(const TiledPlan& plan, int which, float* out, const QsrConst& P, cudaStream_t st,
                          const float* lo_in, float* lo_out) {
    using namespace tiled;
    const auto k = k_step_tiled<L2, L3, N, R, K>;
    constexpr size_t smem = tile_smem_bytes<L2>();
    static std::atomic<unsigned long long> devices{0};
    if (int rc = tiled_smem_limit(k, smem, devices)) return rc;
    if (plan.n_items == 0) return LDG_OK;
    LDG_CUDA(launch_pdl(k, dim3((unsigned)plan.n_items), THREADS, smem, st, plan.tmap[which], plan.bufs[which], out,
                        (const RowMask*)plan.masks, (const TileItem*)plan.items, P, plan.err, lo_in, lo_out));
    return LDG_OK;
}

template <int R, bool K>
inline int tiled_dispatch(const TiledPlan& plan, int which, float* out, const QsrConst& P,
                          bool L2, bool L3, bool noise, cudaStream_t st, const float* lo_in, float* lo_out) {
    const int key = (L2 ? 1 : 0) | (L3 ? 2 : 0) | (noise ? 4 : 0);
    switch (key) {
        case 0: return tiled_launch_t<false, false, false, R, K>(plan, which, out, P, st, lo_in, lo_out);
        case 1: return tiled_launch_t<true, false, false, R, K>(plan, which, out, P, st, lo_in, lo_out);
        case 2: return tiled_launch_t<false, true, false, R, K>(plan, which, out, P, st, lo_in, lo_out);
        case 3: return tiled_launch_t<true, true, false, R, K>(plan, which, out, P, st, lo_in, lo_out);
        case 4: return tiled_launch_t<false, false, true, R, K>(plan, which, out, P, st, lo_in, lo_out);
        case 5: return tiled_launch_t<true, false, true, R, K>(plan, which, out, P, st, lo_in, lo_out);
        case 6: return tiled_launch_t<false, true, true, R, K>(plan, which, out, P, st, lo_in, lo_out);
        default: return tiled_launch_t<true, true, true, R, K>(plan, which, out, P, st, lo_in, lo_out);
    }
}

// One step through the tiled kernel. `in` must be one of the two planned buffers. With lo_out
// set (explicit steps only) the step uses compensated storage: lo_in / lo_out are the low
// words of the input and output buffers.
inline int tiled_step(const TiledPlan& plan, const float* in, float* out, const QsrConst& P,
                      bool L2, bool L3, bool noise, bool rhs, cudaStream_t st, const float* lo_in = nullptr,
                      float* lo_out = nullptr) {
    const int which = (in == plan.bufs[0]) ? 0 : 1;
    if (rhs) return tiled_dispatch<tiled::kRhs, false>(plan, which, out, P, L2, L3, noise, st, nullptr, nullptr);
    if (lo_out) return tiled_dispatch<tiled::kStep, true>(plan, which, out, P, L2, L3, noise, st, lo_in, lo_out);
    return tiled_dispatch<tiled::kStep, false>(plan, which, out, P, L2, L3, noise, st, nullptr, nullptr);
}

inline void tiled_plan_free(TiledPlan& plan) {
    if (plan.items) cudaFree(plan.items);
    if (plan.masks) cudaFree(plan.masks);
    cudaFree(plan.err);
    plan = TiledPlan{};
}
// A sweep plan shares the step plan's error word.
inline void tiled_sweep_free(TiledPlan& plan) {
    plan.err = nullptr;
    tiled_plan_free(plan);
}

// The sweeps' plan of the same grid: the step's changing cells, cut to the sweeps' own item length and
// encoded for one-cell stencils. On failure the plan is empty again.
inline int tiled_sweep_plan(const TiledPlan& step, const long long sc, TiledPlan& plan, cudaStream_t st) {
    plan = TiledPlan{};
    plan.Nx = step.Nx; plan.Ny = step.Ny; plan.Nz = step.Nz;
    plan.sj = step.sj; plan.si = step.si;
    plan.flags = step.flags;
    plan.bands = step.bands;
    plan.err = step.err;
    plan.load = kLoadSweep;
    int rc = tiled_plan_rechunk(plan, tiled_default_length(), st);
    for (int b = 0; b < 2 && rc == LDG_OK; ++b) {
        plan.bufs[b] = step.bufs[b];
        rc = tiled_encode(&plan.tmap[b], step.bufs[b], step.Nx, step.Ny, step.Nz, step.sj, step.si, sc, false);
    }
    plan.ok = rc == LDG_OK;
    if (rc) tiled_sweep_free(plan);
    return rc;
}

// One Jacobi sweep: field `in` (one of the planned buffers) to `out`. tm_rhs: the right-hand side's map.
template <int kMode>
static int tiled_sweep_t(const TiledPlan& plan, const float* in, float* out, const CUtensorMap& tm_rhs, const QsrConst& P,
                         cudaStream_t st) {
    using namespace tiled;
    constexpr size_t smem = tile_smem_bytes<false, kMode>();
    static std::atomic<unsigned long long> devices{0};
    if (int rc = tiled_smem_limit(k_sweep_tiled<kMode>, smem, devices)) return rc;
    if (plan.n_items == 0) return LDG_OK;
    LDG_CUDA(launch_pdl(k_sweep_tiled<kMode>, dim3((unsigned)plan.n_items), THREADS, smem, st,
                        plan.tmap[in == plan.bufs[0] ? 0 : 1], tm_rhs, out, (const RowMask*)plan.masks,
                        (const TileItem*)plan.items, P, plan.err));
    return LDG_OK;
}
inline int tiled_sweep(const TiledPlan& plan, const float* in, float* out, const CUtensorMap& tm_rhs, const QsrConst& P,
                       bool last, cudaStream_t st) {
    LDG_REQUIRE(plan.ok, LDG_ERR_STATE, "Jacobi sweep: no plan");
    return last ? tiled_sweep_t<tiled::kSweepLast>(plan, in, out, tm_rhs, P, st)
                : tiled_sweep_t<tiled::kSweep>(plan, in, out, tm_rhs, P, st);
}

// Reads and clears the device error word (LDG_OK when no bounded wait gave up).
inline int tiled_check(const TiledPlan& plan, cudaStream_t st) {
    if (!plan.err) return LDG_OK;
    int e = 0;
    LDG_CUDA(cudaMemcpyAsync(&e, plan.err, sizeof(int), cudaMemcpyDeviceToHost, st));
    LDG_CUDA(cudaStreamSynchronize(st));
    if (e != 0) {
        LDG_CUDA(cudaMemsetAsync(plan.err, 0, sizeof(int), st));
        set_error("tiled step: a bounded shared-memory pipeline wait gave up");
        return LDG_ERR_TIMEOUT;
    }
    return LDG_OK;
}

}  // namespace ldg
