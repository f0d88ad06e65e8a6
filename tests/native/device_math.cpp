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

extern "C" {

// S and director of n tensors (five stored components each).
void dm_nematic(const double* q, long long n, double iso_cut, double* out) {
    for (long long t = 0; t < n; ++t) {
        const Nematic f = nematic64(q + 5 * t, iso_cut, Nematic{0.0, 0.0, 0.0, 1.0});
        out[4 * t] = f.S, out[4 * t + 1] = f.nx, out[4 * t + 2] = f.ny, out[4 * t + 3] = f.nz;
    }
}

}  // extern "C"
