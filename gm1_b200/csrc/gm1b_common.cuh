// gm1b_common.cuh - shared device/host helpers of libgm1b.so.
//
// Arithmetic contract (all translation units): binary32 storage, binary32
// arithmetic one operation at a time, no fused multiply-add (the library is
// compiled with --fmad=false), IEEE division (-prec-div=true), no flush to
// zero.  This is the contract of the reference kernels
// (src/cm1core/cuda_sound3_periodic.py:1097-1112, --fmad=false --ftz=false
// --prec-div=true) and lets the kernels reproduce the reference's CPU twins
// word for word.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/gm1b.h"

namespace gm1b {

// binary32 constants, each the correctly rounded float32 quotient the
// reference forms at run time (src/cm1core/cuda_psolver3_trajectory.py:282-302)
constexpr float kF5_1 = 0x1.111112p-5f;   //   2/60
constexpr float kF5_2 = -0x1.bbbbbcp-3f;  // -13/60
constexpr float kF5_3 = 0x1.911112p-1f;   //  47/60
constexpr float kF5_4 = 0x1.ccccccp-2f;   //  27/60
constexpr float kF5_5 = -0x1.99999ap-5f;  //  -3/60
constexpr float kF3_1 = -0x1.555556p-3f;  //  -1/6
constexpr float kF3_2 = 0x1.aaaaaap-1f;   //   5/6
constexpr float kF3_3 = 0x1.555556p-2f;   //   2/6
constexpr float kRddcv = 0x1.98fef2p-2f;  // 287.04 / (1005.7 - 287.04)
constexpr float kGrav = 0x1.39eb86p+3f;   // 9.81
constexpr float kTh0r = 300.0f;
constexpr float kSmeps = 0x1.4484cp-100f;  // 1e-30
constexpr float kCp = 0x1.f6d99ap+9f;      // 1005.7
constexpr float kAlph = 0x1.333334p-1f;    // 0.60
constexpr float kKdiv = 0x1.99999ap-4f;    // 0.10

__device__ __forceinline__ float flx3(float s1, float s2, float s3) {
    float r = kF3_1 * s1;
    r = r + kF3_2 * s2;
    return r + kF3_3 * s3;
}

// Correctly rounded binary32 reciprocal on the short path: the hardware's
// approximate reciprocal (PTX rcp.approx.ftz.f32, at most 1 ulp from 1/b)
// refined by one FMA Newton-Raphson step in Markstein's form (P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000
// processor", IBM J. Res. Dev. 34(1), 1990): e = 1 - b*y exactly, then
// y + y*e rounded once.  Used where |b| lies in [2^-125, 2^125]; elsewhere
// (subnormal-adjacent, huge, zero, inf, NaN) it defers to __frcp_rn.
// gm1b_selftest_reciprocal compares it with __frcp_rn on every one of the
// 2^32 binary32 words.
__device__ __forceinline__ bool rcp_short(float b) {  // the short path holds
    const float ab = fabsf(b);
    return ab >= 0x1p-125f && ab <= 0x1p125f;
}
__device__ __forceinline__ float rcp_rn_short(float b) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));
    const float e = fmaf(-b, y, 1.0f);
    return fmaf(y, e, y);
}
__device__ __forceinline__ float rcp_rn(float b) { return rcp_short(b) ? rcp_rn_short(b) : __frcp_rn(b); }

__device__ __forceinline__ float flx5(float s1, float s2, float s3, float s4, float s5) {
    float r = kF5_1 * s1;
    r = r + kF5_2 * s2;
    r = r + kF5_3 * s3;
    r = r + kF5_4 * s4;
    return r + kF5_5 * s5;
}

// Padded-lane extents with the index helpers of the four staggered shapes.
struct Dims {
    int ni, nj, nk;
    __host__ __device__ __forceinline__ size_t s(int k, int j, int i) const {
        return ((size_t)k * (nj + 2) + (size_t)j) * (size_t)(ni + 2) + (size_t)i;
    }
    __host__ __device__ __forceinline__ size_t u(int k, int j, int f) const {
        return ((size_t)k * (nj + 2) + (size_t)j) * (size_t)(ni + 1) + (size_t)f;
    }
    __host__ __device__ __forceinline__ size_t v(int k, int g, int i) const {
        return ((size_t)k * (nj + 1) + (size_t)g) * (size_t)(ni + 2) + (size_t)i;
    }
    __host__ __device__ __forceinline__ size_t w(int k, int j, int i) const {
        return ((size_t)k * nj + (size_t)j) * (size_t)ni + (size_t)i;
    }
    __host__ __device__ __forceinline__ size_t scalar_words() const { return (size_t)(nk + 2) * (nj + 2) * (ni + 2); }
    __host__ __device__ __forceinline__ size_t u_words() const { return (size_t)(nk + 2) * (nj + 2) * (ni + 1); }
    __host__ __device__ __forceinline__ size_t v_words() const { return (size_t)(nk + 2) * (nj + 1) * (ni + 2); }
    __host__ __device__ __forceinline__ size_t w_words() const { return (size_t)(nk + 2) * nj * ni; }
};

__device__ __forceinline__ int wrap(int x, int n) {  // periodic halo index -> live index
    return x == 0 ? n : (x == n + 1 ? 1 : x);
}

// Python modulo for x in [-n, 2n), the only range the stencils produce
// (n >= 5 and offsets of at most +-4 around an index in [-1, n+1]).
__device__ __forceinline__ int pmod(int x, int n) { return x < 0 ? x + n : (x >= n ? x - n : x); }

// Brackets one kernel launch with profiler events when the profiler is on.
class ProfScope {
  public:
    ProfScope(const char *name, cudaStream_t st);
    void stop();

  private:
    const char *name_;
    cudaStream_t st_;
    cudaEvent_t start_;
};

// the composed step's own launches: several open fills (GM1B_FILL_*) at once,
// and theta with the three moisture rows packed into their filled carriers
struct OpenFill {
    int kind;
    float *q;
};
int32_t open_fills(int32_t ni, int32_t nj, int32_t nk, const OpenFill *fills, int n, cudaStream_t st);
int32_t pack_scalars_open(int32_t ni, int32_t nj, int32_t nk, const float *th0, const float *const scalar[4],
                          float *const padded[4], cudaStream_t st);

// The sweep of a column's tridiagonal rows 0 .. n-1 in shared memory (rows at
// stride 32, one lane per column, a whole warp; n >= 1): the eliminated
// coefficients are left in s_c, the solution in s_d.  Bound by the chain of a
// row's multiply, add, reciprocal and multiply, so the reciprocals' range
// check, a branch on the chain, is taken once a chunk of rows: the chunk is
// formed on the short path, and again from its start with rcp_rn if any row's
// pivot of any lane lay outside it.  Against a row at a time with the branch:
// turbu at 189x131x64 71 -> 56 us, turbv 54 -> 45, the acoustic column pass at
// 640x768x80 0.863 -> 0.799 ms.
constexpr int kSweepChunk = 8;  // rows whose words the back substitution reads together

template <int kSweepRows>  // rows of a forward chunk; the next one's words are in flight meanwhile
__device__ __forceinline__ void column_sweep(const float *s_a, const float *s_b, float *s_c, float *s_d, int n) {
    float ec = 0.0f, ed = 0.0f;
    struct Rows {
        float a[kSweepRows], b[kSweepRows], c[kSweepRows], d[kSweepRows];
    };
    auto load = [&](int p0) {
        Rows r;
#pragma unroll
        for (int q = 0; q < kSweepRows; ++q) {
            const int z = min(p0 + q, n - 1) * 32;
            r.a[q] = p0 + q == 0 ? 0.0f : s_a[z], r.b[q] = s_b[z], r.c[q] = s_c[z], r.d[q] = s_d[z];
        }
        return r;
    };
    Rows next = load(0);
    for (int p0 = 0; p0 < n; p0 += kSweepRows) {
        const Rows r = next;
        next = load(p0 + kSweepRows);  // (rows past the last repeat it)
        float e[kSweepRows], f[kSweepRows];
        const float ec0 = ec, ed0 = ed;
        bool rare = false;
#pragma unroll
        for (int q = 0; q < kSweepRows; ++q) {
            const float piv = r.a[q] * ec + r.b[q];
            rare |= !rcp_short(piv);
            const float inv = rcp_rn_short(piv);
            e[q] = ec = -(r.c[q] * inv);
            f[q] = ed = (r.d[q] - r.a[q] * ed) * inv;
        }
        if (__any_sync(0xffffffffu, rare)) {
            ec = ec0, ed = ed0;
#pragma unroll
            for (int q = 0; q < kSweepRows; ++q) {
                const float inv = rcp_rn(r.a[q] * ec + r.b[q]);
                e[q] = ec = -(r.c[q] * inv);
                f[q] = ed = (r.d[q] - r.a[q] * ed) * inv;
            }
        }
#pragma unroll
        for (int q = 0; q < kSweepRows; ++q) {
            if (p0 + q >= n) break;
            s_c[(p0 + q) * 32] = e[q], s_d[(p0 + q) * 32] = f[q];
        }
    }
    float sol = s_d[(n - 1) * 32];
    for (int pb = n - 2; pb >= 0; pb -= kSweepChunk) {
        float ce[kSweepChunk], de[kSweepChunk];
#pragma unroll
        for (int q = 0; q < kSweepChunk; ++q) {
            const int p = max(pb - q, 0);
            ce[q] = s_c[p * 32], de[q] = s_d[p * 32];
        }
#pragma unroll
        for (int q = 0; q < kSweepChunk; ++q) {
            if (pb - q < 0) break;
            sol = ce[q] * sol + de[q];
            s_d[(pb - q) * 32] = sol;
        }
    }
}

// Levels a thread of a memory-bound column march takes: eight, or fewer (two at
// the least) until four CTAs of its 256 threads lie on each of 148 SMs (mass
// fluxes of 128x100x64: eight levels 15.1 us, two 12.8; of 256x256x80: 76 and 93).
// `light`: a march that carries little up takes single levels where two leave
// fewer than 2.5 CTAs an SM (buoyancy of 37x24x24: two levels 4.2 us, one 3.1;
// 53x48x40: 4.8 and 4.3; 26x115x55, with 2.8 CTAs an SM: 5.4 and 5.6).
// The chunks of a column lie in a grid dimension of at most 65535.
inline int level_chunk(size_t tiles, int nk, bool light = false) {
    int chunk = 8;
    while (chunk > 2 && tiles * (size_t)((nk + chunk - 1) / chunk) < 4 * 148) chunk /= 2;
    if (light && 2 * tiles * (size_t)((nk + chunk - 1) / chunk) < 5 * 148) chunk = 1;
    const int least = (int)(((size_t)nk + 65534) / 65535);
    return chunk < least ? least : chunk;
}

}  // namespace gm1b

// thread-local error message of the last failed entry point
void gm1b_set_error(const char *fmt, ...);
