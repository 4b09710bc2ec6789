// advection5.cu - sm_100a kernels of the padded (ng = 3) lane: terrain mass
// flux with its divergence, and fifth-order / WENO5 scalar advection.
//
// Behaviour followed (reference file:line):
//   cpu_terrain_mass_flux5_inplace   src/cm1core/cuda_advection5.py:271-437
//   cpu_scalar_advection5_inplace    src/cm1core/cuda_advection5.py:440-579
//   lateral-side tendency of the reference kernel
//   cm1_adv5_scalar_tendency_v1      src/cm1core/cuda_advection5.py:669
//
// Design (B200): the scalar advection is ONE fused pass in which a warp owns
// a row of 32 x faces and marches up a chunk of levels: the lanes exchange
// their x face fluxes by shuffle (31 cells per 32 lanes), the upper vertical
// flux is carried to the next level as the lower one.  The face-flux scratch
// arrays of the reference (three passes through HBM) are optional outputs
// here.  WENO smoothness weights are binary64 as in the reference.
#include <algorithm>

#include "gm1b_common.cuh"
#include "weno.cuh"

namespace gm1b {
namespace {

constexpr int NG = 3;
constexpr int kAX = 32;  // tile x
constexpr int kAY = 4;   // tile y

// largest binary32 below 1e-20: |x| < 1e-20 (binary64 test of the reference
// twin) is |x| <= this for every binary32 x
constexpr float kDivClamp = 0x1.79ca1p-67f;

struct PaddedDims {
    int ni, nj, nk;
    // 32-bit element offsets: the entry points refuse grids whose padded
    // arrays reach 2^31 words
    __host__ __device__ __forceinline__ unsigned s(int k, int y, int x) const {
        return ((unsigned)k * (unsigned)(nj + 2 * NG) + (unsigned)y) * (unsigned)(ni + 2 * NG) + (unsigned)x;
    }
    __host__ __device__ __forceinline__ unsigned u(int k, int y, int x) const {
        return ((unsigned)k * (unsigned)(nj + 2 * NG) + (unsigned)y) * (unsigned)(ni + 1 + 2 * NG) + (unsigned)x;
    }
    __host__ __device__ __forceinline__ unsigned v(int k, int y, int x) const {
        return ((unsigned)k * (unsigned)(nj + 1 + 2 * NG) + (unsigned)y) * (unsigned)(ni + 2 * NG) + (unsigned)x;
    }
    __host__ __device__ __forceinline__ unsigned c(int k, int j, int i) const {  // (nk', nj, ni)
        return ((unsigned)k * (unsigned)nj + (unsigned)j) * (unsigned)ni + (unsigned)i;
    }
};

template <bool WENO>
__device__ __forceinline__ float recon(float s1, float s2, float s3, float s4, float s5, double eps) {
    if (WENO) return weno5(s1, s2, s3, s4, s5, eps);
    return flx5(s1, s2, s3, s4, s5);
}

// ---------------------------------------------------------------------------
// terrain mass flux, part 1: interior horizontal faces, zero rrw lid/floor
// grid (x over i in 0..ni-1, y over j in 0..nj-1, z over k = 1..nk)
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kAX *kAY)
    mass_flux_horizontal_kernel(gm1b_mass_flux5_arrays a, PaddedDims d) {
    const int i = blockIdx.x * kAX + threadIdx.x;
    const int j = blockIdx.y * kAY + threadIdx.y;
    const int k = blockIdx.z + 1;
    const int ni = d.ni, nj = d.nj, nk = d.nk;
    if (i >= ni || j >= nj) return;
    const int y = j + NG, x = i + NG;
    if (i >= 1) {
        const float density = a.rho0_3d[d.c(k - 1, j, i - 1)] + a.rho0_3d[d.c(k - 1, j, i)];
        a.rru[d.u(k, y, x)] = (0.5f * density) * (a.u3d[d.u(k, y, x)] * a.rgzu[(size_t)j * (ni + 1) + i]);
    }
    if (j >= 1) {
        const float density = a.rho0_3d[d.c(k - 1, j - 1, i)] + a.rho0_3d[d.c(k - 1, j, i)];
        a.rrv[d.v(k, y, x)] = (0.5f * density) * (a.v3d[d.v(k, y, x)] * a.rgzv[(size_t)j * ni + i]);
    }
    if (k == 1) {
        a.rrw[d.s(1, y, x)] = 0.0f;
        a.rrw[d.s(nk + 1, y, x)] = 0.0f;
    }
}

// ---------------------------------------------------------------------------
// terrain mass flux, part 2: one thread per interior column marches up k,
// forming rrw(k) (terrain term included) and the divergence of level k-1
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kAX *kAY)
    mass_flux_column_kernel(gm1b_mass_flux5_arrays a, PaddedDims d, float dz, float rdx, float rdy) {
    const int i = blockIdx.x * kAX + threadIdx.x + 1;
    const int j = blockIdx.y * kAY + threadIdx.y + 1;
    const int ni = d.ni, nj = d.nj, nk = d.nk;
    if (i >= ni - 1 || j >= nj - 1) return;
    const int y = j + NG, x = i + NG;
    const float zt = (float)nk * dz;
    const float rzt = 1.0f / zt;
    const float rdsf = 1.0f / dz;
    const float dzdx = a.dzdx[(size_t)j * ni + i], dzdy = a.dzdy[(size_t)j * ni + i], gz = a.gz[(size_t)j * ni + i];
    float w_lo = 0.0f;  // rrw(k) for the level below (k = 1: zero floor)
    float ru_lo = a.rru[d.u(1, y, x)] + a.rru[d.u(1, y, x + 1)];
    float rv_lo = a.rrv[d.v(1, y, x)] + a.rrv[d.v(1, y + 1, x)];
    for (int k = 1; k <= nk; ++k) {
        float w_hi = 0.0f;
        float ru_hi = 0.0f, rv_hi = 0.0f;
        if (k + 1 <= nk) {
            const int kk = k + 1;
            const float sigmaf = (float)(kk - 1) * dz;
            const float sigma = (float)((double)kk - 1.5) * dz;
            float r2 = (sigmaf - sigma) * (1.0f / dz);
            const float r1 = 0.5f * (1.0f - r2);
            r2 = 0.5f * r2;
            ru_hi = a.rru[d.u(kk, y, x)] + a.rru[d.u(kk, y, x + 1)];
            rv_hi = a.rrv[d.v(kk, y, x)] + a.rrv[d.v(kk, y + 1, x)];
            const float ux = r2 * ru_hi + r1 * ru_lo;
            const float vy = r2 * rv_hi + r1 * rv_lo;
            float terrain = ux * dzdx + vy * dzdy;
            terrain = terrain * (sigmaf - zt);
            terrain = terrain * gz;
            terrain = terrain * rzt;
            w_hi = a.rf0[d.c(kk - 1, j, i)] * a.w3d[d.s(kk, y, x)] + terrain;
            a.rrw[d.s(kk, y, x)] = w_hi;
        }
        float value = (a.rru[d.u(k, y, x + 1)] - a.rru[d.u(k, y, x)]) * rdx +
                      (a.rrv[d.v(k, y + 1, x)] - a.rrv[d.v(k, y, x)]) * rdy;
        value = value + (w_hi - w_lo) * rdsf;
        a.divx[d.c(k - 1, j, i)] = (fabsf(value) <= kDivClamp) ? 0.0f : value;
        w_lo = w_hi;
        ru_lo = ru_hi;
        rv_lo = rv_hi;
    }
}

// the upwind reconstruction at a face from the six points around it (both
// upwind stencils): one reconstruction of selected points, so that a warp
// whose lanes differ in the sign of m does not form both
template <bool WENO>
__device__ __forceinline__ float upwind(float m, float s0, float s1, float s2, float s3, float s4, float s5,
                                        double eps) {
    const bool pos = m >= 0.0f;
    return m * recon<WENO>(pos ? s0 : s5, pos ? s1 : s4, pos ? s2 : s3, pos ? s3 : s2, pos ? s4 : s1, eps);
}

template <bool WENO>
__device__ __forceinline__ float z_face(const float win[6], float m, float c1, float c2, int face, int nk,
                                        double eps, float wepsf) {
    // win[q] holds level face-3+q (q = 0..5), i.e. win[3] = level face
#define L(lev) win[(lev) - face + 3]
    float r;
    if (face == 2) {
        if (m >= 0.0f)
            r = c1 * L(1) + c2 * L(2);
        else if (WENO)
            r = upstrpd(L(3), L(2), L(1), wepsf);
        else
            r = flx3(L(3), L(2), L(1));
    } else if (face == nk) {
        const bool up = WENO ? (m > 0.0f) : (m >= 0.0f);
        if (up)
            r = WENO ? upstrpd(L(face - 2), L(face - 1), L(face), wepsf) : flx3(L(face - 2), L(face - 1), L(face));
        else
            r = c1 * L(face - 1) + c2 * L(face);
    } else if (face == 3) {
        if (m >= 0.0f)
            r = WENO ? upstrpd(L(1), L(2), L(3), wepsf) : flx3(L(1), L(2), L(3));
        else
            r = recon<WENO>(L(5), L(4), L(3), L(2), L(1), eps);
    } else if (face == nk - 1) {
        if (m >= 0.0f)
            r = recon<WENO>(L(face - 3), L(face - 2), L(face - 1), L(face), L(face + 1), eps);
        else if (WENO)
            r = upstrpd(L(face + 1), L(face), L(face - 1), wepsf);
        else
            r = flx3(L(face + 1), L(face), L(face - 1));
    } else {
        return upwind<WENO>(m, L(face - 3), L(face - 2), L(face - 1), L(face), L(face + 1), L(face + 2), eps);
    }
#undef L
    return m * r;
}

// vertical column of the tendency: mode 0 uniform (rdsf = 1/dz); mode 1
// terrain-following stretched, rdsf(k) per level; mode 2 flat stretched,
// ((d*rdz)*mh(k)) with the column's rr0(k) and no gz
// (cuda_gm1_child_stretched_scalar.py:89-153 and :262-352)
struct VertCol {
    int mode;
    const float *rdsf;  // (nk+3,) CM1-indexed
    const float *mh;    // (nk+2,) CM1-indexed
    float rdz;
};

constexpr int kFaceOut = 31;    // cells a warp of 32 x faces completes
constexpr int kFifthRows = 8;   // rows (warps) per CTA of the fifth-order pass, each independent
constexpr int kWenoRows = 8;    // rows per CTA of the WENO pass: 8 rows of y faces complete 7 rows of cells

// levels per chunk when the caller leaves it open: long chunks re-read and
// re-form less (each chunk starts with six window loads and its lower face
// flux), short ones give a small plane warps enough: halve until two rounds of
// 48 (WENO 32) row warps on each of 148 SMs, or at most four levels, are left
inline int default_chunk(int row_warps, int nk, bool weno) {
    const int want = 148 * (weno ? 32 : 48);  // warps in flight worth of work
    int chunk = nk;
    while (chunk > 4 && (long long)row_warps * ((nk + chunk - 1) / chunk) < 2LL * want) chunk = (chunk + 1) / 2;
    return chunk;
}

// One warp = the faces x = x0 .. x0+31 of one row and a chunk of levels.  A
// lane forms the x flux of its face and takes the next face's from the lane
// above, so 31 cells per warp need no second flux and no divergent edge.  The
// fifth-order pass forms both y fluxes of a cell (cheaper than handing one
// down through shared memory behind a barrier); the WENO pass, whose flux
// costs four binary64 divisions, hands each y flux to the row below through
// shared memory, one barrier a level, the eighth row forming a flux only.
// Words come through L1, which holds a row's neighbours: the passes are bound
// by instruction issue (fifth order) and the binary64 weights (WENO).
// Measured on one B200, per launch at 640x768x80: fifth order 1.105 -> 0.430
// ms, WENO 2.572 -> 1.290 against CTAs that stage each level's plane in shared
// memory (WENO with 24 warps an SM 1.336, with 16 rows 1.836; fifth order with
// 24 warps 0.402 but 72 us for 68 at 256x256x80, with 40 warps 0.602; up to 44
// bytes spill at 32).
// Warps away from open sides, at levels away from the column's ends and with
// no flux outputs take a finish without those branches.
template <bool WENO, bool FLAT>
__global__ void __launch_bounds__(32 * (WENO ? kWenoRows : kFifthRows), 4)
    scalar_advection5_march_kernel(const __grid_constant__ gm1b_scalar_advection5_arrays a,
                                   const __grid_constant__ PaddedDims d, int levels_per_chunk, float rdx, float rdy,
                                   float rdsf, double eps, float wepsf, unsigned obc,
                                   const __grid_constant__ VertCol vc) {
    constexpr int ROWS = WENO ? kWenoRows : kFifthRows;
    __shared__ float s_fy[WENO ? 2 : 1][WENO ? ROWS : 1][32], s_vm[WENO ? 2 : 1][WENO ? ROWS : 1][32];
    const int lane = threadIdx.x, ty = threadIdx.y;
    const int ni = d.ni, nj = d.nj, nk = d.nk;
    const int sx = ni + 2 * NG, sy = nj + 2 * NG, ux = ni + 1 + 2 * NG, vy = nj + 1 + 2 * NG;
    const int splane = sx * sy, uplane = ux * sy, vplane = sx * vy, cplane = ni * nj;
    const int xtiles = (ni + kFaceOut - 1) / kFaceOut;  // tiles in one grid dimension, which takes any plane
    const int i = blockIdx.x % xtiles * kFaceOut + lane;
    const int row = blockIdx.x / xtiles * (WENO ? ROWS - 1 : ROWS) + ty;
    if (!WENO && row >= nj) return;  // whole warps: the fifth-order pass has no barrier
    // rows and faces past the domain repeat its last ones and store nothing
    const int j = min(row, WENO ? nj : nj - 1), f = min(i, ni);
    const int x = f + NG, y = j + NG;
    const bool cell = i < ni && row < nj && lane < kFaceOut && (!WENO || ty < ROWS - 1);
    const int k_begin = 1 + blockIdx.y * levels_per_chunk;
    const int k_end = min(nk, k_begin + levels_per_chunk - 1);
    const float *s = a.scalar;
    const bool owned = cell && (obc != 0u || (i >= 3 && i + 3 < ni && j >= 3 && j + 3 < nj));
    const int col = y * sx + x;          // this point in a scalar / w plane
    const int uc = y * ux + x, cc = min(j, nj - 1) * ni + min(f, ni - 1);
    const bool wo = i == 0 && (obc & 15u) == 2u, eo = i + 1 == ni && ((obc >> 4) & 15u) == 2u;
    const bool so = j == 0 && ((obc >> 8) & 15u) == 2u, no = j + 1 == nj && ((obc >> 12) & 15u) == 2u;
    const bool edge = __any_sync(0xffffffffu, wo || eo) || so || no || a.flux_x != nullptr || a.flux_y != nullptr ||
                      a.flux_z != nullptr;
    const float gz = FLAT ? 0.0f : __ldg(a.gz + cc);
    float win[6];  // levels k-3 .. k+2 of this point; shifted to k-2 .. k+3 for face k+1
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        const int lev = k_begin - 3 + q;
        win[q] = (lev >= 0 && lev <= nk + 1) ? __ldg(s + lev * splane + col) : 0.0f;
    }
    float fz_lo = 0.0f;
    if (cell) {
        if (k_begin >= 2) {
            const bool end = k_begin == 2 || k_begin == nk;
            const float m = __ldg(a.rrw + k_begin * splane + col);
            const float c1 = end ? __ldg(a.c1 + (k_begin - 1) * cplane + cc) : 0.0f;
            const float c2 = end ? __ldg(a.c2 + (k_begin - 1) * cplane + cc) : 0.0f;
            fz_lo = z_face<WENO>(win, m, c1, c2, k_begin, nk, eps, wepsf);
        } else if (a.flux_z != nullptr) {
            a.flux_z[splane + col] = 0.0f;
        }
    }
#pragma unroll 1
    for (int k = k_begin; k <= k_end; ++k) {
        const float *pt = s + k * splane + col;
        // the level's words, all in flight together
        const float mw = __ldg(a.rru + k * uplane + uc);
        const float ms = __ldg(a.rrv + k * vplane + col);
        float mn = 0.0f;
        if (!WENO) mn = __ldg(a.rrv + k * vplane + col + sx);
        float px[6], py[7];
#pragma unroll
        for (int q = 0; q < 6; ++q) px[q] = q == 3 ? 0.0f : __ldg(pt + (q - 3));
#pragma unroll
        for (int q = 0; q < 7; ++q) py[q] = (q == 3 || (WENO && q == 6)) ? 0.0f : __ldg(pt + (q - 3) * sx);
        const float zn = k + 3 <= nk + 1 ? __ldg(pt + 3 * splane) : 0.0f;
        const int fz = k + 1;
        const float mz = __ldg(a.rrw + fz * splane + col);  // level nk+1 exists and is not used
        const int c = (k - 1) * cplane + cc;
        const float div = __ldg(a.divx + c);
        const float rr0 = __ldg(a.rr0 + (FLAT ? (k - 1) * cplane : c));
        const float r = FLAT ? __ldg(vc.mh + k) : vc.mode == 1 ? __ldg(vc.rdsf + k) : rdsf;
        const float sv = win[3];
        px[3] = py[3] = sv;
        const float fx = upwind<WENO>(mw, px[0], px[1], px[2], px[3], px[4], px[5], eps);
        const float fy = upwind<WENO>(ms, py[0], py[1], py[2], py[3], py[4], py[5], eps);
        float fw = fx, fe = __shfl_down_sync(0xffffffffu, fx, 1);
        float fs = fy, fn;
        if (WENO) {
            const int buf = k & 1;
            s_fy[buf][ty][lane] = fy;
            s_vm[buf][ty][lane] = ms;
            __syncthreads();
            const int up = min(ty + 1, ROWS - 1);
            fn = s_fy[buf][up][lane];
            mn = s_vm[buf][up][lane];
        } else {
            fn = upwind<WENO>(mn, py[1], py[2], py[3], py[4], py[5], py[6], eps);
        }
#pragma unroll
        for (int q = 0; q < 5; ++q) win[q] = win[q + 1];
        win[5] = zn;
        float fz_hi = 0.0f;
        if (!edge && fz > 3 && fz < nk - 1) {
            fz_hi = upwind<WENO>(mz, win[0], win[1], win[2], win[3], win[4], win[5], eps);
            const float ax = (fw - fe) * rdx, ay = (fs - fn) * rdy;
            const float az = FLAT ? ((-(fz_hi - fz_lo)) * vc.rdz) * r : (fz_lo - fz_hi) * r;
            float total = (ax + ay) + az;
            total = total + sv * div;
            if (owned) a.tendency[c] = FLAT ? total * rr0 : (total * rr0) * gz;
        } else {
            const float ue = __shfl_down_sync(0xffffffffu, mw, 1);
            if (cell) {
                if (a.flux_x != nullptr) {
                    a.flux_x[k * uplane + uc] = fw;
                    if (i == ni - 1) a.flux_x[k * uplane + uc + 1] = fe;
                }
                if (a.flux_y != nullptr) {
                    a.flux_y[k * vplane + col] = fs;
                    if (j == nj - 1) a.flux_y[k * vplane + col + sx] = fn;
                }
                if (fz <= nk) {
                    const bool end = fz == 2 || fz == nk;
                    const float c1 = end ? __ldg(a.c1 + (fz - 1) * cplane + cc) : 0.0f;
                    const float c2 = end ? __ldg(a.c2 + (fz - 1) * cplane + cc) : 0.0f;
                    fz_hi = z_face<WENO>(win, mz, c1, c2, fz, nk, eps, wepsf);
                }
                if (a.flux_z != nullptr) a.flux_z[fz * splane + col] = fz_hi;
                if (owned) {
                    const bool iw = wo && mw >= 0.0f, ie = eo && ue <= 0.0f;
                    const bool js = so && ms >= 0.0f, jn = no && mn <= 0.0f;
                    if (iw) fw = fe;
                    if (ie) fe = fw;
                    if (js) fs = fn;
                    if (jn) fn = fs;
                    float ax = (fw - fe) * rdx;
                    float ay = (fs - fn) * rdy;
                    if (iw) ax = ax - (sv * (ue - mw)) * rdx;
                    if (ie) ax = ax - (sv * (ue - mw)) * rdx;
                    if (js) ay = ay - (sv * (mn - ms)) * rdy;
                    if (jn) ay = ay - (sv * (mn - ms)) * rdy;
                    float az;
                    if (FLAT) {
                        if (k == 1)
                            az = ((-fz_hi) * vc.rdz) * r;
                        else if (k == nk)
                            az = (fz_lo * vc.rdz) * r;
                        else
                            az = ((-(fz_hi - fz_lo)) * vc.rdz) * r;
                    } else {
                        if (k == 1)
                            az = (-fz_hi) * r;
                        else if (k == nk)
                            az = fz_lo * r;
                        else
                            az = (fz_lo - fz_hi) * r;
                    }
                    float total = (ax + ay) + az;
                    total = total + sv * div;
                    a.tendency[c] = FLAT ? total * rr0 : (total * rr0) * gz;
                }
            }
        }
        fz_lo = fz_hi;
    }
}

}  // namespace
}  // namespace gm1b

using namespace gm1b;

extern "C" int32_t gm1b_terrain_mass_flux5(int32_t ni, int32_t nj, int32_t nk, const gm1b_mass_flux5_arrays *arrays,
                                          float dx, float dy, float dz, void *stream) {
    if (arrays == nullptr || ni < 8 || nj < 8 || nk < 8) {
        gm1b_set_error("gm1b_terrain_mass_flux5: need arrays and ni, nj, nk >= 8");
        return GM1B_ERR_ARGUMENT;
    }
    if ((size_t)(nk + 3) * (size_t)(nj + 7) * (size_t)(ni + 7) >= ((size_t)1 << 31)) {
        gm1b_set_error("gm1b_terrain_mass_flux5: a %dx%dx%d grid's padded arrays reach 2^31 words; the kernels index with 32-bit "
                       "offsets", ni, nj, nk);
        return GM1B_ERR_ARGUMENT;
    }
    if (!(dx > 0.0f) || !(dy > 0.0f) || !(dz > 0.0f) || !isfinite(dx) || !isfinite(dy) || !isfinite(dz)) {
        gm1b_set_error("gm1b_terrain_mass_flux5: dx, dy, dz must be finite and > 0");
        return GM1B_ERR_ARGUMENT;
    }
    const float *const *p = reinterpret_cast<const float *const *>(arrays);
    for (size_t q = 0; q < sizeof(gm1b_mass_flux5_arrays) / sizeof(float *); ++q)
        if (p[q] == nullptr) {
            gm1b_set_error("gm1b_terrain_mass_flux5: array #%zu is NULL", q);
            return GM1B_ERR_ARGUMENT;
        }
    const PaddedDims d{ni, nj, nk};
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    {
        ProfScope ps("mass_flux_horizontal_kernel", st);
        mass_flux_horizontal_kernel<<<dim3((ni + kAX - 1) / kAX, (nj + kAY - 1) / kAY, nk), dim3(kAX, kAY), 0, st>>>(
            *arrays, d);
        ps.stop();
    }
    if (cudaPeekAtLastError() != cudaSuccess) {
        gm1b_set_error("mass_flux_horizontal_kernel: %s", cudaGetErrorString(cudaGetLastError()));
        return GM1B_ERR_CUDA;
    }
    const float rdx = 1.0f / dx, rdy = 1.0f / dy;
    {
        ProfScope ps("mass_flux_column_kernel", st);
        mass_flux_column_kernel<<<dim3((ni - 2 + kAX - 1) / kAX, (nj - 2 + kAY - 1) / kAY), dim3(kAX, kAY), 0, st>>>(
            *arrays, d, dz, rdx, rdy);
        ps.stop();
    }
    if (cudaPeekAtLastError() != cudaSuccess) {
        gm1b_set_error("mass_flux_column_kernel: %s", cudaGetErrorString(cudaGetLastError()));
        return GM1B_ERR_CUDA;
    }
    return GM1B_OK;
}

namespace {
int32_t scalar_advection5_launch(int32_t ni, int32_t nj, int32_t nk, const gm1b_scalar_advection5_arrays *arrays,
                                 int32_t nrk, int32_t wflag, float dx, float dy, float dz, double weps,
                                 uint32_t lateral_obc, int32_t levels_per_chunk, VertCol vc, void *stream) {
    if (arrays == nullptr || ni < 8 || nj < 8 || nk < 8) {
        gm1b_set_error("gm1b_scalar_advection5: need arrays and ni, nj, nk >= 8");
        return GM1B_ERR_ARGUMENT;
    }
    if ((size_t)(nk + 3) * (size_t)(nj + 7) * (size_t)(ni + 7) >= ((size_t)1 << 31)) {
        gm1b_set_error("gm1b_scalar_advection5: a %dx%dx%d grid's padded arrays reach 2^31 words; the kernels index with 32-bit "
                       "offsets", ni, nj, nk);
        return GM1B_ERR_ARGUMENT;
    }
    if (nrk < 1 || nrk > 3) {
        gm1b_set_error("gm1b_scalar_advection5: the low-storage RK3 schedule requires nrk = 1..3");
        return GM1B_ERR_ARGUMENT;
    }
    if (!(weps > 0.0) || !isfinite(weps) || !(dx > 0.0f) || !(dy > 0.0f) || !(dz > 0.0f)) {
        gm1b_set_error("gm1b_scalar_advection5: weps, dx, dy, dz must be finite and > 0");
        return GM1B_ERR_ARGUMENT;
    }
    const gm1b_scalar_advection5_arrays &a = *arrays;
    if (!a.scalar || !a.rru || !a.rrv || !a.rrw || !a.c1 || !a.c2 || !a.rr0 || !a.gz || !a.divx || !a.tendency) {
        gm1b_set_error("gm1b_scalar_advection5: a required array is NULL (only the flux outputs may be)");
        return GM1B_ERR_ARGUMENT;
    }
    for (int side = 0; side < 4; ++side) {
        const unsigned code = (lateral_obc >> (4 * side)) & 15u;
        if (lateral_obc != 0u && (code < 1u || code > 4u)) {
            gm1b_set_error("gm1b_scalar_advection5: lateral side codes must be 1..4 (or all 0 for a tile)");
            return GM1B_ERR_ARGUMENT;
        }
    }
    const bool weno = wflag != 0 && nrk == 3;
    const PaddedDims d{ni, nj, nk};
    const int xtiles = (ni + kFaceOut - 1) / kFaceOut;  // a warp's 32 faces complete 31 cells
    const int rows = weno ? kWenoRows - 1 : kFifthRows, ytiles = (nj + rows - 1) / rows;
    const int chunk = levels_per_chunk > 0 ? std::min(levels_per_chunk, nk) : default_chunk(xtiles * nj, nk, weno);
    const dim3 grid(xtiles * ytiles, (nk + chunk - 1) / chunk);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const float rdx = 1.0f / dx, rdy = 1.0f / dy, rdsf = 1.0f / dz;
    ProfScope ps(weno ? "scalar_advection5_weno_kernel" : "scalar_advection5_kernel", st);
    auto launch = [&](auto kernel, int rows_per_cta) {
        kernel<<<grid, dim3(32, rows_per_cta), 0, st>>>(a, d, chunk, rdx, rdy, rdsf, weps, (float)weps, lateral_obc, vc);
    };
    if (weno)
        vc.mode == 2 ? launch(scalar_advection5_march_kernel<true, true>, kWenoRows)
                     : launch(scalar_advection5_march_kernel<true, false>, kWenoRows);
    else
        vc.mode == 2 ? launch(scalar_advection5_march_kernel<false, true>, kFifthRows)
                     : launch(scalar_advection5_march_kernel<false, false>, kFifthRows);
    ps.stop();
    if (cudaPeekAtLastError() != cudaSuccess) {
        gm1b_set_error("scalar_advection5_kernel: %s", cudaGetErrorString(cudaGetLastError()));
        return GM1B_ERR_CUDA;
    }
    return GM1B_OK;
}
}  // namespace

extern "C" int32_t gm1b_scalar_advection5(int32_t ni, int32_t nj, int32_t nk,
                                         const gm1b_scalar_advection5_arrays *arrays, int32_t nrk, int32_t wflag,
                                         float dx, float dy, float dz, double weps, uint32_t lateral_obc,
                                         int32_t levels_per_chunk, void *stream) {
    return scalar_advection5_launch(ni, nj, nk, arrays, nrk, wflag, dx, dy, dz, weps, lateral_obc, levels_per_chunk,
                                    VertCol{0, nullptr, nullptr, 0.0f}, stream);
}

extern "C" int32_t gm1b_scalar_advection5_column(int32_t ni, int32_t nj, int32_t nk,
                                                const gm1b_scalar_advection5_arrays *arrays, int32_t nrk,
                                                int32_t wflag, float dx, float dy, double weps, uint32_t lateral_obc,
                                                int32_t levels_per_chunk, const gm1b_vertical_column *column,
                                                void *stream) {
    if (column == nullptr || (column->flat != 0 && column->flat != 1)) {
        gm1b_set_error("gm1b_scalar_advection5_column: need a vertical column with flat = 0 or 1");
        return GM1B_ERR_ARGUMENT;
    }
    if (column->flat ? (column->mh == nullptr || !(column->rdz > 0.0f) || !isfinite(column->rdz))
                     : column->rdsf == nullptr) {
        gm1b_set_error("gm1b_scalar_advection5_column: a flat column needs mh and rdz > 0, a terrain column rdsf");
        return GM1B_ERR_ARGUMENT;
    }
    const VertCol vc{column->flat ? 2 : 1, column->rdsf, column->mh, column->rdz};
    // dz only forms the uniform reciprocal, which a stretched column never reads
    return scalar_advection5_launch(ni, nj, nk, arrays, nrk, wflag, dx, dy, 1.0f, weps, lateral_obc,
                                    levels_per_chunk, vc, stream);
}
