// SGS stress tendencies of the flat (terrain_flag=.false.) stretched column:
// CM1 gettau and the momentum stress divergence turbu/turbv/turbw with their
// implicit vertical solves.
//
// Behaviour followed (reference file:line):
//   the strain carriers rho*Sij of calcdef's mass and face passes
//       gm1_flat_calcdef_mass_v1 / _face_v1
//       src/cm1core/cuda_gm1_flat_stretched_closure.py:76-114 (turb.F:4772-4786,
//       :4880-4895)
//   gettau with the free-slip lower and upper faces (enqueue_flat_gettau)
//       src/cm1core/cuda_gm1_flat_stretched_closure.py:134-161, :551-571
//       (turb.F:4094-4190, :4281-4433, :4536-4545)
//   turbu/turbuz, turbv/turbvz, turbw (enqueue_flat_momentum_stress, the
//   two-part block off)
//       src/cm1core/cuda_gm1_flat_stretched_closure.py:163-292, :574-618
//       (turbtend.F:1095-1361, :1438-1560, :1860-2128, :2194-2310, :2508-2885)
//
// Binary32 one operation at a time in the reference's statement order
// (--fmad=false; the literal zero factors of vibeta = 0 are formed, so signed
// zeros are what the reference's are).  Open sides are index clamps.
//
//   turbs for theta and the moisture rows (the flat fluxes and turbsz, the
//   open-halo pad/pack copies as index clamps; no surface flux)
//       src/cm1core/cuda_gm1_scalar_turbulence.py:453-466 (pad, pack)
//       src/cm1core/cuda_gm1_flat_stretched_closure.py:335-381 (flux, apply)
//       src/cm1core/cuda_cartesian_closure.py:1566-1633 (the per-scalar loop)
//       (turbtend.F:60-434, :442-692; solve1.F:1169-1233)
//   the dissipative heating, idiss = 1
//       src/cm1core/eqtset2_energy_terms.py:176-215, :375-470 (solve1.F:744-848, :917-975)
//   the upper Rayleigh damping held tendencies, irdamp = 1
//       src/cm1core/cuda_rayleigh_held.py:213-254, :419-488 (solve1.F:412-454)
//
// Design: the strain and gettau passes are grid-stride elementwise kernels
// over the union of their index spaces (one launch each).  A column solve's
// CTA owns 32 columns of a row: eight warps (or four) form the tridiagonal rows
// of their own runs of levels in shared memory ([level][column], conflict-free;
// every load and division spread over the CTA), one warp sweeps them, then all
// warps form the horizontal divergence and the cross term of their levels and
// add the tendency.  Against a thread per column (its loads one level at a time,
// too few columns in flight), 189x131x64: turbu 207 -> 56 us, turbv 141 ->
// 45, turbw 90 -> 39; turbs of theta and the three moisture rows, which share
// the matrix and its reciprocals, 285 -> 99.
#include "gm1b_common.cuh"

namespace gm1b {
namespace {

constexpr int kCX = 32, kCY = 4, kCT = kCX * kCY;  // column tile
constexpr int kEW = 256;                            // elementwise block
constexpr int kColWarps = 8;                        // warps of the scalar solve's CTA, which owns 32 columns of a row
constexpr int kTurbsGroup = 4;                      // scalars the turbs column pass solves together

#define TRY(x)                        \
    do {                              \
        const int r_ = (x);           \
        if (r_ != GM1B_OK) return r_; \
    } while (0)

bool launch_ok(const char *what) {
    const cudaError_t e = cudaPeekAtLastError();
    if (e != cudaSuccess) {
        cudaGetLastError();
        gm1b_set_error("%s: %s", what, cudaGetErrorString(e));
        return false;
    }
    return true;
}

struct StressArgs {
    const float *u, *v, *w, *rho, *rf, *mh, *mf, *mhp, *kmh, *kmv;
    float *s11, *s22, *s33, *s12, *s13, *s23;
    float *t11, *t22, *t33, *t12, *t13, *t23;
    float *uten, *vten, *wten;
    int ni, nj, nk;
    float rdx, rdy, rdz, dt;
};

__device__ __forceinline__ int clampi(int x, int n) { return x < 0 ? 0 : (x >= n ? n - 1 : x); }
__device__ __forceinline__ int clampr(int x, int lo, int hi) { return x < lo ? lo : (x > hi ? hi : x); }
// (k, j, i) of a layout with rows of nx words and ny rows per level
__device__ __forceinline__ unsigned o3(int k, int j, int i, int ny, int nx) {
    return ((unsigned)k * (unsigned)ny + (unsigned)j) * (unsigned)nx + (unsigned)i;
}
// a (.., nj, ni) carrier at a clamped column
__device__ __forceinline__ float cell(const StressArgs &a, const float *p, int k, int j, int i) {
    return p[o3(k, clampi(j, a.nj), clampi(i, a.ni), a.nj, a.ni)];
}

// ---------------------------------------------------------------- strain
__global__ void __launch_bounds__(kEW) flat_strain_kernel(StressArgs a) {
    const int ni = a.ni, nj = a.nj, nk = a.nk, ux = ni + 1, vy = nj + 1;
    const size_t total = (size_t)(nk + 1) * vy * ux;
    for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < total; q += (size_t)gridDim.x * blockDim.x) {
        const int ic = (int)(q % ux), jc = (int)((q / ux) % vy), k = (int)(q / ((size_t)ux * vy));
        if (k < nk) {
            if (ic < ni && jc < nj) {
                const unsigned p = o3(k, jc, ic, nj, ni);
                const float r = a.rho[p];
                a.s11[p] = (r * (a.u[o3(k, jc, ic + 1, nj, ux)] - a.u[o3(k, jc, ic, nj, ux)])) * a.rdx;
                a.s22[p] = (r * (a.v[o3(k, jc + 1, ic, vy, ni)] - a.v[o3(k, jc, ic, vy, ni)])) * a.rdy;
                a.s33[p] = (r * (a.w[o3(k + 1, jc, ic, nj, ni)] - a.w[o3(k, jc, ic, nj, ni)])) * (a.rdz * a.mhp[k + 1]);
            }
            const int ii = clampr(ic, 1, ni - 1), jj = clampr(jc, 1, nj - 1);
            const float x = (a.u[o3(k, jj, ii, nj, ux)] - a.u[o3(k, jj - 1, ii, nj, ux)]) * a.rdy;
            const float y = (a.v[o3(k, jj, ii, vy, ni)] - a.v[o3(k, jj, ii - 1, vy, ni)]) * a.rdx;
            const float rs = (a.rho[o3(k, jj - 1, ii - 1, nj, ni)] + a.rho[o3(k, jj, ii, nj, ni)]) +
                             (a.rho[o3(k, jj, ii - 1, nj, ni)] + a.rho[o3(k, jj - 1, ii, nj, ni)]);
            a.s12[o3(k, jc, ic, vy, ux)] = ((0.5f * (x + y)) * 0.25f) * rs;
        }
        if (k >= 1 && k < nk) {
            const int kf = k;
            if (jc < nj) {
                const int il = clampi(ic - 1, ni), ir = clampi(ic, ni);
                const float dw = (a.w[o3(kf, jc, ir, nj, ni)] - a.w[o3(kf, jc, il, nj, ni)]) * a.rdx;
                const float du = (((a.u[o3(kf, jc, ic, nj, ux)] - a.u[o3(kf - 1, jc, ic, nj, ux)]) * a.rdz) * 0.5f) *
                                 (a.mf[o3(kf, jc, il, nj, ni)] + a.mf[o3(kf, jc, ir, nj, ni)]);
                a.s13[o3(kf, jc, ic, nj, ux)] =
                    ((0.5f * (dw + du)) * 0.5f) * (a.rf[o3(kf, jc, il, nj, ni)] + a.rf[o3(kf, jc, ir, nj, ni)]);
            }
            if (ic < ni) {
                const int js = clampi(jc - 1, nj), jn = clampi(jc, nj);
                const float dw = (a.w[o3(kf, jn, ic, nj, ni)] - a.w[o3(kf, js, ic, nj, ni)]) * a.rdy;
                const float dv = (((a.v[o3(kf, jc, ic, vy, ni)] - a.v[o3(kf - 1, jc, ic, vy, ni)]) * a.rdz) * 0.5f) *
                                 (a.mf[o3(kf, js, ic, nj, ni)] + a.mf[o3(kf, jn, ic, nj, ni)]);
                a.s23[o3(kf, jc, ic, vy, ni)] =
                    ((0.5f * (dw + dv)) * 0.5f) * (a.rf[o3(kf, js, ic, nj, ni)] + a.rf[o3(kf, jn, ic, nj, ni)]);
            }
        }
    }
}

// ---------------------------------------------------------------- gettau
__global__ void __launch_bounds__(kEW) flat_gettau_kernel(StressArgs a) {
    const int ni = a.ni, nj = a.nj, nk = a.nk, ux = ni + 1, vy = nj + 1;
    const size_t total = (size_t)(nk + 1) * vy * ux;
    for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < total; q += (size_t)gridDim.x * blockDim.x) {
        const int ic = (int)(q % ux), jc = (int)((q / ux) % vy), k = (int)(q / ((size_t)ux * vy));
        if (k < nk) {
            if (ic < ni && jc < nj) {
                const unsigned p = o3(k, jc, ic, nj, ni), pu = o3(k + 1, jc, ic, nj, ni);
                const float m = a.kmh[p] + a.kmh[pu];
                a.t11[p] = a.s11[p] * m;
                a.t22[p] = a.s22[p] * m;
                a.t33[p] = a.s33[p] * m;
            }
            const int ii = clampr(ic, 1, ni - 1), jj = clampr(jc, 1, nj - 1);
            const float lo = (a.kmh[o3(k, jj - 1, ii - 1, nj, ni)] + a.kmh[o3(k, jj, ii, nj, ni)]) +
                             (a.kmh[o3(k, jj, ii - 1, nj, ni)] + a.kmh[o3(k, jj - 1, ii, nj, ni)]);
            const float hi = (a.kmh[o3(k + 1, jj - 1, ii - 1, nj, ni)] + a.kmh[o3(k + 1, jj, ii, nj, ni)]) +
                             (a.kmh[o3(k + 1, jj, ii - 1, nj, ni)] + a.kmh[o3(k + 1, jj - 1, ii, nj, ni)]);
            a.t12[o3(k, jc, ic, vy, ux)] = (a.s12[o3(k, jj, ii, vy, ux)] * 0.25f) * (lo + hi);
        }
        const int f = k, ff = f == 0 ? 1 : (f == nk ? nk - 1 : f);
        if (jc < nj)
            a.t13[o3(f, jc, ic, nj, ux)] =
                a.s13[o3(ff, jc, ic, nj, ux)] * (cell(a, a.kmv, ff, jc, ic - 1) + cell(a, a.kmv, ff, jc, ic));
        if (ic < ni)
            a.t23[o3(f, jc, ic, vy, ni)] =
                a.s23[o3(ff, jc, ic, vy, ni)] * (cell(a, a.kmv, ff, jc - 1, ic) + cell(a, a.kmv, ff, jc, ic));
    }
}

// ------------------------------------------------------- turbu and turbv
// DIR 0: a u column (j, f), f in [0, ni]; DIR 1: a v column (f, i), f in [0, nj];
// the cells either side of it are (ja, ia) and (jb, ib).
template <int DIR, int WARPS>
__global__ void __launch_bounds__(32 * WARPS) flat_turb_uv_kernel(const __grid_constant__ StressArgs a) {
    extern __shared__ float s_col[];
    const int lane = threadIdx.x, wy = threadIdx.y;
    const int ni = a.ni, nj = a.nj, K = a.nk, ux = ni + 1, vy = nj + 1;
    const int nx = DIR == 0 ? ux : ni, tiles = (nx + 31) / 32;
    const int c0 = blockIdx.x % tiles * 32 + lane, cy = blockIdx.x / tiles;
    const bool own = c0 < nx;
    const int cx = min(c0, nx - 1);  // lanes past the row's end repeat its last column and store nothing
    // DIR 0: column (j = cy, f = cx); DIR 1: column (f = cy, i = cx)
    const int ja = DIR == 0 ? cy : clampi(cy - 1, nj), jb = clampi(cy, nj);
    const int ia = DIR == 0 ? clampi(cx - 1, ni) : cx, ib = clampi(cx, ni);
    const unsigned ca = o3(0, ja, ia, nj, ni), cb = o3(0, jb, ib, nj, ni), cz = (unsigned)nj * ni;
    const float *q = DIR == 0 ? a.u : a.v;       // the column's wind
    const float *top = DIR == 0 ? a.t13 : a.t23;  // its t13/t23 (face levels)
    float *ten = DIR == 0 ? a.uten : a.vten;
    const unsigned col = (unsigned)cy * nx + cx, lev = DIR == 0 ? (unsigned)nj * ux : (unsigned)vy * ni;
    const float rd = DIR == 0 ? a.rdx : a.rdy, rdz = a.rdz, dt = a.dt;
    float *s_a = s_col + lane, *s_b = s_a + K * 32, *s_c = s_b + K * 32, *s_d = s_c + K * 32;
    auto pair = [&](const float *p, int k) { return p[k * cz + ca] + p[k * cz + cb]; };
    const float rdt = 0.5f / dt;
    const float tema = (((-0.0625f * dt) * 1.0f) * rdz) * rdz;
    const float temb = (((0.0625f * dt) * 0.0f) * rdz) * rdz;
    const float temc = (0.5f * dt) * rdz;
    const int run = (K + WARPS - 1) / WARPS;
    const int lo = min(wy * run, K), hi = min(lo + run, K);
    // the diffusivity product of a face, formed once and carried up
    auto face = [&](int f) { return f >= 1 && f < K ? (pair(a.kmv, f) * pair(a.mf, f)) * pair(a.rf, f) : 0.0f; };
    if (lo < hi) {
        float below = face(lo), qm = lo > 0 ? q[(lo - 1) * lev + col] : 0.0f, qk = q[lo * lev + col];
#pragma unroll 2
        for (int k = lo; k < hi; ++k) {
            const float rr0 = 1.0f / (0.5f * pair(a.rho, k));
            const float mhp = pair(a.mh, k), tem = mhp * rr0;
            const float above = face(k + 1), qp = k + 1 < K ? q[(k + 1) * lev + col] : 0.0f;
            const float r1 = below * tem, r2 = above * tem;
            const float cfa = tema * r1, cfc = tema * r2;
            float cfb, cfd;
            if (k == 0) {
                cfb = 1.0f - cfc;
                cfd = (qk + temb * (r2 * qp - r2 * qk)) - ((temc * top[col]) * mhp) * rr0;
            } else if (k == K - 1) {
                cfb = 1.0f - cfa;
                cfd = (qk + temb * (-(r1 * qk) + r1 * qm)) + ((temc * top[(unsigned)K * lev + col]) * mhp) * rr0;
            } else {
                cfb = (1.0f - cfa) - cfc;
                cfd = qk + temb * ((r2 * qp - (r1 + r2) * qk) + r1 * qm);
            }
            s_a[k * 32] = cfa, s_b[k * 32] = cfb, s_c[k * 32] = cfc, s_d[k * 32] = cfd;
            below = above, qm = qk, qk = qp;
        }
    }
    __syncthreads();
    // (chunks of four rows cost registers and CTAs an SM: 640x768x80 turbu 1115
    // us against 1005, turbw 828 against 541; with two the u columns spill 8 bytes)
    if (wy == 0) column_sweep<2>(s_a, s_b, s_c, s_d, K);
    __syncthreads();
    if (lo >= hi || !own) return;
    // the vertical and horizontal terms and the tendency of each level
    auto cross = [&](int k) {
        return k >= 1 && k < K ? ((((a.w[k * cz + cb] - a.w[k * cz + ca]) * rd) * 0.25f) * pair(a.kmv, k)) * pair(a.rf, k)
                               : 0.0f;
    };
    const unsigned corner = (unsigned)vy * ux, oc = o3(0, cy, cx, vy, ux), ou = oc + (DIR == 0 ? ux : 1);
    const bool ex = DIR == 0 ? cx == 0 || cx == ni : cx == 0 || cx == ni - 1;
    const bool ey = DIR == 0 ? cy == 0 || cy == nj - 1 : cy == 0 || cy == nj;
    const float *diag = DIR == 0 ? a.t11 : a.t22;
    float d7 = cross(lo);
#pragma unroll 2
    for (int k = lo; k < hi; ++k) {
        const unsigned p = (unsigned)k * lev + col;
        const float rho_p = pair(a.rho, k), old = ten[p];
        float tz = (rho_p * (s_d[k * 32] - q[p])) * rdt;
        const float d7_up = cross(k + 1);
        tz = tz + (((d7_up - d7) * rdz) * 0.5f) * pair(a.mh, k);
        d7 = d7_up;
        const float dd = diag[k * cz + cb] - diag[k * cz + ca];
        const float dc = a.t12[k * corner + ou] - a.t12[k * corner + oc];
        const float hx = ex ? 0.0f : (DIR == 0 ? dd : dc) * a.rdx;
        const float hy = ey ? 0.0f : (DIR == 0 ? dc : dd) * a.rdy;
        const float rrk = 1.0f / (0.5f * rho_p);
        ten[p] = old + ((hx + hy) + tz) * rrk;
    }
}

// ----------------------------------------------------------------- turbw
template <int WARPS>
__global__ void __launch_bounds__(32 * WARPS) flat_turbw_kernel(const __grid_constant__ StressArgs a) {
    extern __shared__ float s_col[];
    const int lane = threadIdx.x, wy = threadIdx.y;
    const int ni = a.ni, nj = a.nj, K = a.nk, n = K - 1, ux = ni + 1, vy = nj + 1, tiles = (ni + 31) / 32;
    const int i0 = blockIdx.x % tiles * 32 + lane, j = blockIdx.x / tiles;
    const bool own = i0 < ni;
    const int i = min(i0, ni - 1);  // lanes past the row's end repeat its last column and store nothing
    const unsigned col = (unsigned)j * ni + i, lev = (unsigned)nj * ni;
    const float rdz = a.rdz, dt = a.dt;
    float *s_a = s_col + lane, *s_b = s_a + n * 32, *s_c = s_b + n * 32, *s_d = s_c + n * 32;  // rows f - 1
    const float rdt = 1.0f / dt;
    const float tema = (((-1.0f * dt) * 1.0f) * rdz) * rdz;
    const float temb = ((dt * 0.0f) * rdz) * rdz;
    const float temc = dt * rdz;
    const int run = (n + WARPS - 1) / WARPS;
    const int lo = min(1 + wy * run, K), hi = min(lo + run, K);  // faces lo .. hi-1
    if (lo < hi) {
        unsigned z = (unsigned)lo * lev + col;
        float km = a.kmh[z - lev], k0 = a.kmh[z], mhm = a.mh[z - lev], rhom = a.rho[z - lev], wm = a.w[z - lev],
              wk = a.w[z];
#pragma unroll 2
        for (int f = lo; f < hi; ++f, z += lev) {
            const float rrf = a.mf[z] / a.rf[z];
            const float kp = a.kmh[z + lev], mh = a.mh[z], rho = a.rho[z], wp = a.w[z + lev];
            const float r1 = (((km + k0) * mhm) * rhom) * rrf, r2 = (((k0 + kp) * mh) * rho) * rrf;
            const float cfa = tema * r1, cfc = tema * r2;
            float cfb, cfd;
            if (f == 1) {
                cfb = 1.0f - cfc;
                cfd = (wk + temb * (r2 * wp - r2 * wk)) - (temc * a.t33[col]) * rrf;
            } else if (f == n) {
                cfb = 1.0f - cfa;
                cfd = (wk + temb * (-(r1 * wk) + r1 * wm)) + (temc * a.t33[z]) * rrf;
            } else {
                cfb = (1.0f - cfa) - cfc;
                cfd = wk + temb * ((r2 * wp - (r1 + r2) * wk) + r1 * wm);
            }
            const int p = (f - 1) * 32;
            s_a[p] = cfa, s_b[p] = cfb, s_c[p] = cfc, s_d[p] = cfd;
            km = k0, k0 = kp, mhm = mh, rhom = rho, wm = wk, wk = wp;
        }
    }
    __syncthreads();
    if (wy == 0) column_sweep<2>(s_a, s_b, s_c, s_d, n);
    __syncthreads();
    if (!own) return;
    const bool ex = i == 0 || i == ni - 1, ey = j == 0 || j == nj - 1;
#pragma unroll 2
    for (int f = lo; f < hi; ++f) {
        const unsigned p = (unsigned)f * lev + col, px = o3(f, j, i, nj, ux), py = o3(f, j, i, vy, ni);
        const float rff = a.rf[p], old = a.wten[p];
        const float tz = (rff * (s_d[(f - 1) * 32] - a.w[p])) * rdt;
        const float hx = ex ? 0.0f : (a.t13[px + 1] - a.t13[px]) * a.rdx;
        const float hy = ey ? 0.0f : (a.t23[py + ni] - a.t23[py]) * a.rdy;
        a.wten[p] = old + ((hx + hy) + tz) / rff;
    }
}

// ---------------------------------------------------------- turbs (flat)
// theta ((th0 - 300) + tha) and numq moisture rows.  The open-halo copies of
// the reference's pad/pack texts are index clamps here, so no halo array is
// written.  Two passes: the horizontal pass forms, per cell, the x and y
// flux divergence tx + ty of every scalar into the workspace (each face's
// factor (-0.125*(rho_l + rho_r))*(the four khh) formed once and shared by
// all scalars); the column pass solves turbsz's tridiagonal for each scalar
// and adds ((tx + ty) + tz)*rr, the reference's sum in its order.
struct TurbsArgs {
    const float *th0, *tha, *qa, *rho, *rr, *rf, *mh, *mf, *khh, *khv;
    float *thten, *qten, *work;
    int ni, nj, nk, nsc;
    float dx, dy, dz, dt;
};

__device__ __forceinline__ float tcell(const TurbsArgs &a, const float *p, int k, int j, int i) {
    return p[o3(k, clampi(j, a.nj), clampi(i, a.ni), a.nj, a.ni)];
}
// the open-halo scalar sc (0 theta, 1.. the moisture rows) at a clamped cell
__device__ __forceinline__ float sval(const TurbsArgs &a, int sc, int k, int j, int i) {
    const unsigned p = o3(k, clampi(j, a.nj), clampi(i, a.ni), a.nj, a.ni);
    if (sc > 0) return a.qa[(size_t)(sc - 1) * ((size_t)a.ni * a.nj * a.nk) + p];
    return (a.th0[k] - 300.0f) + a.tha[p];
}
// the face factor (-0.125*(rho(a)+rho(a-1)))*((khh(k)+khh(k)) + (khh(k+1)+khh(k+1)))
// across x face f (cells f-1, f) or y face f (rows f-1, f)
__device__ __forceinline__ float fac_x(const TurbsArgs &a, int k, int j, int f) {
    const float den = tcell(a, a.rho, k, j, f) + tcell(a, a.rho, k, j, f - 1);
    const float kh = (tcell(a, a.khh, k, j, f) + tcell(a, a.khh, k, j, f - 1)) +
                     (tcell(a, a.khh, k + 1, j, f) + tcell(a, a.khh, k + 1, j, f - 1));
    return (-0.125f * den) * kh;
}
__device__ __forceinline__ float fac_y(const TurbsArgs &a, int k, int f, int i) {
    const float den = tcell(a, a.rho, k, f, i) + tcell(a, a.rho, k, f - 1, i);
    const float kh = (tcell(a, a.khh, k, f, i) + tcell(a, a.khh, k, f - 1, i)) +
                     (tcell(a, a.khh, k + 1, f, i) + tcell(a, a.khh, k + 1, f - 1, i));
    return (-0.125f * den) * kh;
}

__global__ void __launch_bounds__(kCT) flat_turbs_horizontal_kernel(TurbsArgs a) {
    const int i = blockIdx.x * kCX + threadIdx.x, j = blockIdx.y * kCY + threadIdx.y, k = blockIdx.z;
    const int ni = a.ni, nj = a.nj;
    if (i >= ni || j >= nj) return;
    const size_t n = (size_t)ni * nj * a.nk, p = o3(k, j, i, nj, ni);
    const float rx = 1.0f / a.dx, ry = 1.0f / a.dy;
    const bool xin = !(i == 0 || i + 1 == ni), yin = !(j == 0 || j + 1 == nj);
    float fw = 0.0f, fe = 0.0f, fs = 0.0f, fn = 0.0f;
    if (xin) {
        fw = fac_x(a, k, j, i);
        fe = fac_x(a, k, j, i + 1);
    }
    if (yin) {
        fs = fac_y(a, k, j, i);
        fn = fac_y(a, k, j + 1, i);
    }
    for (int sc = 0; sc < a.nsc; ++sc) {
        float tx = 0.0f, ty = 0.0f;
        const float s0 = sval(a, sc, k, j, i);
        if (xin) {
            const float xw = (fw * (s0 - sval(a, sc, k, j, i - 1))) * rx;
            const float xe = (fe * (sval(a, sc, k, j, i + 1) - s0)) * rx;
            tx = -((xe - xw) * rx);
        }
        if (yin) {
            const float ys = (fs * (s0 - sval(a, sc, k, j - 1, i))) * ry;
            const float yn = (fn * (sval(a, sc, k, j + 1, i) - s0)) * ry;
            ty = -((yn - ys) * ry);
        }
        a.work[(size_t)sc * n + p] = tx + ty;
    }
}

// The matrix and its reciprocals are the same for every scalar: formed and
// swept once a column, then a warp per scalar of the group sweeps its right
// side.  Shared words per level and column: the matrix rows (the reciprocal in
// the diagonal's place) and one of each scalar.
__global__ void __launch_bounds__(32 * kColWarps) flat_turbs_column_kernel(const __grid_constant__ TurbsArgs a) {
    extern __shared__ float s_col[];
    const int lane = threadIdx.x, wy = threadIdx.y;
    const int ni = a.ni, nj = a.nj, nk = a.nk, tiles = (ni + 31) / 32;
    const int i0 = blockIdx.x % tiles * 32 + lane, j = blockIdx.x / tiles;
    const bool own = i0 < ni;
    const int i = min(i0, ni - 1);  // lanes past the row's end repeat its last column and store nothing
    const size_t n = (size_t)ni * nj * nk;
    const unsigned col = (unsigned)j * ni + i, lev = (unsigned)nj * ni;
    const int words = nk * 32;
    float *s_a = s_col + lane, *s_b = s_a + words, *s_c = s_b + words, *s_d = s_c + words;
    const float rz = 1.0f / a.dz, dt = a.dt, rdt = 1.0f / dt;
    const float tema = (((-1.0f * dt) * 1.0f) * rz) * rz;
    const float temb = ((dt * 0.0f) * rz) * rz;
    const float temc = dt * rz;
    const int run = (nk + kColWarps - 1) / kColWarps;
    const int lo = min(wy * run, nk), hi = min(lo + run, nk);
    auto face = [&](int f) {
        const unsigned z = (unsigned)f * lev + col;
        return f >= 1 && f < nk ? (a.khv[z] * a.mf[z]) * a.rf[z] : 0.0f;
    };
    for (int first = 0; first < a.nsc; first += kTurbsGroup) {
        const int group = min(kTurbsGroup, a.nsc - first);
        const float *src[kTurbsGroup];  // theta is (th0 - 300) + tha
#pragma unroll
        for (int g = 0; g < kTurbsGroup; ++g) {
            const int sc = first + min(g, group - 1);
            src[g] = (sc == 0 ? a.tha : a.qa + (size_t)(sc - 1) * n) + col;
        }
        auto scalar = [&](int g, int k) {
            const float x = src[g][(unsigned)k * lev];
            return first == 0 && g == 0 ? (a.th0[k] - 300.0f) + x : x;
        };
        if (lo < hi) {
            float below = face(lo), sm[kTurbsGroup], sk[kTurbsGroup];
#pragma unroll
            for (int g = 0; g < kTurbsGroup; ++g) {
                sm[g] = lo > 0 ? scalar(g, lo - 1) : 0.0f;
                sk[g] = scalar(g, lo);
            }
            for (int k = lo; k < hi; ++k) {
                const unsigned z = (unsigned)k * lev + col;
                const float mh = a.mh[z], rr = a.rr[z], above = face(k + 1);
                const float r1 = (below * mh) * rr, r2 = (above * mh) * rr;
                const float cfa = tema * r1, cfc = tema * r2, bc = ((temc * 0.0f) * mh) * rr;
                if (first == 0) {
                    s_a[k * 32] = cfa, s_c[k * 32] = cfc;
                    s_b[k * 32] = k == 0 ? 1.0f - cfc : k == nk - 1 ? 1.0f - cfa : (1.0f - cfa) - cfc;
                }
#pragma unroll
                for (int g = 0; g < kTurbsGroup; ++g) {
                    if (g >= group) break;
                    const float sp = k + 1 < nk ? scalar(g, k + 1) : 0.0f;
                    float cfd;
                    if (k == 0) {
                        const float ex = (-r2) * sk[g] + r2 * sp;
                        cfd = (sk[g] + temb * ex) + bc;
                    } else if (k == nk - 1) {
                        const float ex = r1 * sm[g] - r1 * sk[g];
                        cfd = (sk[g] + temb * ex) - bc;
                    } else {
                        const float ex = (r1 * sm[g] - (r1 + r2) * sk[g]) + r2 * sp;
                        cfd = sk[g] + temb * ex;
                    }
                    s_d[g * words + k * 32] = cfd;
                    sm[g] = sk[g], sk[g] = sp;
                }
                below = above;
            }
        }
        __syncthreads();
        if (first == 0) {
            if (wy == 0) {
                float cprev = 0.0f;
#pragma unroll 4
                for (int k = 0; k < nk; ++k) {
                    const float inv = rcp_rn(k == 0 ? s_b[0] : s_a[k * 32] * cprev + s_b[k * 32]);
                    cprev = (-s_c[k * 32]) * inv;
                    s_b[k * 32] = inv, s_c[k * 32] = cprev;
                }
            }
            __syncthreads();
        }
        if (wy < group) {
            float *d = s_d + wy * words;
            float prev = d[0] * s_b[0];
            d[0] = prev;
#pragma unroll 8
            for (int k = 1; k < nk; ++k) {
                prev = (d[k * 32] - s_a[k * 32] * prev) * s_b[k * 32];
                d[k * 32] = prev;
            }
#pragma unroll 8
            for (int k = nk - 2; k >= 0; --k) {
                prev = s_c[k * 32] * prev + d[k * 32];
                d[k * 32] = prev;
            }
        }
        __syncthreads();
        if (own) {
            for (int k = lo; k < hi; ++k) {
                const unsigned z = (unsigned)k * lev + col;
                const float rho = a.rho[z], rr = a.rr[z];
#pragma unroll
                for (int g = 0; g < kTurbsGroup; ++g) {
                    if (g >= group) break;
                    const int sc = first + g;
                    float *target = sc == 0 ? a.thten : a.qten + (size_t)(sc - 1) * n;
                    const float tz = (rho * (s_d[g * words + k * 32] - scalar(g, k))) * rdt;
                    target[z] = target[z] + (a.work[(size_t)sc * n + z] + tz) * rr;
                }
            }
        }
        __syncthreads();  // the next group's right sides take these words
    }
}

// ------------------------------------------------------ Rayleigh (upper)
// irdamp = 1: uten1 = ((-rdalpha*0.5)*(tauh(i-1)+tauh(i)))*(ua - u0(k)), vten1
// across j, wten1 = (-rdalpha*tauf)*wa, thten1 = (-rdalpha*taus)*tha.  tau
// as one-halo 3-D arrays (the reference's layout) or as column profiles;
// add_momentum adds the damping into the momentum outputs (the closure's
// held sum uten1 + uten) and assigns thten1.
struct RayArgs {
    const float *tauh, *taus, *tauf, *u0, *v0, *ua, *va, *wa, *tha;
    float *uten1, *vten1, *wten1, *thten1;
    int ni, nj, nk;
    float rdalpha;
    int profiles, add_momentum;
};

__device__ __forceinline__ float tau_at(const RayArgs &a, const float *tau, int k, int jh, int ih) {
    return a.profiles ? tau[k] : tau[((size_t)k * (a.nj + 2) + jh) * (size_t)(a.ni + 2) + ih];
}

__global__ void __launch_bounds__(kEW) rayleigh_held_kernel(RayArgs a) {
    const int ni = a.ni, nj = a.nj, nk = a.nk;
    const size_t first = (size_t)blockIdx.x * blockDim.x + threadIdx.x, step = (size_t)gridDim.x * blockDim.x;
    const size_t nu = (size_t)nk * nj * (ni + 1), nv = (size_t)nk * (nj + 1) * ni, ns = (size_t)nk * nj * ni;
    const float neg = -a.rdalpha, negh = neg * 0.5f;
    for (size_t z = first; z < nu; z += step) {
        const int f = (int)(z % (ni + 1)), j = (int)((z / (ni + 1)) % nj), k = (int)(z / ((size_t)(ni + 1) * nj));
        const float pair = tau_at(a, a.tauh, k, j + 1, f) + tau_at(a, a.tauh, k, j + 1, f + 1);
        const float d = (negh * pair) * (a.ua[z] - a.u0[k]);
        a.uten1[z] = a.add_momentum ? d + a.uten1[z] : d;
    }
    for (size_t z = first; z < nv; z += step) {
        const int i = (int)(z % ni), f = (int)((z / ni) % (nj + 1)), k = (int)(z / ((size_t)ni * (nj + 1)));
        const float pair = tau_at(a, a.tauh, k, f, i + 1) + tau_at(a, a.tauh, k, f + 1, i + 1);
        const float d = (negh * pair) * (a.va[z] - a.v0[k]);
        a.vten1[z] = a.add_momentum ? d + a.vten1[z] : d;
    }
    for (size_t z = first; z < ns; z += step) {
        const int i = (int)(z % ni), j = (int)((z / ni) % nj), k = (int)(z / ((size_t)ni * nj));
        const float dw = (neg * tau_at(a, a.tauf, k, j + 1, i + 1)) * a.wa[z];
        a.wten1[z] = a.add_momentum ? dw + a.wten1[z] : dw;
        a.thten1[z] = (neg * tau_at(a, a.taus, k, j + 1, i + 1)) * a.tha[z];
    }
}


// ---------------------------------------------------- dissipative heating
// idiss = 1: thten1 += (0.5*(dissten(k)+dissten(k+1))) /
// ((cpdcv*cvm)*(pi0+ppi)), cvm = ((cv + cvv*qv) + cpl*ql) + cpi*qice.
struct DissArgs {
    const float *dissten, *pi0, *ppi, *qa;
    float *thten1;
    int ni, nj, nk;
};

__global__ void __launch_bounds__(kEW) dissipative_heating_kernel(DissArgs a) {
    const float rd = 287.04f, cp = 1005.7f, cpv = 1870.0f, rv = 461.5f, cpl = 4190.0f, cpi = 2106.0f;
    const float cv = cp - rd, cvv = cpv - rv, cpdcv = cp / cv;
    const size_t plane = (size_t)a.ni * a.nj, n = plane * a.nk;
    for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (size_t)gridDim.x * blockDim.x) {
        const int k = (int)(q / plane);
        const float ql = a.qa[n + q] + a.qa[2 * n + q];
        const float qice = (a.qa[3 * n + q] + a.qa[4 * n + q]) + a.qa[5 * n + q];
        float cvm = cv + cvv * a.qa[q];
        cvm = cvm + cpl * ql;
        cvm = cvm + cpi * qice;
        const float epsd = 0.5f * (a.dissten[q] + a.dissten[q + plane]);
        const float den = (cpdcv * cvm) * (a.pi0[k] + a.ppi[q]);
        a.thten1[q] = a.thten1[q] + epsd / den;
    }
}

// ------------------------------------------------------------------ host
int stress_args(int32_t ni, int32_t nj, int32_t nk, const gm1b_flat_stress_arrays *s, float dx, float dy, float rdz,
                float dt, bool need_dt, StressArgs &a, const char *what) {
    if (s == nullptr || ni < 3 || nj < 3 || nk < 3) {
        gm1b_set_error("%s: need arrays, ni >= 3, nj >= 3, nk >= 3", what);
        return GM1B_ERR_ARGUMENT;
    }
    if ((double)(nk + 1) * (nj + 1) * (ni + 1) >= 2147483648.0) {
        gm1b_set_error("%s: a %dx%dx%d grid reaches 2^31 words; the kernels index with 32-bit offsets", what, ni, nj,
                       nk);
        return GM1B_ERR_ARGUMENT;
    }
    if (!(dx > 0.0f && dy > 0.0f && rdz > 0.0f) || !isfinite(dx) || !isfinite(dy) || !isfinite(rdz) ||
        (need_dt && !(dt > 0.0f && isfinite(dt)))) {
        gm1b_set_error("%s: dx, dy, rdz%s must be finite and > 0", what, need_dt ? ", dt" : "");
        return GM1B_ERR_ARGUMENT;
    }
    a = StressArgs{};
    a.u = s->u3d;
    a.v = s->v3d;
    a.w = s->w3d;
    a.rho = s->rho;
    a.rf = s->rf;
    a.mh = s->mh;
    a.mf = s->mf;
    a.mhp = s->mh_profile;
    a.kmh = s->kmh;
    a.kmv = s->kmv;
    a.s11 = s->s11;
    a.s22 = s->s22;
    a.s33 = s->s33;
    a.s12 = s->s12;
    a.s13 = s->s13;
    a.s23 = s->s23;
    a.t11 = s->t11;
    a.t22 = s->t22;
    a.t33 = s->t33;
    a.t12 = s->t12;
    a.t13 = s->t13;
    a.t23 = s->t23;
    a.uten = s->uten;
    a.vten = s->vten;
    a.wten = s->wten;
    a.ni = ni;
    a.nj = nj;
    a.nk = nk;
    a.rdx = 1.0f / dx;
    a.rdy = 1.0f / dy;
    a.rdz = rdz;
    a.dt = dt;
    return GM1B_OK;
}

bool all_set(std::initializer_list<const void *> ps) {
    for (const void *p : ps)
        if (p == nullptr) return false;
    return true;
}

unsigned ew_blocks(int ni, int nj, int nk) {
    const size_t total = (size_t)(nk + 1) * (nj + 1) * (ni + 1);
    const size_t want = (total + kEW - 1) / kEW, cap = (size_t)148 * 16;
    return (unsigned)(want < cap ? want : cap);
}

int enqueue_strain(const StressArgs &a, cudaStream_t st) {
    ProfScope ps("flat_strain_kernel", st);
    flat_strain_kernel<<<ew_blocks(a.ni, a.nj, a.nk), kEW, 0, st>>>(a);
    ps.stop();
    return launch_ok("flat_strain_kernel") ? GM1B_OK : GM1B_ERR_CUDA;
}

int enqueue_gettau(const StressArgs &a, cudaStream_t st) {
    ProfScope ps("flat_gettau_kernel", st);
    flat_gettau_kernel<<<ew_blocks(a.ni, a.nj, a.nk), kEW, 0, st>>>(a);
    ps.stop();
    return launch_ok("flat_gettau_kernel") ? GM1B_OK : GM1B_ERR_CUDA;
}

template <typename Kernel>
int configure(Kernel kernel, size_t smem, const char *name) {
    if (smem <= 48 * 1024) return GM1B_OK;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) {
        cudaGetLastError();
        gm1b_set_error("cudaFuncSetAttribute(%s): %s", name, cudaGetErrorString(e));
        return GM1B_ERR_CUDA;
    }
    return GM1B_OK;
}

template <int WARPS>
int momentum_solves(const StressArgs &a, cudaStream_t st) {
    const size_t words = (size_t)4 * a.nk * 32 * sizeof(float);
    TRY(configure(flat_turb_uv_kernel<0, WARPS>, words, "flat_turb_uv_kernel<0>"));
    TRY(configure(flat_turb_uv_kernel<1, WARPS>, words, "flat_turb_uv_kernel<1>"));
    TRY(configure(flat_turbw_kernel<WARPS>, words, "flat_turbw_kernel"));
    const dim3 cta(32, WARPS);
    auto tiles = [](int nx, int ny) { return (unsigned)((nx + 31) / 32) * (unsigned)ny; };
    {
        ProfScope ps("flat_turbu_kernel", st);
        flat_turb_uv_kernel<0, WARPS><<<tiles(a.ni + 1, a.nj), cta, words, st>>>(a);
        ps.stop();
        if (!launch_ok("flat_turbu_kernel")) return GM1B_ERR_CUDA;
    }
    {
        ProfScope ps("flat_turbv_kernel", st);
        flat_turb_uv_kernel<1, WARPS><<<tiles(a.ni, a.nj + 1), cta, words, st>>>(a);
        ps.stop();
        if (!launch_ok("flat_turbv_kernel")) return GM1B_ERR_CUDA;
    }
    ProfScope ps("flat_turbw_kernel", st);
    flat_turbw_kernel<WARPS><<<tiles(a.ni, a.nj), cta, words, st>>>(a);
    ps.stop();
    return launch_ok("flat_turbw_kernel") ? GM1B_OK : GM1B_ERR_CUDA;
}

int enqueue_momentum(const StressArgs &a, cudaStream_t st) {
    if (a.nk > 200) {
        gm1b_set_error("gm1b_flat_momentum_stress: nk=%d exceeds the column solves' shared memory (nk <= 200)", a.nk);
        return GM1B_ERR_ARGUMENT;
    }
    // Four warps a CTA for columns of up to 40 levels on a plane that gives nine
    // CTAs an SM, else eight: short runs of levels form their end faces twice, and
    // the other warps wait for the sweep.  The three solves of 640x500x24 with
    // eight and four warps 524 and 477 us (a thread per column 508), 256x256x40
    // 198 and 196, 640x500x56 1119 and 1362, 128x100x24 38 and 47.
    const size_t tiles = (size_t)((a.ni + 31) / 32) * a.nj;
    return a.nk <= 40 && tiles >= 9 * 148 ? momentum_solves<4>(a, st) : momentum_solves<8>(a, st);
}

}  // namespace
}  // namespace gm1b

using namespace gm1b;

extern "C" int32_t gm1b_flat_strain(int32_t ni, int32_t nj, int32_t nk, const gm1b_flat_stress_arrays *arrays,
                                    float dx, float dy, float rdz, void *stream) {
    StressArgs a;
    TRY(stress_args(ni, nj, nk, arrays, dx, dy, rdz, 1.0f, false, a, "gm1b_flat_strain"));
    if (!all_set({a.u, a.v, a.w, a.rho, a.rf, a.mf, a.mhp, a.s11, a.s22, a.s33, a.s12, a.s13, a.s23})) {
        gm1b_set_error("gm1b_flat_strain: a required array is NULL");
        return GM1B_ERR_ARGUMENT;
    }
    return enqueue_strain(a, static_cast<cudaStream_t>(stream));
}

extern "C" int32_t gm1b_flat_gettau(int32_t ni, int32_t nj, int32_t nk, const gm1b_flat_stress_arrays *arrays,
                                    void *stream) {
    StressArgs a;
    TRY(stress_args(ni, nj, nk, arrays, 1.0f, 1.0f, 1.0f, 1.0f, false, a, "gm1b_flat_gettau"));
    if (!all_set({a.s11, a.s22, a.s33, a.s12, a.s13, a.s23, a.kmh, a.kmv, a.t11, a.t22, a.t33, a.t12, a.t13, a.t23})) {
        gm1b_set_error("gm1b_flat_gettau: a required array is NULL");
        return GM1B_ERR_ARGUMENT;
    }
    return enqueue_gettau(a, static_cast<cudaStream_t>(stream));
}

extern "C" int32_t gm1b_flat_momentum_stress(int32_t ni, int32_t nj, int32_t nk,
                                             const gm1b_flat_stress_arrays *arrays, float dx, float dy, float rdz,
                                             float dt, void *stream) {
    StressArgs a;
    TRY(stress_args(ni, nj, nk, arrays, dx, dy, rdz, dt, true, a, "gm1b_flat_momentum_stress"));
    if (!all_set({a.t11, a.t22, a.t33, a.t12, a.t13, a.t23, a.kmh, a.kmv, a.rho, a.rf, a.mh, a.mf, a.u, a.v, a.w,
                  a.uten, a.vten, a.wten})) {
        gm1b_set_error("gm1b_flat_momentum_stress: a required array is NULL");
        return GM1B_ERR_ARGUMENT;
    }
    return enqueue_momentum(a, static_cast<cudaStream_t>(stream));
}

extern "C" int32_t gm1b_flat_sgs_stress(int32_t ni, int32_t nj, int32_t nk, const gm1b_flat_stress_arrays *arrays,
                                        float dx, float dy, float rdz, float dt, void *stream) {
    TRY(gm1b_flat_strain(ni, nj, nk, arrays, dx, dy, rdz, stream));
    TRY(gm1b_flat_gettau(ni, nj, nk, arrays, stream));
    return gm1b_flat_momentum_stress(ni, nj, nk, arrays, dx, dy, rdz, dt, stream);
}

extern "C" int64_t gm1b_flat_scalar_turbulence_workspace_words(int32_t ni, int32_t nj, int32_t nk, int32_t numq) {
    if (ni < 1 || nj < 1 || nk < 1 || numq < 0) return 0;
    return (int64_t)(numq + 1) * ni * nj * nk;
}

extern "C" int32_t gm1b_flat_scalar_turbulence(int32_t ni, int32_t nj, int32_t nk, int32_t numq,
                                               const gm1b_flat_scalar_turbulence_arrays *arrays, float dx, float dy,
                                               float dz, float dt, void *stream) {
    const gm1b_flat_scalar_turbulence_arrays *s = arrays;
    if (s == nullptr || ni < 3 || nj < 3 || nk < 3 || numq < 0 || numq > 6) {
        gm1b_set_error("gm1b_flat_scalar_turbulence: need arrays, ni >= 3, nj >= 3, nk >= 3, numq in 0..6");
        return GM1B_ERR_ARGUMENT;
    }
    if ((double)(nk + 1) * nj * ni >= 2147483648.0) {
        gm1b_set_error("gm1b_flat_scalar_turbulence: a %dx%dx%d grid is too large for 32-bit offsets", ni, nj, nk);
        return GM1B_ERR_ARGUMENT;
    }
    if (!(dx > 0.0f && dy > 0.0f && dz > 0.0f && dt > 0.0f) || !isfinite(dx) || !isfinite(dy) || !isfinite(dz) ||
        !isfinite(dt)) {
        gm1b_set_error("gm1b_flat_scalar_turbulence: dx, dy, dz, dt must be finite and > 0");
        return GM1B_ERR_ARGUMENT;
    }
    if (!all_set({s->th0, s->tha, s->rho, s->rr, s->rf, s->mh, s->mf, s->khh, s->khv, s->thten, s->workspace}) ||
        (numq > 0 && !all_set({s->qa, s->qten}))) {
        gm1b_set_error("gm1b_flat_scalar_turbulence: a required array (or the workspace) is NULL");
        return GM1B_ERR_ARGUMENT;
    }
    // nk <= 200: 179200 bytes for a full group
    const size_t smem = (size_t)(3 + (numq + 1 < kTurbsGroup ? numq + 1 : kTurbsGroup)) * nk * 32 * sizeof(float);
    if (nk > 200) {
        gm1b_set_error("gm1b_flat_scalar_turbulence: nk=%d exceeds the column solve's shared memory (nk <= 200)", nk);
        return GM1B_ERR_ARGUMENT;
    }
    TRY(configure(flat_turbs_column_kernel, smem, "flat_turbs_column_kernel"));
    TurbsArgs a{s->th0, s->tha, s->qa, s->rho, s->rr, s->rf, s->mh, s->mf, s->khh, s->khv, s->thten, s->qten,
                s->workspace, ni, nj, nk, numq + 1, dx, dy, dz, dt};
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const dim3 tile(kCX, kCY), cols((ni + kCX - 1) / kCX, (nj + kCY - 1) / kCY);
    {
        ProfScope ps("flat_turbs_horizontal_kernel", st);
        flat_turbs_horizontal_kernel<<<dim3(cols.x, cols.y, nk), tile, 0, st>>>(a);
        ps.stop();
        if (!launch_ok("flat_turbs_horizontal_kernel")) return GM1B_ERR_CUDA;
    }
    ProfScope ps("flat_turbs_column_kernel", st);
    flat_turbs_column_kernel<<<(unsigned)((ni + 31) / 32) * (unsigned)nj, dim3(32, kColWarps), smem, st>>>(a);
    ps.stop();
    return launch_ok("flat_turbs_column_kernel") ? GM1B_OK : GM1B_ERR_CUDA;
}

extern "C" int32_t gm1b_rayleigh_held(int32_t ni, int32_t nj, int32_t nk, const gm1b_rayleigh_held_arrays *arrays,
                                      int32_t profiles, int32_t add_momentum, float rdalpha, void *stream) {
    const gm1b_rayleigh_held_arrays *s = arrays;
    if (s == nullptr || ni < 1 || nj < 1 || nk < 1 || (profiles != 0 && profiles != 1) ||
        (add_momentum != 0 && add_momentum != 1)) {
        gm1b_set_error("gm1b_rayleigh_held: need arrays, ni, nj, nk >= 1, profiles and add_momentum 0 or 1");
        return GM1B_ERR_ARGUMENT;
    }
    if (!(rdalpha >= 0.0f) || !isfinite(rdalpha)) {
        gm1b_set_error("gm1b_rayleigh_held: rdalpha must be finite and >= 0");
        return GM1B_ERR_ARGUMENT;
    }
    if (!all_set({s->tauh, s->taus, s->tauf, s->u0, s->v0, s->ua, s->va, s->wa, s->tha, s->uten1, s->vten1, s->wten1,
                  s->thten1})) {
        gm1b_set_error("gm1b_rayleigh_held: a required array is NULL");
        return GM1B_ERR_ARGUMENT;
    }
    RayArgs a{s->tauh, s->taus, s->tauf, s->u0,    s->v0,    s->ua,    s->va,    s->wa, s->tha,
              s->uten1, s->vten1, s->wten1, s->thten1, ni, nj, nk, rdalpha, profiles, add_momentum};
    const size_t most = (size_t)nk * (nj + 1) * (ni + 1);
    const size_t want = (most + kEW - 1) / kEW, cap = (size_t)148 * 16;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    ProfScope ps("rayleigh_held_kernel", st);
    rayleigh_held_kernel<<<(unsigned)(want < cap ? want : cap), kEW, 0, st>>>(a);
    ps.stop();
    return launch_ok("rayleigh_held_kernel") ? GM1B_OK : GM1B_ERR_CUDA;
}

extern "C" int32_t gm1b_dissipative_heating(int32_t ni, int32_t nj, int32_t nk,
                                            const gm1b_dissipative_heating_arrays *arrays, void *stream) {
    const gm1b_dissipative_heating_arrays *s = arrays;
    if (s == nullptr || ni < 1 || nj < 1 || nk < 1) {
        gm1b_set_error("gm1b_dissipative_heating: need arrays and ni, nj, nk >= 1");
        return GM1B_ERR_ARGUMENT;
    }
    if (!all_set({s->dissten, s->pi0, s->ppi, s->qa, s->thten1})) {
        gm1b_set_error("gm1b_dissipative_heating: a required array is NULL");
        return GM1B_ERR_ARGUMENT;
    }
    DissArgs a{s->dissten, s->pi0, s->ppi, s->qa, s->thten1, ni, nj, nk};
    const size_t n = (size_t)ni * nj * nk, want = (n + kEW - 1) / kEW, cap = (size_t)148 * 16;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    ProfScope ps("dissipative_heating_kernel", st);
    dissipative_heating_kernel<<<(unsigned)(want < cap ? want : cap), kEW, 0, st>>>(a);
    ps.stop();
    return launch_ok("dissipative_heating_kernel") ? GM1B_OK : GM1B_ERR_CUDA;
}
