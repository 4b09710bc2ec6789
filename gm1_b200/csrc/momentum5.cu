// momentum5.cu - sm_100a kernels of the terrain/open fifth-order momentum
// advection of the padded (ng = 3) lane: the mass fluxes rru, rrv, rrw (with
// the terrain term), the divergence divx, and the advu / advv / advw
// increments of uten / vten / wten, for CM1's lateral families.
//
// Behaviour followed (reference file:line):
//   cpu_terrain_open_momentum_advection5_inplace
//       src/cm1core/cuda_momentum_advection5.py:753-1068
//   lateral families (periodic wrap, open-side inflow substitution and
//   edits)  :103-208
//
// Design (B200): two launches instead of the reference's six.  (1) every mass
// flux and divx, in a march of the cells' columns; (2) one momentum pass whose
// warps march rows of u, v or w faces up the column.
// Upwind face fluxes read the six points that hold both upwind stencils
// before the mass-flux sign is known, so no load waits on it.
// Binary32 one operation at a time in the reference's order: word-identical.
#include "gm1b_common.cuh"

namespace gm1b {
namespace {

constexpr int G = 3;

struct MomArgs {
    const float *u3d, *v3d, *w3d, *uh, *vh;
    const float *rho0, *rf0, *rrf0, *c2, *gz, *gzu, *gzv, *rgzu, *rgzv, *dzdx, *dzdy;
    float *uten, *vten, *wten, *rru, *rrv, *rrw, *divx;
    int ni, nj, nk;
    int per[4], opn[4];  // west, east, south, north
    float rdx, rdy, rdz, dz;
    // vertical column: 0 uniform (dz); 1 terrain branch on a stretched column
    // (sigma, sigmaf, rds, rdsf profiles, physical top ztop, base density from
    // the padded rho0p); 2 flat column (rdz*mh / rdz*mf, the column's rho0p,
    // rf0, rr0, rrf0; no terrain terms), cuda_gm1_child_stretched_momentum.py:56-330
    int vmode;
    const float *rho0p, *sigma, *sigmaf, *rds, *rdsf, *mh, *mf, *rr0;
    float ztop, rdzm;
};

// 32-bit element offsets (the host refuses grids whose padded arrays reach
// 2^31 words)
__device__ __forceinline__ unsigned iu(const MomArgs &a, int k, int y, int x) {
    return ((unsigned)k * (unsigned)(a.nj + 2 * G) + (unsigned)y) * (unsigned)(a.ni + 1 + 2 * G) + (unsigned)x;
}
__device__ __forceinline__ unsigned iv(const MomArgs &a, int k, int y, int x) {
    return ((unsigned)k * (unsigned)(a.nj + 1 + 2 * G) + (unsigned)y) * (unsigned)(a.ni + 2 * G) + (unsigned)x;
}
__device__ __forceinline__ unsigned iw(const MomArgs &a, int k, int y, int x) {
    return ((unsigned)k * (unsigned)(a.nj + 2 * G) + (unsigned)y) * (unsigned)(a.ni + 2 * G) + (unsigned)x;
}
__device__ __forceinline__ unsigned ic(const MomArgs &a, int k, int j, int i) {
    return ((unsigned)k * (unsigned)a.nj + (unsigned)j) * (unsigned)a.ni + (unsigned)i;
}
__device__ __forceinline__ int clampn(int x, int n) { return x < 0 ? 0 : (x >= n ? n - 1 : x); }
// periodic wraps of a cell (c*) and a face (f*) index
__device__ __forceinline__ int cxw(const MomArgs &a, int i) {
    return (a.per[0] && i < 0) ? i + a.ni : ((a.per[1] && i >= a.ni) ? i - a.ni : i);
}
__device__ __forceinline__ int fxw(const MomArgs &a, int i) {
    return (a.per[0] && i < 0) ? i + a.ni : ((a.per[1] && i > a.ni) ? i - a.ni : i);
}
__device__ __forceinline__ int cyw(const MomArgs &a, int j) {
    return (a.per[2] && j < 0) ? j + a.nj : ((a.per[3] && j >= a.nj) ? j - a.nj : j);
}
__device__ __forceinline__ int fyw(const MomArgs &a, int j) {
    return (a.per[2] && j < 0) ? j + a.nj : ((a.per[3] && j > a.nj) ? j - a.nj : j);
}
// x * the column's vertical reciprocal at mass level k (uniform rdz, the
// terrain branch's rdsf(k), or the flat column's (x*rdz)*mh(k))
template <bool FLAT> __device__ __forceinline__ float zmass(const MomArgs &a, float x, int k) {
    if (FLAT) return (x * a.rdzm) * __ldg(a.mh + k);
    return x * (a.vmode == 1 ? __ldg(a.rdsf + k) : a.rdz);
}
// the same at w level kf (rds(kf) / (x*rdz)*mf(kf))
template <bool FLAT> __device__ __forceinline__ float zface(const MomArgs &a, float x, int kf) {
    if (FLAT) return (x * a.rdzm) * __ldg(a.mf + kf);
    return x * (a.vmode == 1 ? __ldg(a.rds + kf) : a.rdz);
}
// a boundary correction: uniform and terrain ((q*c)*(r*h)) as adv.F is
// grouped in the uniform text; the flat text groups it ((q*c)*r)*h
template <bool FLAT> __device__ __forceinline__ float bcorr(float q, float c, float r, float h) {
    return FLAT ? ((q * c) * r) * h : q * (c * (r * h));
}

__device__ __forceinline__ float up5(float m, float s0, float s1, float s2, float s3, float s4, float s5) {
    const bool pos = m >= 0.0f;
    const float r = flx5(pos ? s0 : s5, pos ? s1 : s4, pos ? s2 : s3, pos ? s3 : s2, pos ? s4 : s1);
    return m * r;
}

#define LU(k, y, x) __ldg(a.u3d + iu(a, (k), (y), (x)))
#define LV(k, y, x) __ldg(a.v3d + iv(a, (k), (y), (x)))
#define LW(k, y, x) __ldg(a.w3d + iw(a, (k), (y), (x)))
#define RU(k, y, x) a.rru[iu(a, (k), (y), (x))]
#define RV(k, y, x) a.rrv[iv(a, (k), (y), (x))]
#define RW(k, y, x) a.rrw[iw(a, (k), (y), (x))]

// (1) the mass fluxes rru, rrv, rrw and their divergence divx.  A thread owns
// a column of cells and marches a chunk of levels: it forms the fluxes of its
// four side faces (and writes the west and south ones), carries them and its
// lower vertical flux up, so the five outputs leave from one read of the
// winds.  Bound by memory.  Against
// the horizontal fluxes and the rest in two passes of a thread per point:
// 640x768x80 flat 0.474 -> 0.259 ms, 256x256x80 111 -> 66 us (two levels a
// trip 0.268 and 76, two levels a thread 0.312 and 93).
// ((ni+31)/32)*((nj+7)/8) tiles in grid.x, chunks of levels in grid.y.
constexpr int kFluxRows = 8;
template <int VM>
__global__ void __launch_bounds__(32 * kFluxRows) mom5_flux_kernel(const __grid_constant__ MomArgs a, int chunk) {
    const int ni = a.ni, nj = a.nj, nk = a.nk, tiles = (ni + 31) / 32;
    const int i = blockIdx.x % tiles * 32 + threadIdx.x, j = blockIdx.x / tiles * kFluxRows + threadIdx.y;
    if (i >= ni || j >= nj) return;
    const int y = j + G, x = i + G;
    const int wi = max(i - 1, 0), ie = min(i + 1, ni - 1), js = max(j - 1, 0), jn = min(j + 1, nj - 1);
    float gu0 = 0.0f, gu1 = 0.0f, gv0 = 0.0f, gv1 = 0.0f, dzdx = 0.0f, dzdy = 0.0f, gz = 0.0f;
    if (VM != 2) {
        const size_t c2d = (size_t)j * ni + i, u2d = (size_t)j * (ni + 1) + i;
        gu0 = __ldg(a.rgzu + u2d), gu1 = __ldg(a.rgzu + u2d + 1);
        gv0 = __ldg(a.rgzv + c2d), gv1 = __ldg(a.rgzv + c2d + ni);
        dzdx = __ldg(a.dzdx + c2d), dzdy = __ldg(a.dzdy + c2d), gz = __ldg(a.gz + c2d);
    }
    struct Flux {
        float w, e, s, n;
    };
    auto flux = [&](int k) {
        Flux f;
        const float u0 = LU(k, y, x), u1 = LU(k, y, x + 1), v0 = LV(k, y, x), v1 = LV(k, y + 1, x);
        if (VM == 2) {  // flat column: rho0(1,1,k) u and rho0(1,1,k) v
            const float r0 = __ldg(a.rho0p + iw(a, k, G, G));
            f.w = r0 * u0, f.e = r0 * u1, f.s = r0 * v0, f.n = r0 * v1;
            return f;
        }
        float c, w, e, so, n;
        if (VM == 1) {
            c = __ldg(a.rho0p + iw(a, k, y, x));
            w = __ldg(a.rho0p + iw(a, k, y, x - 1)), e = __ldg(a.rho0p + iw(a, k, y, x + 1));
            so = __ldg(a.rho0p + iw(a, k, y - 1, x)), n = __ldg(a.rho0p + iw(a, k, y + 1, x));
        } else {
            c = __ldg(a.rho0 + ic(a, k - 1, j, i));
            w = __ldg(a.rho0 + ic(a, k - 1, j, wi)), e = __ldg(a.rho0 + ic(a, k - 1, j, ie));
            so = __ldg(a.rho0 + ic(a, k - 1, js, i)), n = __ldg(a.rho0 + ic(a, k - 1, jn, i));
        }
        f.w = (0.5f * (w + c)) * (u0 * gu0), f.e = (0.5f * (c + e)) * (u1 * gu1);
        f.s = (0.5f * (so + c)) * (v0 * gv0), f.n = (0.5f * (c + n)) * (v1 * gv1);
        return f;
    };
    // rrw at level k from the fluxes of levels k (h) and k-1 (l); 0 at levels 1 and nk+1
    auto vertical = [&](int k, const Flux &h, const Flux &l) {
        if (k <= 1 || k >= nk + 1) return 0.0f;
        if (VM == 2) return __ldg(a.rf0 + ic(a, k - 1, 0, 0)) * LW(k, y, x);
        const float zt = VM == 1 ? a.ztop : (float)nk * a.dz, rzt = 1.0f / zt, rdz0 = 1.0f / a.dz;
        const float sigmaf = VM == 1 ? __ldg(a.sigmaf + k) : (float)(k - 1) * a.dz;
        const float sigma = VM == 1 ? __ldg(a.sigma + k - 1) : ((float)k - 1.5f) * a.dz;
        float r2 = (sigmaf - sigma) * (VM == 1 ? __ldg(a.rds + k) : rdz0);
        const float r1 = 0.5f * (1.0f - r2);
        r2 = 0.5f * r2;
        const float ux = r2 * (h.w + h.e) + r1 * (l.w + l.e);
        const float vy = r2 * (h.s + h.n) + r1 * (l.s + l.n);
        float terrain = ux * dzdx + vy * dzdy;
        terrain = terrain * (sigmaf - zt);
        terrain = terrain * gz;
        terrain = terrain * rzt;
        return __ldg(a.rf0 + ic(a, k - 1, j, i)) * LW(k, y, x) + terrain;
    };
    const int k_lo = 1 + blockIdx.y * chunk, k_hi = min(nk, k_lo + chunk - 1);
    Flux cur = flux(k_lo);
    float lo = k_lo == 1 ? 0.0f : vertical(k_lo, cur, VM == 2 ? cur : flux(k_lo - 1));
#pragma unroll 1
    for (int k = k_lo; k <= k_hi; ++k) {
        const Flux next = k < nk ? flux(k + 1) : cur;
        const float hi = vertical(k + 1, next, cur);
        float value = (cur.e - cur.w) * a.rdx + (cur.n - cur.s) * a.rdy;
        if (VM == 2) {  // the flat column's ((d*rdz)*mh(k)) with cm1.F's smeps 1e-30
            value = value + ((hi - lo) * a.rdzm) * __ldg(a.mh + k);
            if (fabsf(value) < 1.0e-30f) value = 0.0f;
        } else {
            value = value + (hi - lo) * (VM == 1 ? __ldg(a.rdsf + k) : a.rdz);
            if (fabsf(value) < 1.0e-20f) value = 0.0f;
        }
        RU(k, y, x) = cur.w;
        if (i == ni - 1) RU(k, y, x + 1) = cur.e;
        RV(k, y, x) = cur.s;
        if (j == nj - 1) RV(k, y + 1, x) = cur.n;
        RW(k, y, x) = lo;
        if (k == nk) RW(k + 1, y, x) = hi;
        a.divx[ic(a, k - 1, j, i)] = value;
        cur = next, lo = hi;
    }
}

// ---------------------------------------------------------------------------
// (2) advu / advv / advw.  A warp owns 32 x faces of one row of one component
// and marches up a chunk of levels: each lane forms the x flux of one face
// and takes the next face's from the lane above (31 points per 32 lanes, no
// divergent edge), the upper vertical flux is carried down as the next
// level's lower one and the column's six levels stay in registers; only the
// two y fluxes of a point are formed apart.  The three components of a tile
// are neighbouring CTAs (blockIdx.x % 3), so their shared mass fluxes meet in
// L2.  Bound by instruction issue (the upwind selects on the half-rate ALU).
// Measured on one B200, per launch at 640x768x80: 3.085 ms with a thread per
// point forming all its fluxes, 1.596 with one finish for every line, 1.127
// here (32 warps an SM, the terrain instantiation spilling 16 bytes; 24 warps
// 1.169, 40 warps 1.267, two levels a trip 1.353).
// ---------------------------------------------------------------------------
constexpr int kMomOut = 31;   // points a warp of 32 faces completes
constexpr int kMomRows = 4;   // rows (independent warps) per CTA

// vertical flux of u or v at Fortran face kf from levels kf-3 .. kf+2 (win)
__device__ __forceinline__ float uv_z(const float win[6], float m, float c2, int kf, int nk) {
#define Q(l) win[(l) - kf + 3]
    float r;
    if (kf == 2)
        r = m >= 0.0f ? (1.0f - c2) * Q(1) + c2 * Q(2) : flx3(Q(3), Q(2), Q(1));
    else if (kf == nk)
        r = m >= 0.0f ? flx3(Q(kf - 2), Q(kf - 1), Q(kf)) : (1.0f - c2) * Q(kf - 1) + c2 * Q(kf);
    else if (kf == 3)
        r = m >= 0.0f ? flx3(Q(1), Q(2), Q(3)) : flx5(Q(5), Q(4), Q(3), Q(2), Q(1));
    else if (kf == nk - 1)
        r = m >= 0.0f ? flx5(Q(kf - 3), Q(kf - 2), Q(kf - 1), Q(kf), Q(kf + 1)) : flx3(Q(kf + 1), Q(kf), Q(kf - 1));
    else
        return up5(m, Q(kf - 3), Q(kf - 2), Q(kf - 1), Q(kf), Q(kf + 1), Q(kf + 2));
#undef Q
    return m * r;
}

// vertical flux of w at mass level k from levels k-2 .. k+3 (win)
__device__ __forceinline__ float w_z(const float win[6], float m, int k, int nk) {
#define Q(l) win[(l) - k + 2]
    float r;
    if (k == 1)
        r = m >= 0.0f ? 0.5f * (Q(1) + Q(2)) : flx3(Q(3), Q(2), Q(1));
    else if (k == 2)
        r = m >= 0.0f ? flx3(Q(1), Q(2), Q(3)) : flx5(Q(5), Q(4), Q(3), Q(2), Q(1));
    else if (k == nk - 1)
        r = m >= 0.0f ? flx5(Q(k - 2), Q(k - 1), Q(k), Q(k + 1), Q(k + 2)) : flx3(Q(k + 2), Q(k + 1), Q(k));
    else if (k == nk)
        r = m >= 0.0f ? flx3(Q(k - 1), Q(k), Q(k + 1)) : 0.5f * (Q(k) + Q(k + 1));
    else
        return up5(m, Q(k - 2), Q(k - 1), Q(k), Q(k + 1), Q(k + 2), Q(k + 3));
#undef Q
    return m * r;
}

// six points of a row (the two upwind stencils of a face) around p[0], and
// the seven of a column of row stride sy (both faces of a point); the centre
// is the column window's
__device__ __forceinline__ void row6(const float *p, float c, float q[6]) {
#pragma unroll
    for (int e = 0; e < 6; ++e) q[e] = e == 3 ? c : __ldg(p + (e - 3));
}
__device__ __forceinline__ void col7(const float *p, int sy, float c, float q[7]) {
#pragma unroll
    for (int e = 0; e < 7; ++e) q[e] = e == 3 ? c : __ldg(p + (e - 3) * sy);
}
__device__ __forceinline__ float below(float v) { return __shfl_down_sync(0xffffffffu, v, 1); }  // the next face's
__device__ __forceinline__ void shift(float win[6], float next) {
#pragma unroll
    for (int q = 0; q < 5; ++q) win[q] = win[q + 1];
    win[5] = next;
}

// advu at the faces f of row j
template <bool FLAT>
__device__ __forceinline__ void march_u(const MomArgs &a, int tile, int j, int k_lo, int k_hi) {
    const int ni = a.ni, nj = a.nj, nk = a.nk, lane = threadIdx.x;
    if (j >= nj) return;
    const int ff = a.per[0] ? 0 : 1, lf = a.per[1] ? ni : ni - 1;
    if (ff + tile * kMomOut > lf) return;
    const int f = min(ff + tile * kMomOut + lane, lf + 1);  // the flux u_fx(f - 1)
    const bool own = lane < kMomOut && ff + tile * kMomOut + lane <= lf;
    const int ux = ni + 1 + 2 * G, sx = ni + 2 * G, uz = (nj + 2 * G) * ux, vz = (nj + 1 + 2 * G) * sx,
              wz = (nj + 2 * G) * sx, cz = ni * nj;
    const int y = j + G, o = y * ux + f + G;
    const int ra = y * ux + fxw(a, f - 1) + G, rb = y * ux + fxw(a, f) + G;
    const int e = cxw(a, f), w = cxw(a, f - 1);
    const int se = y * sx + e + G, sw = y * sx + w + G;          // rrv / rrw columns east and west of the face
    const int ce = j * ni + clampn(e, ni), cw = j * ni + clampn(w, ni);  // divx and rho0
    const int c2e = j * ni + clampn(f, ni), c2w = j * ni + clampn(f - 1, ni);
    const bool so = j == 0 && a.opn[2], no = j == nj - 1 && a.opn[3], edge = so || no;
    const float gzu = FLAT ? 0.0f : __ldg(a.gzu + j * (ni + 1) + min(f, ni)), vh = __ldg(a.vh + y);
    float win[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        const int l = k_lo - 3 + q;
        win[q] = l >= 0 && l <= nk + 1 ? __ldg(a.u3d + l * uz + o) : 0.0f;
    }
    auto c2f = [&](int kf) {
        return kf == 2 || kf == nk ? 0.5f * (__ldg(a.c2 + (kf - 1) * cz + c2w) + __ldg(a.c2 + (kf - 1) * cz + c2e)) : 0.0f;
    };
    float zlo = 0.0f;
    if (k_lo >= 2)
        zlo = uv_z(win, 0.5f * (__ldg(a.rrw + k_lo * wz + se) + __ldg(a.rrw + k_lo * wz + sw)), c2f(k_lo), k_lo, nk);
#pragma unroll 1
    for (int k = k_lo; k <= k_hi; ++k) {
        const float *pt = a.u3d + k * uz + o;
        const float uc = win[3];
        float px[6], py[7];
        row6(pt, uc, px);
        col7(pt, ux, uc, py);
        const float next = k + 3 <= nk + 1 ? __ldg(pt + 3 * uz) : 0.0f;
        const float ma = __ldg(a.rru + k * uz + ra), mb = __ldg(a.rru + k * uz + rb);
        const float *rv = a.rrv + k * vz;
        const float vse = __ldg(rv + se), vsw = __ldg(rv + sw), vne = __ldg(rv + se + sx), vnw = __ldg(rv + sw + sx);
        // (level nk+1's is not used)
        const float mz = 0.5f * (__ldg(a.rrw + (k + 1) * wz + se) + __ldg(a.rrw + (k + 1) * wz + sw));
        const float de = __ldg(a.divx + (k - 1) * cz + ce), dw = __ldg(a.divx + (k - 1) * cz + cw);
        float *out = a.uten + k * uz + o;
        const float ten = own ? *out : 0.0f;
        const float scale = FLAT ? __ldg(a.rr0 + (k - 1) * cz)
                                         : gzu / (0.5f * (__ldg(a.rho0 + (k - 1) * cz + cw) + __ldg(a.rho0 + (k - 1) * cz + ce)));
        const float fw = up5(0.5f * (ma + mb), px[0], px[1], px[2], px[3], px[4], px[5]);
        const float fe = below(fw);
        const float ms = vse + vsw, mn = vne + vnw;
        const float fs0 = up5(0.5f * ms, py[0], py[1], py[2], py[3], py[4], py[5]);
        const float fn0 = up5(0.5f * mn, py[1], py[2], py[3], py[4], py[5], py[6]);
        shift(win, next);
        const float advx = -(fe - fw) * a.rdx;
        float advy, advz, zhi;
        if (!edge && k >= 3 && k < nk - 2) {
            zhi = up5(mz, win[0], win[1], win[2], win[3], win[4], win[5]);
            advy = -(fn0 - fs0) * a.rdy;
            advz = zmass<FLAT>(a, -(zhi - zlo), k);
        } else {
            // inflow through an open side's face takes the inner neighbour's flux
            const bool sub_s = so && ms >= 0.0f, sub_n = no && mn <= 0.0f;
            zhi = k < nk ? uv_z(win, mz, c2f(k + 1), k + 1, nk) : 0.0f;
            advy = -((sub_n ? fs0 : fn0) - (sub_s ? fn0 : fs0)) * a.rdy;
            if (sub_s || sub_n) {
                const float corr = (vnw - vsw) + (vne - vse);
                advy = advy - bcorr<FLAT>(uc * 0.5f, corr, a.rdy, vh);
            }
            advz = zmass<FLAT>(a, k == 1 ? -zhi : k == nk ? zlo : -(zhi - zlo), k);
        }
        float total = (advx + advy) + advz;
        total = total + uc * (0.5f * (de + dw));
        if (own) *out = ten + total * scale;
        zlo = zhi;
    }
}

// advv at the faces g of rows, columns i
template <bool FLAT>
__device__ __forceinline__ void march_v(const MomArgs &a, int tile, int g, int k_lo, int k_hi) {
    const int ni = a.ni, nj = a.nj, nk = a.nk, lane = threadIdx.x;
    const int fr = a.per[2] ? 0 : 1, lr = a.per[3] ? nj : nj - 1;
    if (g < fr || g > lr || tile * kMomOut >= ni) return;
    const int i0 = tile * kMomOut + lane, i = min(i0, ni);  // the flux v_fx(i)
    const bool own = lane < kMomOut && i0 < ni;
    const int ux = ni + 1 + 2 * G, sx = ni + 2 * G, uz = (nj + 2 * G) * ux, vz = (nj + 1 + 2 * G) * sx,
              wz = (nj + 2 * G) * sx, cz = ni * nj;
    const int y = g + G, x = i + G, o = y * sx + x;
    const int north = cyw(a, g), south = cyw(a, g - 1);
    const int un = (north + G) * ux + x, us = (south + G) * ux + x;
    const int rs = (fyw(a, g - 1) + G) * sx + x, rc = (fyw(a, g) + G) * sx + x, rn = (fyw(a, g + 1) + G) * sx + x;
    const int sn = (north + G) * sx + x, ss = (south + G) * sx + x;  // rrw
    const int ic0 = min(i, ni - 1);
    const int cn = clampn(north, nj) * ni + ic0, cs = clampn(south, nj) * ni + ic0;
    const int c2n = clampn(g, nj) * ni + ic0, c2s = clampn(g - 1, nj) * ni + ic0;
    const bool wo = i == 0 && a.opn[0], eo = i == ni - 1 && a.opn[1], edge = __any_sync(0xffffffffu, wo || eo);
    const float gzv = FLAT ? 0.0f : __ldg(a.gzv + g * ni + ic0), uh = __ldg(a.uh + x);
    float win[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        const int l = k_lo - 3 + q;
        win[q] = l >= 0 && l <= nk + 1 ? __ldg(a.v3d + l * vz + o) : 0.0f;
    }
    auto c2f = [&](int kf) {
        return kf == 2 || kf == nk ? 0.5f * (__ldg(a.c2 + (kf - 1) * cz + c2s) + __ldg(a.c2 + (kf - 1) * cz + c2n)) : 0.0f;
    };
    float zlo = 0.0f;
    if (k_lo >= 2)
        zlo = uv_z(win, 0.5f * (__ldg(a.rrw + k_lo * wz + sn) + __ldg(a.rrw + k_lo * wz + ss)), c2f(k_lo), k_lo, nk);
#pragma unroll 1
    for (int k = k_lo; k <= k_hi; ++k) {
        const float *pt = a.v3d + k * vz + o;
        const float vc = win[3];
        float px[6], py[7];
        row6(pt, vc, px);
        col7(pt, sx, vc, py);
        const float next = k + 3 <= nk + 1 ? __ldg(pt + 3 * vz) : 0.0f;
        const float uN = __ldg(a.rru + k * uz + un), uS = __ldg(a.rru + k * uz + us);
        const float *rv = a.rrv + k * vz;
        const float ma = __ldg(rv + rs), mb = __ldg(rv + rc), mc = __ldg(rv + rn);
        const float mz = 0.5f * (__ldg(a.rrw + (k + 1) * wz + sn) + __ldg(a.rrw + (k + 1) * wz + ss));
        const float dn = __ldg(a.divx + (k - 1) * cz + cn), ds = __ldg(a.divx + (k - 1) * cz + cs);
        float *out = a.vten + k * vz + o;
        const float ten = own ? *out : 0.0f;
        const float scale = FLAT ? __ldg(a.rr0 + (k - 1) * cz)
                                         : gzv / (0.5f * (__ldg(a.rho0 + (k - 1) * cz + cs) + __ldg(a.rho0 + (k - 1) * cz + cn)));
        const float mw = uN + uS;
        const float fw0 = up5(0.5f * mw, px[0], px[1], px[2], px[3], px[4], px[5]);
        const float fe0 = below(fw0);
        const float fs = up5(0.5f * (ma + mb), py[0], py[1], py[2], py[3], py[4], py[5]);
        const float fn = up5(0.5f * (mb + mc), py[1], py[2], py[3], py[4], py[5], py[6]);
        shift(win, next);
        const float advy = -(fn - fs) * a.rdy;
        float advx, advz, zhi;
        if (!edge && k >= 3 && k < nk - 2) {
            zhi = up5(mz, win[0], win[1], win[2], win[3], win[4], win[5]);
            advx = -(fe0 - fw0) * a.rdx;
            advz = zmass<FLAT>(a, -(zhi - zlo), k);
        } else {
            const float me = below(mw), uNe = below(uN), uSe = below(uS);
            const bool sub_w = wo && mw >= 0.0f, sub_e = eo && me <= 0.0f;
            zhi = k < nk ? uv_z(win, mz, c2f(k + 1), k + 1, nk) : 0.0f;
            advx = -((sub_e ? fw0 : fe0) - (sub_w ? fe0 : fw0)) * a.rdx;
            if (sub_w || sub_e) {
                const float corr = (uSe - uS) + (uNe - uN);
                advx = advx - bcorr<FLAT>(vc * 0.5f, corr, a.rdx, uh);
            }
            advz = zmass<FLAT>(a, k == 1 ? -zhi : k == nk ? zlo : -(zhi - zlo), k);
        }
        float total = (advx + advy) + advz;
        total = total + vc * (0.5f * (dn + ds));
        if (own) *out = ten + total * scale;
        zlo = zhi;
    }
}

// advw at the w levels kf = k + 1 (2..nk) of row j, columns i
template <bool FLAT>
__device__ __forceinline__ void march_w(const MomArgs &a, int tile, int j, int k_lo, int k_hi) {
    const int ni = a.ni, nj = a.nj, nk = a.nk, lane = threadIdx.x;
    if (j >= nj || tile * kMomOut >= ni || k_lo >= nk) return;
    const int i0 = tile * kMomOut + lane, i = min(i0, ni);  // the flux w_fx(i)
    const bool own = lane < kMomOut && i0 < ni;
    const int ux = ni + 1 + 2 * G, sx = ni + 2 * G, uz = (nj + 2 * G) * ux, vz = (nj + 1 + 2 * G) * sx,
              wz = (nj + 2 * G) * sx, cz = ni * nj;
    const int y = j + G, x = i + G, o = y * sx + x, ou = y * ux + x;
    const int ic0 = min(i, ni - 1), cc = j * ni + ic0;
    const int cw = j * ni + clampn(i - 1, ni), ce = j * ni + clampn(i, ni);
    const int cs = clampn(j - 1, nj) * ni + ic0, cn = clampn(j + 1, nj) * ni + ic0;
    const bool wo = i == 0 && a.opn[0], eo = i == ni - 1 && a.opn[1];
    const bool so = j == 0 && a.opn[2], no = j == nj - 1 && a.opn[3];
    const bool edge = __any_sync(0xffffffffu, wo || eo) || so || no;
    const float uh = __ldg(a.uh + min(x, ni + 2 * G - 1)), vh = __ldg(a.vh + y);
    const float gz = FLAT ? 0.0f : __ldg(a.gz + cc);
    float win[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        const int l = k_lo - 2 + q;
        win[q] = l >= 0 && l <= nk + 2 ? __ldg(a.w3d + l * wz + o) : 0.0f;
    }
    float rw = __ldg(a.rrw + (k_lo + 1) * wz + o);  // rrw(kf)
    float zlo = w_z(win, 0.5f * (__ldg(a.rrw + k_lo * wz + o) + rw), k_lo, nk);
    float rul = __ldg(a.rru + k_lo * uz + ou), rsl = __ldg(a.rrv + k_lo * vz + o), rnl = __ldg(a.rrv + k_lo * vz + o + sx);
    float dl = __ldg(a.divx + (k_lo - 1) * cz + cc);
#pragma unroll 1
    for (int k = k_lo; k <= k_hi && k < nk; ++k) {
        const int kf = k + 1;
        const float *pt = a.w3d + kf * wz + o;
        const float wc = win[3];  // the window still ends at kf + 2
        float px[6], py[7];
        row6(pt, wc, px);
        col7(pt, sx, wc, py);
        const float next = kf + 3 <= nk + 2 ? __ldg(pt + 3 * wz) : 0.0f;
        const float *c2p = a.c2 + (kf - 1) * cz;
        const float kw = __ldg(c2p + cw), ke = __ldg(c2p + ce), ks = __ldg(c2p + cs), kn = __ldg(c2p + cn), c2 = __ldg(c2p + cc);
        const float ru = __ldg(a.rru + kf * uz + ou), rs = __ldg(a.rrv + kf * vz + o), rn = __ldg(a.rrv + kf * vz + o + sx);
        const float rwn = __ldg(a.rrw + (kf + 1) * wz + o), dh = __ldg(a.divx + (kf - 1) * cz + cc);
        float *out = a.wten + kf * wz + o;
        const float ten = own ? *out : 0.0f;
        const float scale = FLAT ? __ldg(a.rrf0 + (kf - 1) * cz) : __ldg(a.rrf0 + (kf - 1) * cz + cc) * gz;
        const float c1 = 1.0f - c2;
        const float c2x = 0.5f * (kw + ke), c2s = 0.5f * (ks + c2), c2n = 0.5f * (c2 + kn);
        const float mw = c2x * ru + (1.0f - c2x) * rul;
        const float ms = c2s * rs + (1.0f - c2s) * rsl, mn = c2n * rn + (1.0f - c2n) * rnl;
        const float fw0 = up5(mw, px[0], px[1], px[2], px[3], px[4], px[5]);
        const float fe0 = below(fw0);
        const float fs0 = up5(ms, py[0], py[1], py[2], py[3], py[4], py[5]);
        const float fn0 = up5(mn, py[1], py[2], py[3], py[4], py[5], py[6]);
        shift(win, next);
        const float mz = 0.5f * (rw + rwn);
        float advx, advy, zhi;
        if (!edge && kf > 2 && kf < nk - 1) {
            zhi = up5(mz, win[0], win[1], win[2], win[3], win[4], win[5]);
            const float dfx = -(fe0 - fw0), dfy = -(fn0 - fs0);
            advx = FLAT ? (dfx * a.rdx) * uh : dfx * (a.rdx * uh);
            advy = FLAT ? (dfy * a.rdy) * vh : dfy * (a.rdy * vh);
        } else {
            const float me = below(mw), rue = below(ru), rule = below(rul);
            const float fw = wo && mw >= 0.0f ? fe0 : fw0, fe = eo && me <= 0.0f ? fw0 : fe0;
            const float fs = so && ms >= 0.0f ? fn0 : fs0, fn = no && mn <= 0.0f ? fs0 : fn0;
            zhi = w_z(win, mz, kf, nk);
            const float dfx = -(fe - fw), dfy = -(fn - fs);
            advx = FLAT ? (dfx * a.rdx) * uh : dfx * (a.rdx * uh);
            advy = FLAT ? (dfy * a.rdy) * vh : dfy * (a.rdy * vh);
            // the open sides' corrections weigh with the cell's own c2
            if ((wo && c2 * ru + c1 * rul >= 0.0f) || (eo && c2 * rue + c1 * rule <= 0.0f)) {
                const float corr = c1 * (rule - rul) + c2 * (rue - ru);
                advx = advx - bcorr<FLAT>(wc, corr, a.rdx, uh);
            }
            if ((so && c2 * rs + c1 * rsl >= 0.0f) || (no && c2 * rn + c1 * rnl <= 0.0f)) {
                const float corr = c1 * (rnl - rsl) + c2 * (rn - rs);
                advy = advy - bcorr<FLAT>(wc, corr, a.rdy, vh);
            }
        }
        const float advz = zface<FLAT>(a, -(zhi - zlo), kf);
        float total = (advx + advy) + advz;
        total = total + wc * (c2 * dh + c1 * dl);
        if (own) *out = ten + total * scale;
        zlo = zhi, rw = rwn, rul = ru, rsl = rs, rnl = rn, dl = dh;
    }
}

// (lines of points away from open sides, at levels away from the column's
// ends, take a finish without those branches)
template <bool FLAT>
__global__ void __launch_bounds__(32 * kMomRows, 8) mom5_adv_kernel(const __grid_constant__ MomArgs a,
                                                                     int levels_per_chunk) {
    // all tiles in one grid dimension, which takes any plane
    const int tiles = a.ni / kMomOut + 1, bt = blockIdx.x / 3;
    const int tile = bt % tiles, row = bt / tiles * kMomRows + threadIdx.y;
    const int k_lo = 1 + blockIdx.y * levels_per_chunk, k_hi = min(a.nk, k_lo + levels_per_chunk - 1);
    const int component = blockIdx.x % 3;
    if (component == 0)
        march_u<FLAT>(a, tile, row, k_lo, k_hi);
    else if (component == 1)
        march_v<FLAT>(a, tile, row, k_lo, k_hi);
    else
        march_w<FLAT>(a, tile, row, k_lo, k_hi);
}

bool launch_ok(const char *what) {
    cudaError_t e = cudaPeekAtLastError();
    if (e != cudaSuccess) {
        cudaGetLastError();
        gm1b_set_error("%s: %s", what, cudaGetErrorString(e));
        return false;
    }
    return true;
}

}  // namespace
}  // namespace gm1b

using namespace gm1b;

namespace {

int mom_args(int ni, int nj, int nk, const gm1b_momentum5_arrays *s, uint32_t lateral_obc, float dx, float dy,
             float dz, MomArgs &a, const char *what) {
    a.vmode = 0;
    a.rho0p = a.sigma = a.sigmaf = a.rds = a.rdsf = a.mh = a.mf = a.rr0 = nullptr;
    a.ztop = a.rdzm = 0.0f;
    if (s == nullptr || ni < 7 || nj < 7 || nk < 8) {
        gm1b_set_error("%s: need arrays, ni >= 7, nj >= 7, nk >= 8", what);
        return GM1B_ERR_ARGUMENT;
    }
    if ((size_t)(nk + 3) * (size_t)(nj + 7) * (size_t)(ni + 7) >= ((size_t)1 << 31)) {
        gm1b_set_error("%s: a %dx%dx%d grid's padded arrays reach 2^31 words; the kernels index with 32-bit offsets",
                       what, ni, nj, nk);
        return GM1B_ERR_ARGUMENT;
    }
    if (!(dx > 0.0f) || !(dy > 0.0f) || !(dz > 0.0f) || !isfinite(dx) || !isfinite(dy) || !isfinite(dz)) {
        gm1b_set_error("%s: dx, dy, dz must be finite and > 0", what);
        return GM1B_ERR_ARGUMENT;
    }
    int side[4];
    for (int q = 0; q < 4; ++q) {
        side[q] = (int)((lateral_obc >> (4 * q)) & 15u);
        if (side[q] < 1 || side[q] > 4) {
            gm1b_set_error("%s: lateral side codes must be 1..4 (wbc|ebc<<4|sbc<<8|nbc<<12)", what);
            return GM1B_ERR_ARGUMENT;
        }
    }
    if ((side[0] == 1) != (side[1] == 1) || (side[2] == 1) != (side[3] == 1)) {
        gm1b_set_error("%s: a direction cannot be periodic on one side only", what);
        return GM1B_ERR_ARGUMENT;
    }
    const void *need[] = {s->u3d, s->uten, s->rru, s->v3d, s->vten, s->rrv, s->w3d, s->wten, s->rrw, s->uh, s->vh,
                          s->rho0_3d, s->rf0, s->rrf0, s->c2, s->gz, s->gzu, s->gzv, s->rgzu, s->rgzv, s->dzdx,
                          s->dzdy, s->divx};
    for (const void *q : need)
        if (q == nullptr) {
            gm1b_set_error("%s: a required array is NULL", what);
            return GM1B_ERR_ARGUMENT;
        }
    a.u3d = s->u3d;
    a.v3d = s->v3d;
    a.w3d = s->w3d;
    a.uh = s->uh;
    a.vh = s->vh;
    a.rho0 = s->rho0_3d;
    a.rf0 = s->rf0;
    a.rrf0 = s->rrf0;
    a.c2 = s->c2;
    a.gz = s->gz;
    a.gzu = s->gzu;
    a.gzv = s->gzv;
    a.rgzu = s->rgzu;
    a.rgzv = s->rgzv;
    a.dzdx = s->dzdx;
    a.dzdy = s->dzdy;
    a.uten = s->uten;
    a.vten = s->vten;
    a.wten = s->wten;
    a.rru = s->rru;
    a.rrv = s->rrv;
    a.rrw = s->rrw;
    a.divx = s->divx;
    a.ni = ni;
    a.nj = nj;
    a.nk = nk;
    for (int q = 0; q < 4; ++q) {
        a.per[q] = side[q] == 1;
        a.opn[q] = side[q] == 2;
    }
    a.rdx = 1.0f / dx;
    a.rdy = 1.0f / dy;
    a.rdz = 1.0f / dz;
    a.dz = dz;
    return GM1B_OK;
}

int enqueue_mass(const MomArgs &a, cudaStream_t st) {
    const unsigned tiles = (unsigned)((a.ni + 31) / 32) * (unsigned)((a.nj + kFluxRows - 1) / kFluxRows);
    const int chunk = level_chunk(tiles, a.nk);
    const dim3 grid(tiles, (a.nk + chunk - 1) / chunk), block(32, kFluxRows);
    ProfScope ps("mom5_flux_kernel", st);
    if (a.vmode == 2)
        mom5_flux_kernel<2><<<grid, block, 0, st>>>(a, chunk);
    else if (a.vmode == 1)
        mom5_flux_kernel<1><<<grid, block, 0, st>>>(a, chunk);
    else
        mom5_flux_kernel<0><<<grid, block, 0, st>>>(a, chunk);
    ps.stop();
    return launch_ok("mom5_flux_kernel") ? GM1B_OK : GM1B_ERR_CUDA;
}

int enqueue_transport(const MomArgs &a, cudaStream_t st) {
    const int tiles = a.ni / kMomOut + 1, ytiles = (a.nj + 1 + kMomRows - 1) / kMomRows;
    // long chunks re-load and re-form less (each starts with six window loads
    // and its lower flux), short ones give a small plane warps enough: halve
    // until two rounds of 24 warps on each of 148 SMs, or at most four levels,
    // are left
    int chunk = a.nk;
    while (chunk > 4 && 3LL * tiles * (a.nj + 1) * ((a.nk + chunk - 1) / chunk) < 2LL * 148 * 24) chunk = (chunk + 1) / 2;
    ProfScope ps("mom5_adv_kernel", st);
    const dim3 grid(3 * tiles * ytiles, (a.nk + chunk - 1) / chunk), block(32, kMomRows);
    if (a.vmode == 2)
        mom5_adv_kernel<true><<<grid, block, 0, st>>>(a, chunk);
    else
        mom5_adv_kernel<false><<<grid, block, 0, st>>>(a, chunk);
    ps.stop();
    return launch_ok("mom5_adv_kernel") ? GM1B_OK : GM1B_ERR_CUDA;
}

}  // namespace

extern "C" int32_t gm1b_momentum_mass_flux5(int32_t ni, int32_t nj, int32_t nk, const gm1b_momentum5_arrays *s,
                                            uint32_t lateral_obc, float dx, float dy, float dz, void *stream) {
    MomArgs a;
    const int r = mom_args(ni, nj, nk, s, lateral_obc, dx, dy, dz, a, "gm1b_momentum_mass_flux5");
    return r != GM1B_OK ? r : enqueue_mass(a, static_cast<cudaStream_t>(stream));
}

extern "C" int32_t gm1b_momentum_transport5(int32_t ni, int32_t nj, int32_t nk, const gm1b_momentum5_arrays *s,
                                            uint32_t lateral_obc, float dx, float dy, float dz, void *stream) {
    MomArgs a;
    const int r = mom_args(ni, nj, nk, s, lateral_obc, dx, dy, dz, a, "gm1b_momentum_transport5");
    return r != GM1B_OK ? r : enqueue_transport(a, static_cast<cudaStream_t>(stream));
}

extern "C" int32_t gm1b_momentum_advection5(int32_t ni, int32_t nj, int32_t nk, const gm1b_momentum5_arrays *s,
                                            uint32_t lateral_obc, float dx, float dy, float dz, void *stream) {
    MomArgs a;
    const int r = mom_args(ni, nj, nk, s, lateral_obc, dx, dy, dz, a, "gm1b_momentum_advection5");
    if (r != GM1B_OK) return r;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int m = enqueue_mass(a, st);
    return m != GM1B_OK ? m : enqueue_transport(a, st);
}

// ---------------------------------------------------------------------------
// the same operator on a stretched column (launch_cuda_gm1_child_stretched_momentum5,
// src/cm1core/cuda_gm1_child_stretched_momentum.py:540-780): terrain branch
// (rdsf / rds / sigma / sigmaf and the physical top) or flat column
// (rdz*mh / rdz*mf and the column's base state)
// ---------------------------------------------------------------------------
namespace {
int column_args(int ni, int nj, int nk, const gm1b_momentum5_arrays *s, uint32_t lateral_obc, float dx, float dy,
                const gm1b_momentum_column *c, MomArgs &a, const char *what) {
    if (c == nullptr || (c->flat != 0 && c->flat != 1) || c->rho0_padded == nullptr) {
        gm1b_set_error("%s: need a column with flat = 0 or 1 and the padded base density", what);
        return GM1B_ERR_ARGUMENT;
    }
    if (c->flat ? (c->mh == nullptr || c->mf == nullptr || c->rr0 == nullptr || !(c->rdz > 0.0f) ||
                   !isfinite(c->rdz))
                : (c->sigma == nullptr || c->sigmaf == nullptr || c->rds == nullptr || c->rdsf == nullptr ||
                   !(c->ztop > 0.0f) || !isfinite(c->ztop))) {
        gm1b_set_error("%s: a flat column needs mh, mf, rr0 and rdz > 0; a terrain column sigma, sigmaf, rds, rdsf "
                       "and ztop > 0", what);
        return GM1B_ERR_ARGUMENT;
    }
    // dz forms only the uniform reciprocals, which a stretched column never reads
    const int r = mom_args(ni, nj, nk, s, lateral_obc, dx, dy, 1.0f, a, what);
    if (r != GM1B_OK) return r;
    a.vmode = c->flat ? 2 : 1;
    a.rho0p = c->rho0_padded, a.sigma = c->sigma, a.sigmaf = c->sigmaf, a.rds = c->rds, a.rdsf = c->rdsf;
    a.mh = c->mh, a.mf = c->mf, a.rr0 = c->rr0, a.ztop = c->ztop, a.rdzm = c->rdz;
    return GM1B_OK;
}
}  // namespace

extern "C" int32_t gm1b_momentum_mass_flux5_column(int32_t ni, int32_t nj, int32_t nk, const gm1b_momentum5_arrays *s,
                                                   uint32_t lateral_obc, float dx, float dy,
                                                   const gm1b_momentum_column *column, void *stream) {
    MomArgs a;
    const int r = column_args(ni, nj, nk, s, lateral_obc, dx, dy, column, a, "gm1b_momentum_mass_flux5_column");
    return r != GM1B_OK ? r : enqueue_mass(a, static_cast<cudaStream_t>(stream));
}

extern "C" int32_t gm1b_momentum_transport5_column(int32_t ni, int32_t nj, int32_t nk, const gm1b_momentum5_arrays *s,
                                                   uint32_t lateral_obc, float dx, float dy,
                                                   const gm1b_momentum_column *column, void *stream) {
    MomArgs a;
    const int r = column_args(ni, nj, nk, s, lateral_obc, dx, dy, column, a, "gm1b_momentum_transport5_column");
    return r != GM1B_OK ? r : enqueue_transport(a, static_cast<cudaStream_t>(stream));
}

extern "C" int32_t gm1b_momentum_advection5_column(int32_t ni, int32_t nj, int32_t nk, const gm1b_momentum5_arrays *s,
                                                   uint32_t lateral_obc, float dx, float dy,
                                                   const gm1b_momentum_column *column, void *stream) {
    MomArgs a;
    const int r = column_args(ni, nj, nk, s, lateral_obc, dx, dy, column, a, "gm1b_momentum_advection5_column");
    if (r != GM1B_OK) return r;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int m = enqueue_mass(a, st);
    return m != GM1B_OK ? m : enqueue_transport(a, st);
}
