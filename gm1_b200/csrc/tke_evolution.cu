// tke_evolution.cu - sm_100a kernels of the TKE evolution on the terrain
// lane: turbt (horizontal TKE flux divergence with the terrain correction
// and the vertically implicit diffusion) and the flux-form RK stages.
//
// Behaviour followed (reference file:line):
//   cpu_tke_evolution_inplace   src/cm1core/cuda_tke_evolution.py:206-327
//   launch_cuda_tke_diffusion / _rk_stage / _commit / _evolution   :421-492
//   flat column: gm1_flat_turbt_v1 and gm1_flat_tke_advw_rk_v1
//               src/cm1core/cuda_gm1_flat_stretched_closure.py:314-359, :401-449
//               (enqueue_flat_turbt :631; CartesianClosure.tke_rk, cuda_cartesian_closure.py:1658-1663)
//
// Design (B200):
//  * turbt is one kernel per 32 columns of a row: eight warps (or three) form the
//    tridiagonal rows of their own runs of levels (the mf/rf divisions and
//    every load spread over the CTA), one warp sweeps them in shared memory
//    (the reference's thread-per-column kernel keeps five local arrays of 74
//    words, which spill), then all warps add the horizontal flux divergence
//    and the vertical diffusion of their levels to tketen, each face flux of
//    a column formed once and carried up.  No device scratch.
//  * an RK stage marches warps of 32 x faces up the face levels: each x and
//    vertical face flux (fifth order, WENO5 at nrk = 3) is formed once, from
//    the stage-start field.
//  * binary32 one operation at a time in the reference's order, binary64
//    WENO weights: word-identical to the reference twin.
#include "gm1b_common.cuh"
#include "weno.cuh"

namespace gm1b {
namespace {

constexpr int kTurbtWarps = 8;  // warps of a flat turbt CTA, which owns 32 columns of a row
constexpr int kTurbtMostNk = 201;
constexpr int kG = 3;                                    // padded-lane halo of rru/rrv/rrw

struct TkeArgs {
    const float *t, *kmh, *kmv, *rho, *rf, *mh, *mf, *gz, *rgz, *rgzu, *rgzv;
    const float *tkea, *c2, *rrf0, *rru, *rrv, *rrw, *divx;
    const float *mfp;  // flat column: the mf profile (nk+3, CM1-indexed)
    float *tketen;
    int ni, nj, nk;
    float rdx, rdy, rdz, dz, zt;  // flat column: rdz is the coordinate's reference 1/dz
};

__device__ __forceinline__ int clampi(int x, int n) { return x < 0 ? 0 : (x >= n ? n - 1 : x); }
// 32-bit element offsets (the entry points refuse grids whose padded arrays
// reach 2^31 words)
// x TKE flux at face level f (1..nk-1) between the cells l and r (offsets in a
// level), y likewise with rd = rdy
__device__ __forceinline__ float tke_flux(const TkeArgs &a, int f, int l, int r, float gl, float gr, float rgl, float rgr,
                                          float rd) {
    if (f <= 0 || f >= a.nk) return 0.0f;
    const unsigned cz = (unsigned)a.ni * a.nj, z = (unsigned)f * cz;
    const float *t = a.t + z, *tu = t + cz, *tl = t - cz;
    const float cl = t[l], cr = t[r];
    const float den = gr * a.rf[z + r] + gl * a.rf[z + l];
    const float kval = a.kmh[z + r] + a.kmh[z + l];
    float term = (cr * rgr - cl * rgl) * rd;
    const float up = (a.zt - ((float)f + 0.5f) * a.dz) * (0.5f * (cl + tu[l]) + 0.5f * (cr + tu[r]));
    const float lo = (a.zt - ((float)f - 0.5f) * a.dz) * (0.5f * (tl[l] + cl) + 0.5f * (tl[r] + cr));
    term = term + 0.5f * ((up - lo) * (a.rdz * ((rgr - rgl) * rd)));
    return -0.25f * (den * (2.0f * (kval * term)));
}

// dynamic shared memory: the four tridiagonal words of each of the nk-1 rows
// of 32 columns.  256x256x80: 405 us with a thread per column (its loads a
// level at a time, most of the chip idle), 220 here with eight warps.  Three
// warps where short columns of a large plane make enough CTAs of them: a run
// of levels forms the face fluxes of one level more at either end, and one
// warp sweeps while the others wait (turbt_warps).
template <int WARPS>
__global__ void __launch_bounds__(32 * WARPS, 24 / WARPS) tke_turbt_kernel(const __grid_constant__ TkeArgs a, float dt) {
    extern __shared__ float s_col[];
    const int lane = threadIdx.x, wy = threadIdx.y;
    const int ni = a.ni, nj = a.nj, nk = a.nk, n = nk - 1, cz = ni * nj, tiles = (ni + 31) / 32;
    const int i0 = blockIdx.x % tiles * 32 + lane, j = blockIdx.x / tiles;
    const bool own = i0 < ni;
    const int i = min(i0, ni - 1), c = j * ni + i;  // lanes past the row's end repeat its last column
    float *s_a = s_col + lane, *s_b = s_a + n * 32, *s_c = s_b + n * 32, *s_d = s_c + n * 32;  // rows f - 1
    const float rdt = 1.0f / dt, tema = -1.0f * (dt * (a.rdz * a.rdz));
    const int run = (n + WARPS - 1) / WARPS;
    const int f_lo = 1 + wy * run, f_hi = min(n, f_lo + run - 1);
    if (f_lo <= f_hi) {
        unsigned z = (unsigned)f_lo * (unsigned)cz + (unsigned)c;
        // level f-1's and f's words ride in registers
        float km = a.kmv[z - cz], k0 = a.kmv[z], mhm = a.mh[z - cz], rhom = a.rho[z - cz];
#pragma unroll 4
        for (int f = f_lo; f <= f_hi; ++f, z += cz) {
            const float kp = a.kmv[z + cz], mh = a.mh[z], rho = a.rho[z];
            const float rrf = a.mf[z] / a.rf[z];
            const float r1 = (km + k0) * (mhm * (rhom * rrf)), r2 = (k0 + kp) * (mh * (rho * rrf));
            const float cfa = tema * r1, cfc = tema * r2;
            const int q = (f - 1) * 32;
            s_a[q] = cfa, s_c[q] = cfc, s_d[q] = a.t[z];
            s_b[q] = f == 1 ? 1.0f - cfc : f == n ? 1.0f - cfa : (1.0f - cfa) - cfc;
            km = k0, k0 = kp, mhm = mh, rhom = rho;
        }
    }
    __syncthreads();
    if (wy == 0) column_sweep<4>(s_a, s_b, s_c, s_d, n);
    __syncthreads();
    if (f_lo > f_hi || !own) return;
    // horizontal divergence of the run's levels: the four face fluxes of the
    // levels f-1, f and f+1, each formed once and carried up
    const int w = j * ni + max(i - 1, 0), e = j * ni + min(i + 1, ni - 1), s = max(j - 1, 0) * ni + i,
              t = min(j + 1, nj - 1) * ni + i;
    const float g = a.gz[c], gw = a.gz[w], ge = a.gz[e], gs = a.gz[s], gt = a.gz[t];
    const float rg = a.rgz[c], rgw = a.rgz[w], rge = a.rgz[e], rgs = a.rgz[s], rgt = a.rgz[t];
    const float ru0 = a.rgzu[(unsigned)j * (ni + 1) + i], ru1 = a.rgzu[(unsigned)j * (ni + 1) + i + 1];
    const float rv0 = a.rgzv[(unsigned)j * ni + i], rv1 = a.rgzv[(unsigned)(j + 1) * ni + i];
    const bool ex = i == 0 || i == ni - 1, ey = j == 0 || j == nj - 1;
    auto fluxes = [&](int f, float q[4]) {
        q[0] = ex ? 0.0f : tke_flux(a, f, w, c, gw, g, rgw, rg, a.rdx);
        q[1] = ex ? 0.0f : tke_flux(a, f, c, e, g, ge, rg, rge, a.rdx);
        q[2] = ey ? 0.0f : tke_flux(a, f, s, c, gs, g, rgs, rg, a.rdy);
        q[3] = ey ? 0.0f : tke_flux(a, f, c, t, g, gt, rg, rgt, a.rdy);
    };
    float lo4[4], cur[4], up4[4];
    fluxes(f_lo - 1, lo4);
    fluxes(f_lo, cur);
#pragma unroll 1
    for (int f = f_lo; f <= f_hi; ++f) {
        fluxes(f + 1, up4);
        const unsigned z = (unsigned)f * (unsigned)cz + (unsigned)c;
        const float hi_z = a.zt - ((float)f + 0.5f) * a.dz, lo_z = a.zt - ((float)f - 0.5f) * a.dz;
        auto part = [&](int q, float m0, float m1, float rd) {
            const float x0 = cur[q], x1 = cur[q + 1];
            float x = -1.0f * ((x1 * m1 - x0 * m0) * (g * rd));
            const float f0 = 0.5f * (x0 + up4[q]), f1 = 0.5f * (x1 + up4[q + 1]);
            const float b0 = 0.5f * (lo4[q] + x0), b1 = 0.5f * (lo4[q + 1] + x1);
            const float up = hi_z * (f0 + f1), lo = lo_z * (b0 + b1);
            return x - 0.5f * ((up - lo) * (a.rdz * ((m1 - m0) * (g * rd))));
        };
        const float hx = ex ? 0.0f : part(0, ru0, ru1, a.rdx), hy = ey ? 0.0f : part(2, rv0, rv1, a.rdy);
        const float rfz = a.rf[z];
        const float vz = rfz * ((s_d[(f - 1) * 32] - a.t[z]) * rdt);
        a.tketen[z] = a.tketen[z] + ((hx + hy) + vz) / rfz;
#pragma unroll
        for (int q = 0; q < 4; ++q) lo4[q] = cur[q], cur[q] = up4[q];
    }
}

// ------------------------------------------------- turbt, flat column
// gm1_flat_turbt_v1 (src/cm1core/cuda_gm1_flat_stretched_closure.py:314-359;
// turbtend.F:729-1044 with terrain_flag=.false.): the x/y face fluxes
// -0.25*(rf(a)+rf(a-1))*2*(kmh(a)+kmh(a-1))*(t(a)-t(a-1))*rdx, no terrain
// correction, and the implicit diffusion with rdz and the 3-D mh/mf.  One
// CTA per 32 columns of a row: kTurbtWarps warps form the tridiagonal rows of
// their own runs of levels (the mf/rf divisions and every load spread over
// the CTA), one warp sweeps them in shared memory, then all warps add the
// horizontal and vertical parts of their levels.  Four shared words per level
// and column leave five CTAs on an SM at nk = 80.  640x768x80: 3.653 -> 0.603
// ms against a thread per column (two 128-thread CTAs an SM, its loads one
// level at a time).
// the flux through the face between the cells l and r (rd = rdx or rdy)
__device__ __forceinline__ float tke_flux_flat(float rfr, float rfl, float kr, float kl, float tr, float tl, float rd) {
    const float rs = rfr + rfl, ks = kr + kl, dt = tr - tl;
    return -(((((0.25f * rs) * 2.0f) * ks) * dt) * rd);
}

__global__ void __launch_bounds__(32 * kTurbtWarps, 5) tke_turbt_flat_kernel(TkeArgs a, float dt) {
    extern __shared__ float s_col[];
    const int lane = threadIdx.x, wy = threadIdx.y;
    const int ni = a.ni, nj = a.nj, nk = a.nk, n = nk - 1, cz = ni * nj;
    const int tiles = (ni + 31) / 32;
    const int i0 = blockIdx.x % tiles * 32 + lane, j = blockIdx.x / tiles;
    const bool own = i0 < ni;
    const int i = min(i0, ni - 1), c = j * ni + i;  // lanes past the row's end repeat its last column
    float *s_a = s_col + lane, *s_b = s_a + n * 32, *s_c = s_b + n * 32, *s_d = s_c + n * 32;  // rows f - 1
    const float rdt = 1.0f / dt;
    const float tema = (((-1.0f * dt) * 1.0f) * a.rdz) * a.rdz;
    const float temb = ((dt * 0.0f) * a.rdz) * a.rdz;
    const int run = (n + kTurbtWarps - 1) / kTurbtWarps;
    const int f_lo = 1 + wy * run, f_hi = min(n, f_lo + run - 1);
    if (f_lo <= f_hi) {
        unsigned z = (unsigned)f_lo * (unsigned)cz + (unsigned)c;
        // level f-1's and f's words ride in registers
        float tm = a.t[z - cz], tf = a.t[z], km = a.kmv[z - cz], k0 = a.kmv[z];
        float mhm = a.mh[z - cz], rhom = a.rho[z - cz];
#pragma unroll 4
        for (int f = f_lo; f <= f_hi; ++f, z += cz) {
            const float tp = a.t[z + cz], kp = a.kmv[z + cz];
            const float rrf = a.mf[z] / a.rf[z];
            const float mh = f < nk ? a.mh[z] : 0.0f, rho = f < nk ? a.rho[z] : 0.0f;
            const float r1 = (((km + k0) * mhm) * rhom) * rrf;
            const float r2 = (((k0 + kp) * mh) * rho) * rrf;
            const float cfa = tema * r1, cfc = tema * r2;
            float cfb, cfd;
            if (f == 1) {
                cfb = 1.0f - cfc;
                cfd = tf + temb * ((r2 * tp) - (r2 * tf));
            } else if (f == n) {
                cfb = 1.0f - cfa;
                cfd = tf + temb * ((-(r1 * tf)) + (r1 * tm));
            } else {
                cfb = (1.0f - cfa) - cfc;
                cfd = tf + temb * (((r2 * tp) - ((r1 + r2) * tf)) + (r1 * tm));
            }
            const int q = (f - 1) * 32;
            s_a[q] = cfa, s_b[q] = cfb, s_c[q] = cfc, s_d[q] = cfd;
            tm = tf, tf = tp, km = k0, k0 = kp, mhm = mh, rhom = rho;
        }
    }
    __syncthreads();
    // (chunks of four rows at 58 registers, four CTAs an SM: 640x768x80 885 us
    // against 602)
    if (wy == 0) column_sweep<2>(s_a, s_b, s_c, s_d, n);
    __syncthreads();
    if (!own) return;
    const int dw = i > 0 ? -1 : 0, de = i < ni - 1 ? 1 : 0, ds = j > 0 ? -ni : 0, dn = j < nj - 1 ? ni : 0;
    const bool ex = dw == 0 || de == 0, ey = ds == 0 || dn == 0;
#pragma unroll 2
    for (int f = f_lo; f <= f_hi; ++f) {
        const unsigned z = (unsigned)f * (unsigned)cz + (unsigned)c;
        const float rfz = a.rf[z], kz = a.kmh[z], t = a.t[z], ten = a.tketen[z];
        const float fw = tke_flux_flat(rfz, a.rf[z + dw], kz, a.kmh[z + dw], t, a.t[z + dw], a.rdx);
        const float fe = tke_flux_flat(a.rf[z + de], rfz, a.kmh[z + de], kz, a.t[z + de], t, a.rdx);
        const float fs = tke_flux_flat(rfz, a.rf[z + ds], kz, a.kmh[z + ds], t, a.t[z + ds], a.rdy);
        const float fn = tke_flux_flat(a.rf[z + dn], rfz, a.kmh[z + dn], kz, a.t[z + dn], t, a.rdy);
        const float hx = ex ? 0.0f : -((fe - fw) * a.rdx);
        const float hy = ey ? 0.0f : -((fn - fs) * a.rdy);
        const float tz = (rfz * (s_d[(f - 1) * 32] - t)) * rdt;
        a.tketen[z] = ten + ((hx + hy) + tz) / rfz;
    }
}

// ------------------------------------------------------------- RK stage
template <bool W>
__device__ __forceinline__ float rec5(float s1, float s2, float s3, float s4, float s5, double eps) {
    if (W) return weno5(s1, s2, s3, s4, s5, eps);
    return flx5(s1, s2, s3, s4, s5);
}

// the upwind flux at a face from the six points around it: one reconstruction
// of selected points, so a warp of mixed signs does not form both
template <bool W>
__device__ __forceinline__ float up6(float m, float s0, float s1, float s2, float s3, float s4, float s5, double eps) {
    const bool pos = m >= 0.0f;
    return m * rec5<W>(pos ? s0 : s5, pos ? s1 : s4, pos ? s2 : s3, pos ? s3 : s2, pos ? s4 : s1, eps);
}

// vertical flux at staggered index ks (cuda_tke_evolution.py:194-203) from
// levels ks-3 .. ks+2 of the column (win)
template <bool W>
__device__ __forceinline__ float vert_flux(const float win[6], float m, int ks, int nk, double eps) {
    const float wf = (float)eps;
#define Q(k) win[(k) - ks + 3]
    float r;
    if (ks == 1) {
        r = m >= 0.0f ? 0.5f * (Q(0) + Q(1)) : (W ? upstrpd(Q(2), Q(1), Q(0), wf) : flx3(Q(2), Q(1), Q(0)));
    } else if (ks == 2) {
        r = m >= 0.0f ? (W ? upstrpd(Q(0), Q(1), Q(2), wf) : flx3(Q(0), Q(1), Q(2)))
                      : rec5<W>(Q(4), Q(3), Q(2), Q(1), Q(0), eps);
    } else if (ks == nk - 1) {
        r = (W ? m > 0.0f : m >= 0.0f) ? rec5<W>(Q(ks - 3), Q(ks - 2), Q(ks - 1), Q(ks), Q(ks + 1), eps)
                                       : (W ? upstrpd(Q(ks + 1), Q(ks), Q(ks - 1), wf) : flx3(Q(ks + 1), Q(ks), Q(ks - 1)));
    } else if (ks == nk) {
        r = (W ? m > 0.0f : m >= 0.0f) ? (W ? upstrpd(Q(ks - 2), Q(ks - 1), Q(ks), wf) : flx3(Q(ks - 2), Q(ks - 1), Q(ks)))
                                       : 0.5f * (Q(ks - 1) + Q(ks));
    } else {
        return up6<W>(m, Q(ks - 3), Q(ks - 2), Q(ks - 1), Q(ks), Q(ks + 1), Q(ks + 2), eps);
    }
#undef Q
    return m * r;
}

constexpr int kStageOut = 31;   // cells a warp of 32 x faces completes
constexpr int kStageRows = 4;   // rows per CTA of the fifth-order stage, each independent
constexpr int kStageWRows = 8;  // rows per CTA of the WENO stage: 8 rows of y faces complete 7 rows of cells

// A warp owns the x faces i0 .. i0+31 of one row and marches up a chunk of
// face levels: each lane forms the x flux of one face and takes the next
// face's from the lane above, the upper vertical flux and the mass fluxes of
// the level above are carried down, the column's six levels stay in
// registers.  The fifth-order stage forms both y fluxes of a cell; the WENO
// stage hands each to the row below through shared memory (one barrier a
// level), the last row forming a flux only.  Columns beyond the open sides
// repeat the edge ones.  Bound by instruction issue (fifth order) and the
// binary64 weights (WENO); a step's three flat stages at 640x768x80 took 5.04 ms
// with six fluxes per cell and take 2.52 here (a fifth-order stage 0.497 ms,
// 0.624 with every offset clamped; WENO 1.524, and 1.787 with 16 warps an SM).
// FLAT: the flat column's advw (gm1_flat_tke_advw_rk_v1,
// src/cm1core/cuda_gm1_flat_stretched_closure.py:401-449; adv.F:3252-3355
// with terrain_flag=.false.): vertical divergence -(dumz(k)-dumz(k-1))*rdz
// *mf(k), the column's c1/c2 in the divergence correction and its rrf0, the
// open-side divergence piece (q*d)*rdx evaluated left to right, no gz.
template <bool W, bool FLAT>
__global__ void __launch_bounds__(32 * (W ? kStageWRows : kStageRows), W ? 3 : 8)
    tke_rk_stage_kernel(const __grid_constant__ TkeArgs a, const float *__restrict__ cur, float *__restrict__ nxt, float *__restrict__ nxt2,
                        int levels_per_chunk, float dttmp, double eps) {
    constexpr int ROWS = W ? kStageWRows : kStageRows;
    __shared__ float s_fy[W ? 2 : 1][W ? ROWS : 1][32], s_my[W ? 2 : 1][W ? ROWS : 1][32];
    const int lane = threadIdx.x, ty = threadIdx.y;
    const int ni = a.ni, nj = a.nj, nk = a.nk;
    const int ux = ni + 1 + 2 * kG, sx = ni + 2 * kG, uz = (nj + 2 * kG) * ux, vz = (nj + 1 + 2 * kG) * sx,
              wz = (nj + 2 * kG) * sx, cz = ni * nj;
    const int tiles = (ni + kStageOut - 1) / kStageOut;  // all tiles in one grid dimension, which takes any plane
    const int i0 = blockIdx.x % tiles * kStageOut + lane, row = blockIdx.x / tiles * (W ? ROWS - 1 : ROWS) + ty;
    if (!W && row >= nj) return;  // whole warps: the fifth-order stage has no barrier
    // faces and rows past the domain repeat its last ones and store nothing
    const int i = min(i0, ni), j = min(row, W ? nj : nj - 1);
    const bool own = i0 < ni && row < nj && lane < kStageOut && (!W || ty < ROWS - 1);
    const int jc = min(j, nj - 1), ic = min(i, ni - 1), cc = jc * ni + ic;
    const int ou = (jc + kG) * ux + i + kG, ov = (j + kG) * sx + ic + kG, ow = (jc + kG) * sx + ic + kG;
    // a warp whose stencils stay inside the plane loads them at fixed offsets,
    // one at its edge at clamped columns and rows
    const bool inside = __all_sync(0xffffffffu, i >= 3 && i + 2 < ni) && j >= 3 && j + 3 < nj;
    auto xo = [&](int q) { return jc * ni + clampi(i + q - 3, ni); };
    auto yo = [&](int q) { return clampi(j + q - 3, nj) * ni + ic; };
    // window of the own column: levels f_lo-4 .. f_lo+1, shifted to f-3 .. f+2
    const int f_lo = blockIdx.y * levels_per_chunk, f_hi = min(nk, f_lo + levels_per_chunk - 1);
    if (f_lo == 0 && own) {
        nxt[cc] = 0.0f;
        if (nxt2) nxt2[cc] = 0.0f;
    }
    if (f_hi == nk && own) {
        const unsigned z = (unsigned)nk * (unsigned)cz + (unsigned)cc;
        nxt[z] = 0.0f;
        if (nxt2) nxt2[z] = 0.0f;
    }
    const int k_lo = max(f_lo, 1), k_hi = min(f_hi, nk - 1);
    if (k_lo > k_hi) return;  // the whole CTA
    float win[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        const int l = k_lo - 3 + q;
        win[q] = l >= 0 && l <= nk ? cur[l * cz + cc] : 0.0f;
    }
    float rw = __ldg(a.rrw + (k_lo + 1) * wz + ow);
    float zlo = vert_flux<W>(win, 0.5f * (__ldg(a.rrw + k_lo * wz + ow) + rw), k_lo, nk, eps);
    float rul = __ldg(a.rru + k_lo * uz + ou), rsl = __ldg(a.rrv + k_lo * vz + ov), rnl = 0.0f;
    if (!W) rnl = __ldg(a.rrv + k_lo * vz + ov + sx);
    float dl = __ldg(a.divx + (k_lo - 1) * cz + cc);
    const float gz = FLAT ? 0.0f : __ldg(a.gz + cc);
    // WENO rows of cells away from the open sides, at levels away from the
    // column's ends, take a finish without those branches (256x256x80: 249 ->
    // 234 us; the fifth-order stage gains nothing from it, 86 against 89)
    const bool edge = !W || __any_sync(0xffffffffu, i == 0 || i == ni - 1) || j == 0 || j == nj - 1;
#pragma unroll 1
    for (int f = k_lo; f <= k_hi; ++f) {
        const float *lev = cur + f * cz;
        const float q = win[3];
        const float *c2p = a.c2 + f * cz;
        float px[6], py[7], kw, ks, kn = 0.0f;
        px[3] = py[3] = q;  // the centre is the own column's
        py[6] = 0.0f;
        if (inside) {
            const float *pt = lev + cc, *pc = c2p + cc;
            kw = __ldg(pc - 1), ks = __ldg(pc - ni);
            if (!W) kn = __ldg(pc + ni);
#pragma unroll
            for (int e = 0; e < 6; ++e)
                if (e != 3) px[e] = __ldg(pt + (e - 3));
#pragma unroll
            for (int e = 0; e < (W ? 6 : 7); ++e)
                if (e != 3) py[e] = __ldg(pt + (e - 3) * ni);
        } else {
            kw = __ldg(c2p + xo(2)), ks = __ldg(c2p + yo(2));
            if (!W) kn = __ldg(c2p + yo(4));
#pragma unroll
            for (int e = 0; e < 6; ++e)
                if (e != 3) px[e] = __ldg(lev + xo(e));
#pragma unroll
            for (int e = 0; e < (W ? 6 : 7); ++e)
                if (e != 3) py[e] = __ldg(lev + yo(e));
        }
        const float next = f + 3 <= nk ? __ldg(lev + 3 * cz + cc) : 0.0f;
        const float c2 = __ldg(c2p + cc);
        const float ru = __ldg(a.rru + (f + 1) * uz + ou), rs = __ldg(a.rrv + (f + 1) * vz + ov);
        const float rwn = __ldg(a.rrw + (f + 2) * wz + ow), dh = __ldg(a.divx + f * cz + cc);
        const unsigned z = (unsigned)f * (unsigned)cz + (unsigned)cc;
        const float base = a.tkea[z], ten = __ldg(a.tketen + z);
        const float rrf = FLAT ? __ldg(a.rrf0 + f * cz) : __ldg(a.rrf0 + z);
        const float c2x = 0.5f * (kw + c2), c2y = 0.5f * (ks + c2);
        const float mw = c2x * ru + (1.0f - c2x) * rul, ms = c2y * rs + (1.0f - c2y) * rsl;
        const float fx0 = up6<W>(mw, px[0], px[1], px[2], px[3], px[4], px[5], eps);
        const float fy0 = up6<W>(ms, py[0], py[1], py[2], py[3], py[4], py[5], eps);
        const float fx1 = __shfl_down_sync(0xffffffffu, fx0, 1);
        float fy1, mn, rn = 0.0f;
        if (W) {
            s_fy[f & 1][ty][lane] = fy0;
            s_my[f & 1][ty][lane] = ms;
            __syncthreads();
            const int up = min(ty + 1, ROWS - 1);
            fy1 = s_fy[f & 1][up][lane];
            mn = s_my[f & 1][up][lane];
        } else {
            rn = __ldg(a.rrv + (f + 1) * vz + ov + sx);
            const float c2n = 0.5f * (c2 + kn);
            mn = c2n * rn + (1.0f - c2n) * rnl;
            fy1 = up6<W>(mn, py[1], py[2], py[3], py[4], py[5], py[6], eps);
        }
#pragma unroll
        for (int e = 0; e < 5; ++e) win[e] = win[e + 1];
        win[5] = next;
        const float mz = 0.5f * (rw + rwn), c1 = 1.0f - c2;
        float ax, ay, zhi;
        if (!edge && f >= 2 && f < nk - 2) {
            zhi = up6<W>(mz, win[0], win[1], win[2], win[3], win[4], win[5], eps);
            ax = -1.0f * ((fx1 - fx0) * a.rdx);
            ay = -1.0f * ((fy1 - fy0) * a.rdy);
        } else {
            const float me = __shfl_down_sync(0xffffffffu, mw, 1), rue = __shfl_down_sync(0xffffffffu, ru, 1);
            const float rule = __shfl_down_sync(0xffffffffu, rul, 1);
            // inflow through an open side's face takes the inner neighbour's flux
            const bool sw = i == 0 && mw >= 0.0f, se = i == ni - 1 && me <= 0.0f;
            const bool ss = j == 0 && ms >= 0.0f, sn = j == nj - 1 && mn <= 0.0f;
            zhi = vert_flux<W>(win, mz, f + 1, nk, eps);
            ax = -1.0f * (((se ? fx0 : fx1) - (sw ? fx1 : fx0)) * a.rdx);
            ay = -1.0f * (((sn ? fy0 : fy1) - (ss ? fy1 : fy0)) * a.rdy);
            if (sw || se) {
                const float du = c1 * (rule - rul) + c2 * (rue - ru);
                ax = FLAT ? ax - ((q * du) * a.rdx) : ax - q * (du * a.rdx);
            }
            if (ss || sn) {
                const float rnh = W ? __ldg(a.rrv + (f + 1) * vz + ov + sx) : rn;
                const float rnk = W ? __ldg(a.rrv + f * vz + ov + sx) : rnl;
                const float dv = c1 * (rnk - rsl) + c2 * (rnh - rs);
                ay = FLAT ? ay - ((q * dv) * a.rdy) : ay - q * (dv * a.rdy);
            }
        }
        const float dvf = zhi - zlo;
        const float az = FLAT ? ((-dvf) * a.rdz) * __ldg(a.mfp + f + 1) : -1.0f * (dvf * a.rdz);
        float total = (ax + ay) + az;
        // the divergence correction: the flat text reads the column's c2 here
        // (the open-side pieces above read the cell's)
        const float c2d = FLAT ? __ldg(c2p) : c2, c1d = FLAT ? 1.0f - c2d : c1;
        total = total + q * (c2d * dh + c1d * dl);
        const float wten = FLAT ? ten + total * rrf : ten + total * (rrf * gz);
        const float value = base + dttmp * wten;
        if (own) {
            const float out = value < 1e-10f ? 0.0f : value;
            nxt[z] = out;
            if (nxt2) nxt2[z] = out;
        }
        zlo = zhi, rw = rwn, rul = ru, rsl = rs, dl = dh;
        if (!W) rnl = rn;
    }
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

int tke_args(int ni, int nj, int nk, const gm1b_tke_evolution_arrays *s, float dx, float dy, float dz, float dt,
             TkeArgs &a, const char *what) {
    if (s == nullptr || ni < 3 || nj < 3 || nk < 6) {
        gm1b_set_error("%s: need arrays, ni >= 3, nj >= 3, nk >= 6", what);
        return GM1B_ERR_ARGUMENT;
    }
    if ((size_t)(nk + 3) * (size_t)(nj + 7) * (size_t)(ni + 7) >= ((size_t)1 << 31)) {
        gm1b_set_error("%s: a %dx%dx%d grid's padded arrays reach 2^31 words; the kernels index with 32-bit offsets",
                       what, ni, nj, nk);
        return GM1B_ERR_ARGUMENT;
    }
    const float v[4] = {dx, dy, dz, dt};
    for (float x : v)
        if (!(x > 0.0f) || !isfinite(x)) {
            gm1b_set_error("%s: dx, dy, dz, dt must be finite and > 0", what);
            return GM1B_ERR_ARGUMENT;
        }
    const void *need[] = {s->tkea, s->tke3d, s->tketen, s->kmh, s->kmv, s->rho, s->rf, s->mh, s->mf, s->gz,
                          s->rgz, s->rgzu, s->rgzv, s->c1, s->c2, s->rrf0, s->rru, s->rrv, s->rrw, s->divx};
    for (const void *q : need)
        if (q == nullptr) {
            gm1b_set_error("%s: a required array is NULL", what);
            return GM1B_ERR_ARGUMENT;
        }
    a.t = s->tke3d;
    a.kmh = s->kmh;
    a.kmv = s->kmv;
    a.rho = s->rho;
    a.rf = s->rf;
    a.mh = s->mh;
    a.mf = s->mf;
    a.gz = s->gz;
    a.rgz = s->rgz;
    a.rgzu = s->rgzu;
    a.rgzv = s->rgzv;
    a.tkea = s->tkea;
    a.c2 = s->c2;
    a.rrf0 = s->rrf0;
    a.rru = s->rru;
    a.rrv = s->rrv;
    a.rrw = s->rrw;
    a.divx = s->divx;
    a.tketen = s->tketen;
    a.ni = ni;
    a.nj = nj;
    a.nk = nk;
    a.rdx = 1.0f / dx;
    a.rdy = 1.0f / dy;
    a.rdz = 1.0f / dz;
    a.dz = dz;
    a.zt = (float)nk * dz;
    return GM1B_OK;
}

// four tridiagonal words of each of the nk-1 rows of 32 columns
size_t turbt_smem(int nk) { return (size_t)4 * (nk - 1) * 32 * sizeof(float); }

// Three warps a CTA for columns of up to 64 levels on a plane that gives the
// eight-warp CTAs (three an SM) three rounds of 148 SMs, else eight.  Eight and
// three warps, us: 256x256 of 24 levels 61 and 47, 40 levels 104 and 86, 64
// levels 159 and 148, 80 levels 196 and 249; 512x400x30 264 and 209; 179x261x32
// 58 and 51; 128x100x24 15 and 19.  (A thread per column: 47, 88, 312, 401;
// 233; 61; 39.)
int turbt_warps(unsigned tiles, int nk) { return nk <= 64 && tiles >= 3 * 3 * 148 ? 3 : 8; }

int enqueue_diffusion(const TkeArgs &a, float dt, cudaStream_t st) {
    const size_t smem = turbt_smem(a.nk);
    if (a.nk > kTurbtMostNk) {
        gm1b_set_error("gm1b_tke_diffusion: nk=%d exceeds the column solve's shared memory (nk <= 201)", a.nk);
        return GM1B_ERR_ARGUMENT;
    }
    static size_t configured[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64 && configured[dev] < smem) {
        cudaError_t e =
            cudaFuncSetAttribute(tke_turbt_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(tke_turbt_kernel<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        if (e != cudaSuccess) {
            cudaGetLastError();
            gm1b_set_error("cudaFuncSetAttribute(tke_turbt_kernel): %s", cudaGetErrorString(e));
            return GM1B_ERR_CUDA;
        }
        configured[dev] = 200 * 1024;
    }
    const unsigned tiles = (unsigned)((a.ni + 31) / 32) * (unsigned)a.nj;
    ProfScope ps("tke_turbt_kernel", st);
    if (turbt_warps(tiles, a.nk) == 3)
        tke_turbt_kernel<3><<<tiles, dim3(32, 3), smem, st>>>(a, dt);
    else
        tke_turbt_kernel<8><<<tiles, dim3(32, 8), smem, st>>>(a, dt);
    ps.stop();
    return launch_ok("tke_turbt_kernel") ? GM1B_OK : GM1B_ERR_CUDA;
}

// Levels per chunk: long chunks re-load and re-form less (each starts with
// six window loads and its lower flux), short ones give a small plane warps
// enough: halve until two rounds of `warps` on each of 148 SMs, or at most
// four levels, are left, and to two where eight warps an SM are not (a WENO
// stage: 37x24x24 12.9 -> 8.5 us, 28x44x49 13.0 -> 10.2, a thread per cell 10.7
// and 11.7; 64x64x64 gains nothing, 128x100x64 loses 5%).
int stage_chunk(const TkeArgs &a, int warps) {
    const long long rows = (long long)((a.ni + kStageOut - 1) / kStageOut) * a.nj;
    int chunk = a.nk + 1;
    auto row_warps = [&] { return rows * ((a.nk + chunk) / chunk); };
    while (chunk > 4 && row_warps() < 2LL * 148 * warps) chunk = (chunk + 1) / 2;
    if (chunk > 2 && row_warps() < 148 * 8) chunk = 2;
    return chunk;
}

template <bool FLAT>
int enqueue_stage(const TkeArgs &a, const float *cur, float *nxt, float *nxt2, int nrk, float dt, cudaStream_t st) {
    const float dttmp = dt / (float)(4 - nrk);
    const double eps = (double)(100.0f * 1e-18f);
    const bool weno = nrk == 3;
    const int rows = weno ? kStageWRows - 1 : kStageRows, chunk = stage_chunk(a, weno ? 16 : 24);
    const dim3 grid((a.ni + kStageOut - 1) / kStageOut * ((a.nj + rows - 1) / rows), (a.nk + chunk) / chunk);
    const char *name = FLAT ? "tke_rk_stage_flat_kernel" : "tke_rk_stage_kernel";
    ProfScope ps(name, st);
    if (weno)
        tke_rk_stage_kernel<true, FLAT><<<grid, dim3(32, kStageWRows), 0, st>>>(a, cur, nxt, nxt2, chunk, dttmp, eps);
    else
        tke_rk_stage_kernel<false, FLAT><<<grid, dim3(32, kStageRows), 0, st>>>(a, cur, nxt, nxt2, chunk, dttmp, eps);
    ps.stop();
    return launch_ok(name) ? GM1B_OK : GM1B_ERR_CUDA;
}

// Flat column arguments: the arrays the flat turbt and RK stage read.
int tke_args_flat(int ni, int nj, int nk, const gm1b_tke_evolution_arrays *s, float dx, float dy, float rdz,
                  float dt, TkeArgs &a, bool stage, const float *mf_profile, const char *what) {
    if (s == nullptr || ni < 3 || nj < 3 || nk < 6) {
        gm1b_set_error("%s: need arrays, ni >= 3, nj >= 3, nk >= 6", what);
        return GM1B_ERR_ARGUMENT;
    }
    if ((size_t)(nk + 3) * (size_t)(nj + 7) * (size_t)(ni + 7) >= ((size_t)1 << 31)) {
        gm1b_set_error("%s: a %dx%dx%d grid's padded arrays reach 2^31 words; the kernels index with 32-bit offsets",
                       what, ni, nj, nk);
        return GM1B_ERR_ARGUMENT;
    }
    const float v[4] = {dx, dy, rdz, dt};
    for (float x : v)
        if (!(x > 0.0f) || !isfinite(x)) {
            gm1b_set_error("%s: dx, dy, rdz, dt must be finite and > 0", what);
            return GM1B_ERR_ARGUMENT;
        }
    const void *turbt_need[] = {s->tke3d, s->tketen, s->kmh, s->kmv, s->rho, s->rf, s->mh, s->mf};
    const void *stage_need[] = {s->tkea, s->tketen, s->c2, s->rrf0, s->rru, s->rrv, s->rrw, s->divx, mf_profile};
    if (stage) {
        for (const void *q : stage_need)
            if (q == nullptr) {
                gm1b_set_error("%s: a required array is NULL", what);
                return GM1B_ERR_ARGUMENT;
            }
    } else {
        for (const void *q : turbt_need)
            if (q == nullptr) {
                gm1b_set_error("%s: a required array is NULL", what);
                return GM1B_ERR_ARGUMENT;
            }
    }
    a = TkeArgs{};
    a.t = s->tke3d;
    a.kmh = s->kmh;
    a.kmv = s->kmv;
    a.rho = s->rho;
    a.rf = s->rf;
    a.mh = s->mh;
    a.mf = s->mf;
    a.tkea = s->tkea;
    a.c2 = s->c2;
    a.rrf0 = s->rrf0;
    a.rru = s->rru;
    a.rrv = s->rrv;
    a.rrw = s->rrw;
    a.divx = s->divx;
    a.tketen = s->tketen;
    a.mfp = mf_profile;
    a.ni = ni;
    a.nj = nj;
    a.nk = nk;
    a.rdx = 1.0f / dx;
    a.rdy = 1.0f / dy;
    a.rdz = rdz;
    return GM1B_OK;
}

}  // namespace

extern "C" int32_t gm1b_tke_diffusion(int32_t ni, int32_t nj, int32_t nk, const gm1b_tke_evolution_arrays *arrays,
                                      float dx, float dy, float dz, float dt, void *stream) {
    TkeArgs a;
    const int r = tke_args(ni, nj, nk, arrays, dx, dy, dz, dt, a, "gm1b_tke_diffusion");
    if (r != GM1B_OK) return r;
    return enqueue_diffusion(a, dt, static_cast<cudaStream_t>(stream));
}

extern "C" int32_t gm1b_tke_diffusion_flat(int32_t ni, int32_t nj, int32_t nk,
                                           const gm1b_tke_evolution_arrays *arrays, float dx, float dy, float rdz,
                                           float dt, void *stream) {
    TkeArgs a;
    const int r = tke_args_flat(ni, nj, nk, arrays, dx, dy, rdz, dt, a, false, nullptr, "gm1b_tke_diffusion_flat");
    if (r != GM1B_OK) return r;
    const size_t smem = turbt_smem(nk);
    if (nk > kTurbtMostNk) {
        gm1b_set_error("gm1b_tke_diffusion_flat: nk=%d exceeds the column solve's shared memory (nk <= 201)", nk);
        return GM1B_ERR_ARGUMENT;
    }
    static size_t configured[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64 && configured[dev] < smem) {
        const cudaError_t e =
            cudaFuncSetAttribute(tke_turbt_flat_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        if (e != cudaSuccess) {
            cudaGetLastError();
            gm1b_set_error("cudaFuncSetAttribute(tke_turbt_flat_kernel): %s", cudaGetErrorString(e));
            return GM1B_ERR_CUDA;
        }
        configured[dev] = 200 * 1024;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    ProfScope ps("tke_turbt_flat_kernel", st);
    tke_turbt_flat_kernel<<<(ni + 31) / 32 * nj, dim3(32, kTurbtWarps), smem, st>>>(a, dt);
    ps.stop();
    return launch_ok("tke_turbt_flat_kernel") ? GM1B_OK : GM1B_ERR_CUDA;
}

extern "C" int32_t gm1b_tke_rk_stage_flat(int32_t ni, int32_t nj, int32_t nk,
                                          const gm1b_tke_evolution_arrays *arrays, const float *mf_profile,
                                          const float *cur, float *nxt, int32_t nrk, float dx, float dy, float rdz,
                                          float dt, void *stream) {
    TkeArgs a;
    const int r = tke_args_flat(ni, nj, nk, arrays, dx, dy, rdz, dt, a, true, mf_profile, "gm1b_tke_rk_stage_flat");
    if (r != GM1B_OK) return r;
    if (cur == nullptr || nxt == nullptr || cur == nxt || nrk < 1 || nrk > 3) {
        gm1b_set_error("gm1b_tke_rk_stage_flat: need distinct cur and nxt and nrk in 1..3");
        return GM1B_ERR_ARGUMENT;
    }
    return enqueue_stage<true>(a, cur, nxt, nullptr, nrk, dt, static_cast<cudaStream_t>(stream));
}

extern "C" int32_t gm1b_tke_rk_stage(int32_t ni, int32_t nj, int32_t nk, const gm1b_tke_evolution_arrays *arrays,
                                     const float *cur, float *nxt, int32_t nrk, float dx, float dy, float dz, float dt,
                                     void *stream) {
    TkeArgs a;
    const int r = tke_args(ni, nj, nk, arrays, dx, dy, dz, dt, a, "gm1b_tke_rk_stage");
    if (r != GM1B_OK) return r;
    if (cur == nullptr || nxt == nullptr || cur == nxt || nrk < 1 || nrk > 3) {
        gm1b_set_error("gm1b_tke_rk_stage: need distinct cur and nxt and nrk in 1..3");
        return GM1B_ERR_ARGUMENT;
    }
    return enqueue_stage<false>(a, cur, nxt, nullptr, nrk, dt, static_cast<cudaStream_t>(stream));
}

extern "C" int32_t gm1b_tke_evolution(int32_t ni, int32_t nj, int32_t nk, const gm1b_tke_evolution_arrays *arrays,
                                      float *workspace, float dx, float dy, float dz, float dt, void *stream) {
    TkeArgs a;
    const int r = tke_args(ni, nj, nk, arrays, dx, dy, dz, dt, a, "gm1b_tke_evolution");
    if (r != GM1B_OK) return r;
    if (workspace == nullptr) {
        gm1b_set_error("gm1b_tke_evolution: need a workspace of (nk+1)*nj*ni floats");
        return GM1B_ERR_ARGUMENT;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    float *tke3d = arrays->tke3d, *tkea = arrays->tkea;
    int s = enqueue_diffusion(a, dt, st);
    // stage 1: tke3d -> workspace; stage 2: workspace -> tke3d; stage 3:
    // tke3d -> tkea (each cell reads only its own tkea word) and workspace
    if (s == GM1B_OK) s = enqueue_stage<false>(a, tke3d, workspace, nullptr, 1, dt, st);
    if (s == GM1B_OK) s = enqueue_stage<false>(a, workspace, tke3d, nullptr, 2, dt, st);
    if (s == GM1B_OK) s = enqueue_stage<false>(a, tke3d, workspace, tkea, 3, dt, st);
    if (s != GM1B_OK) return s;
    const size_t bytes = (size_t)(nk + 1) * nj * ni * sizeof(float);
    const cudaError_t e = cudaMemcpyAsync(tke3d, workspace, bytes, cudaMemcpyDeviceToDevice, st);
    if (e != cudaSuccess) {
        gm1b_set_error("gm1b_tke_evolution: commit copy: %s", cudaGetErrorString(e));
        return GM1B_ERR_CUDA;
    }
    return GM1B_OK;
}
