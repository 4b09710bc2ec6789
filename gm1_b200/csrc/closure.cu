// closure.cu - sm_100a kernels of the two inputs of the TKE source:
// deformation (CM1 calcdef, Cartesian terrain branch, four open sides) and
// the moist squared buoyancy frequency (CM1 calcnm, six-species ice-aware
// branch).
//
// Behaviour followed (reference file:line):
//   cpu_terrain_deformation_inplace   src/cm1core/cuda_terrain_deformation.py:234-736
//   enqueue_flat_calcdef (flat column) src/cm1core/cuda_gm1_flat_stretched_closure.py:524-553, texts :76-136
//   cpu_moist_nm_inplace              src/cm1core/cuda_moist_nm.py:292-396
//
// Design (B200):
//  * calcdef is one z-marching kernel.  A warp owns 32 cells of a row and
//    walks a chunk of face levels upwards: each lane forms its cell's diagonal
//    strains, the corner shear s12 of its lower left corner, and the face
//    shears s13 and s23 of its west and south faces, and takes the other
//    corners and faces from the next lane (shuffle) and the next row (shared
//    memory).  The levels' velocities, their face-level sums and the corner
//    sums ride in registers from one level to the next, so every word is
//    loaded once a warp and nothing goes through device memory between stages
//    (the reference stores six scratch volumes and runs three launches).
//  * calcnm is elementwise per face level: each thread forms the cell
//    diagnostics of its own level and of the level below and the face value
//    between them, so columns need no serial walk; the branch counts are
//    reduced per CTA with __syncthreads_count before one atomicAdd.
//  * Arithmetic is binary32 one operation at a time in the reference's
//    order (the library is built with --fmad=false), so calcdef is
//    word-identical to the reference; calcnm passes through logf/expf.
#include "gm1b_common.cuh"

namespace gm1b {
namespace {

constexpr int kDefRows = 8;  // rows of corners per calcdef CTA; they complete 7 rows of cells
constexpr int kDefOut = 31;  // cells a warp of 32 corners completes

struct DefArgs {
    const float *u, *v, *w, *rho, *rf, *c1, *c2, *gz, *rgz, *rgzu, *rgzv, *gx, *gy;
    const float *mf3, *mhp;  // flat column: face mf (nk+1, nj, ni) and the mh profile (nk+2, CM1-indexed)
    float *defv, *defh;
    int ni, nj, nk;
    float rdx, rdy, rds, zt, dz;
    float rdz;  // flat column: the vertical coordinate's reference 1/dz
};

// 32-bit element offsets (the entry points refuse grids whose arrays reach
// 2^31 words)
__device__ __forceinline__ unsigned i3(int k, int j, int i, int ny, int nx) {
    return ((unsigned)k * (unsigned)ny + (unsigned)j) * (unsigned)nx + (unsigned)i;
}

// face-level value of a column (nk levels, `stride` words apart)
__device__ __forceinline__ float atw(const float *q, unsigned kf, unsigned nk, unsigned stride) {
    if (kf != 0 && kf != nk) return 0.5f * (q[(kf - 1) * stride] + q[kf * stride]);
    const unsigned k0 = kf == 0 ? 0 : nk - 1, k1 = kf == 0 ? 1 : nk - 2, k2 = kf == 0 ? 2 : nk - 3;
    float r = 1.875f * q[k0 * stride];
    r = r + (-1.25f) * q[k1 * stride];
    return r + 0.375f * q[k2 * stride];
}

__device__ __forceinline__ float sq(float x) { return x * x; }

// Face levels k_lo .. k_hi of a chunk, after the mass level k_lo - 1 below
// them.  FLAT selects the flat column's strain texts, rdz*mh(k) / rdz*mf(k)
// (gm1_flat_calcdef_mass_v1 / _face_v1,
// src/cm1core/cuda_gm1_flat_stretched_closure.py:76-112; turb.F:4772-4786,
// :4880-4895); the deformation reduction of turb.F:5361-5385 is the same in
// both branches.  Corners at the open sides are the nearest interior ones
// (constant extension).  Bound by instruction issue and the loads' latency.
// One CTA per 32 x 8 columns with every strain in shared memory (33 x 9 corners
// take its 256 threads two passes, ~125 loads a level) took 473 us at
// 256x256x80 on terrain and 0.84 ms at 640x768x80 flat; this takes 146 and
// 0.59 (24 and 32 warps an SM; 16 and 24: 193 and 0.74).  At 24 warps the
// terrain strains spill 132 bytes; with 16 and no spill 256x256x80 takes 161 us
// for 140, 300x301x30 85 for 77, and the smallest planes less (53x48x40 7.4 for
// 9.1).
template <bool FLAT>
__global__ void __launch_bounds__(32 * kDefRows, FLAT ? 4 : 3)
    calcdef_march_kernel(const __grid_constant__ DefArgs p, int levels_per_chunk) {
    __shared__ float s_12[2][kDefRows][32], s_23[2][kDefRows][32];
    const int lane = threadIdx.x, ty = threadIdx.y;
    const int ni = p.ni, nj = p.nj, nk = p.nk, ux = ni + 1, vy = nj + 1;
    const int tiles = (ni + kDefOut - 1) / kDefOut;
    const int i0 = blockIdx.x % tiles * kDefOut + lane, row = blockIdx.x / tiles * (kDefRows - 1) + ty;
    const bool own = i0 < ni && row < nj && lane < kDefOut && ty < kDefRows - 1;
    const int i = min(i0, ni), j = min(row, nj);  // faces past the domain repeat its last ones
    const int ic = min(i, ni - 1), jc = min(j, nj - 1), iw = max(i - 1, 0), js = max(j - 1, 0);
    const int ii = min(max(i, 1), ni - 1), jj = min(max(j, 1), nj - 1);  // the corner
    const unsigned uz = (unsigned)nj * ux, vz = (unsigned)vy * ni, cz = (unsigned)nj * ni;
    const unsigned oc = i3(0, jc, ic, nj, ni), ow = i3(0, jc, iw, nj, ni), os = i3(0, js, ic, nj, ni);
    const unsigned oua = i3(0, jj, ii, nj, ux), oub = oua - ux, ouc = i3(0, jc, i, nj, ux);
    const unsigned ova = i3(0, jj, ii, vy, ni), ovb = ova - 1, ovc = i3(0, j, ic, vy, ni),
                   ovd = i3(0, min(j + 1, nj), ic, vy, ni);
    const unsigned orr = i3(0, jj, ii, nj, ni);  // the corner's north-east cell
    const int k_lo = 1 + blockIdx.y * levels_per_chunk, k_hi = min(nk - 1, k_lo + levels_per_chunk - 1);
    const unsigned k0 = k_lo - 1;
    // a, b: the corner's two faces of each field; c (and d): the cell's
    float ua = p.u[k0 * uz + oua], ub = p.u[k0 * uz + oub], uc = p.u[k0 * uz + ouc], um = 0.0f;
    float va = p.v[k0 * vz + ova], vb = p.v[k0 * vz + ovb], vc = p.v[k0 * vz + ovc], vd = p.v[k0 * vz + ovd], vm = 0.0f;
    float wc = p.w[k0 * cz + oc], ww = p.w[k0 * cz + ow], ws = p.w[k0 * cz + os];
    // sums at the lower face level of the two faces of each kind, and the
    // metric there
    float xl = 0.0f, yl = 0.0f, gl = 0.0f, hl = 0.0f, wlx = 0.0f, wly = 0.0f;
    if (!FLAT) {
        xl = atw(p.u + oub, k0, nk, uz) + atw(p.u + oua, k0, nk, uz);
        yl = atw(p.v + ovb, k0, nk, vz) + atw(p.v + ova, k0, nk, vz);
        const float fu = atw(p.u + ouc, k0, nk, uz);
        gl = p.gx[k0 * cz + oc] * (fu + __shfl_down_sync(0xffffffffu, fu, 1));
        hl = p.gy[k0 * cz + oc] * (atw(p.v + ovc, k0, nk, vz) + atw(p.v + ovd, k0, nk, vz));
    }
    float g = 0.0f, gw = 0.0f, gs = 0.0f, rg = 0.0f, rgw = 0.0f, rgs = 0.0f;
    float ga = 0.0f, gb = 0.0f, gc = 0.0f, gd = 0.0f, rua = 0.0f, rub = 0.0f, ruc = 0.0f, rue = 0.0f, rva = 0.0f,
          rvb = 0.0f, rvc = 0.0f, rvd = 0.0f;
    if (!FLAT) {
        g = p.gz[oc], gw = p.gz[ow], gs = p.gz[os], rg = p.rgz[oc], rgw = p.rgz[ow], rgs = p.rgz[os];
        ga = p.gz[orr], gb = p.gz[orr - 1], gc = p.gz[orr - ni], gd = p.gz[orr - ni - 1];
        rua = p.rgzu[oua], rub = p.rgzu[oub], ruc = p.rgzu[ouc];
        rue = __shfl_down_sync(0xffffffffu, ruc, 1);
        rva = p.rgzv[ova], rvb = p.rgzv[ovb], rvc = p.rgzv[ovc], rvd = p.rgzv[ovd];
    }
    float p11 = 0.0f, p22 = 0.0f, p33 = 0.0f, lo12 = 0.0f;  // the mass level below
#pragma unroll 1
    for (int kf = k_lo - 1; kf <= k_hi; ++kf) {
        const unsigned k = kf, z = k * cz;
        const bool more = kf + 1 < nk;
        const unsigned un = (k + 1) * uz, vn = (k + 1) * vz;
        const float nua = more ? p.u[un + oua] : 0.0f, nub = more ? p.u[un + oub] : 0.0f, nuc = more ? p.u[un + ouc] : 0.0f;
        const float nva = more ? p.v[vn + ova] : 0.0f, nvb = more ? p.v[vn + ovb] : 0.0f,
                    nvc = more ? p.v[vn + ovc] : 0.0f, nvd = more ? p.v[vn + ovd] : 0.0f;
        const float nwc = p.w[z + cz + oc], nww = p.w[z + cz + ow], nws = p.w[z + cz + os];
        const float rfc = p.rf[z + oc], rfw = p.rf[z + ow], rfs = p.rf[z + os];
        const float a = p.c1[z + oc], b = p.c2[z + oc];
        const float r = p.rho[z + oc], ra = p.rho[z + orr], rb = p.rho[z + orr - 1], rc = p.rho[z + orr - ni],
                    rd = p.rho[z + orr - ni - 1];
        const float ue = __shfl_down_sync(0xffffffffu, uc, 1);
        float c11, c22, c33, c12, c13 = 0.0f, c23 = 0.0f;
        if (FLAT) {
            c11 = (r * (ue - uc)) * p.rdx;
            c22 = (r * (vd - vc)) * p.rdy;
            c33 = (r * (nwc - wc)) * (p.rdz * p.mhp[kf + 1]);
            const float x = (ua - ub) * p.rdy, y = (va - vb) * p.rdx;
            c12 = ((0.5f * (x + y)) * 0.25f) * ((rd + ra) + (rb + rc));
            if (kf >= k_lo) {
                const float mc = p.mf3[z + oc], mw = p.mf3[z + ow], ms = p.mf3[z + os];
                const float du = (((uc - um) * p.rdz) * 0.5f) * (mw + mc);
                c13 = ((0.5f * ((wc - ww) * p.rdx + du)) * 0.5f) * (rfw + rfc);
                const float dv = (((vc - vm) * p.rdz) * 0.5f) * (ms + mc);
                c23 = ((0.5f * ((wc - ws) * p.rdy + dv)) * 0.5f) * (rfs + rfc);
            }
        } else {
            // the velocities at the upper face level
            float xu, yu, fu, fv;
            if (more) {
                xu = 0.5f * (ub + nub) + 0.5f * (ua + nua);
                yu = 0.5f * (vb + nvb) + 0.5f * (va + nva);
                fu = 0.5f * (uc + nuc);
                fv = 0.5f * (vc + nvc) + 0.5f * (vd + nvd);
            } else {
                xu = atw(p.u + oub, nk, nk, uz) + atw(p.u + oua, nk, nk, uz);
                yu = atw(p.v + ovb, nk, nk, vz) + atw(p.v + ova, nk, nk, vz);
                fu = atw(p.u + ouc, nk, nk, uz);
                fv = atw(p.v + ovc, nk, nk, vz) + atw(p.v + ovd, nk, nk, vz);
            }
            const float gu = p.gx[z + cz + oc] * (fu + __shfl_down_sync(0xffffffffu, fu, 1));
            const float hu = p.gy[z + cz + oc] * fv;
            float hor = (g * (ue * rue - uc * ruc)) * p.rdx;
            c11 = (hor + ((gu - gl) * 0.5f) * p.rds) * r;
            hor = (g * (vd * rvd - vc * rvc)) * p.rdy;
            c22 = (hor + ((hu - hl) * 0.5f) * p.rds) * r;
            c33 = (((nwc - wc) * p.rds) * g) * r;
            const float z_hi = p.zt - (float)(kf + 1) * p.dz, z_lo = p.zt - (float)kf * p.dz;
            const float r1 = 0.25f * ((rd * gd + ra * ga) + (rb * gb + rc * gc));
            const float x1 = (r1 * (ua * rua - ub * rub)) * p.rdy;
            const float x2 = ((((0.5f * (z_hi * xu - z_lo * xl)) * p.rds) * r1) * (rua - rub)) * p.rdy;
            const float y1 = (r1 * (va * rva - vb * rvb)) * p.rdx;
            const float y2 = ((((0.5f * (z_hi * yu - z_lo * yl)) * p.rds) * r1) * (rva - rvb)) * p.rdx;
            c12 = 0.5f * ((x1 + x2) + (y1 + y2));
            const float zm_u = p.zt - ((float)kf + 0.5f) * p.dz, zm_l = p.zt - ((float)kf - 0.5f) * p.dz;
            const float hc = 0.5f * (wc + nwc), wux = hc + 0.5f * (ww + nww), wuy = hc + 0.5f * (ws + nws);
            if (kf >= k_lo) {
                const float du = (uc - um) * p.rds, hx = (wc * rg - ww * rgw) * p.rdx;
                const float tx = (((0.5f * p.rds) * (zm_u * wux - zm_l * wlx)) * (rg - rgw)) * p.rdx;
                c13 = (0.5f * ((du + hx) + tx)) * (0.5f * (gw * rfw + g * rfc));
                const float dv = (vc - vm) * p.rds, hy = (wc * rg - ws * rgs) * p.rdy;
                const float ty2 = (((0.5f * p.rds) * (zm_u * wuy - zm_l * wly)) * (rg - rgs)) * p.rdy;
                c23 = (0.5f * ((dv + hy) + ty2)) * (0.5f * (gs * rfs + g * rfc));
            }
            xl = xu, yl = yu, gl = gu, hl = hu, wlx = wux, wly = wuy;
        }
        s_12[kf & 1][ty][lane] = c12;
        s_23[kf & 1][ty][lane] = c23;
        __syncthreads();
        const int up = min(ty + 1, kDefRows - 1);
        const float n12 = s_12[kf & 1][up][lane], ne12 = s_12[kf & 1][up][min(lane + 1, 31)];
        const float e12 = __shfl_down_sync(0xffffffffu, c12, 1), e13 = __shfl_down_sync(0xffffffffu, c13, 1);
        const float hi12 = (sq(c12) + sq(ne12)) + (sq(n12) + sq(e12));
        if (kf >= k_lo && own) {
            const float t11 = a * sq(p11) + b * sq(c11);
            const float t22 = a * sq(p22) + b * sq(c22);
            const float t33 = a * sq(p33) + b * sq(c33);
            const float t12 = 0.25f * (a * lo12 + b * hi12);
            const float t13 = 0.5f * (sq(c13) + sq(e13));
            const float t23 = 0.5f * (sq(c23) + sq(s_23[kf & 1][up][lane]));
            const float rrf = rcp_rn(rfc * rfc);
            p.defv[z + oc] = (4.0f * (t13 + t23)) * rrf;
            p.defh[z + oc] = ((2.0f * ((t11 + t22) + t33)) + 4.0f * t12) * rrf;
        }
        p11 = c11, p22 = c22, p33 = c33, lo12 = hi12;
        um = uc, uc = nuc, ua = nua, ub = nub;
        vm = vc, vc = nvc, vd = nvd, va = nva, vb = nvb;
        wc = nwc, ww = nww, ws = nws;
    }
    if (own && blockIdx.y == 0) {
        p.defv[oc] = 0.0f;
        p.defh[oc] = 0.0f;
        p.defv[(unsigned)nk * cz + oc] = 0.0f;
        p.defh[(unsigned)nk * cz + oc] = 0.0f;
    }
}

// ---------------------------------------------------------------- calcnm
struct NmConsts {
    float g, rd, cp, cpv, cpl, cpi, eps, reps, lv1, lv2, ls1, ls2;
};

struct NmArgs {
    const float *c1, *c2, *mf, *pi0, *th0, *prs, *pp3d, *th3d, *q3d;
    float *nm, *temperature, *qt, *thv, *qvci;
    uint8_t *mask;
    unsigned long long *counts;
    int ni, nj, nk;
    float rdz;
    NmConsts c;
};

struct NmCell {
    float t, qt, thv, qvci;
};

__device__ __forceinline__ NmCell nm_cell(const NmArgs &a, int k, unsigned p) {
    const unsigned cells = (unsigned)a.nk * a.nj * a.ni;
    NmCell r;
    const float qv = a.q3d[p];
    r.qvci = (qv + a.q3d[cells + p]) + a.q3d[3 * cells + p];
    float t = 0.0f;
#pragma unroll
    for (int s = 0; s < 6; ++s) t = t + a.q3d[s * cells + p];
    r.qt = t;
    const float theta = a.th0[k] + a.th3d[p];
    const float exner = a.pi0[k] + a.pp3d[p];
    r.t = theta * exner;
    const float tv = theta * (1.0f + a.c.reps * qv);
    r.thv = tv / (1.0f + t);
    return r;
}

__device__ __forceinline__ float sat_liquid(float p, float t, float eps) {
    const float x = (17.67f * (t - 273.15f)) / (t - 29.65f);
    float es = 611.2f * expf(x);
    const float h = p * 0.5f;
    if (h < es) es = h;
    return (eps * es) / (p - es);
}

__device__ __forceinline__ float sat_ice(float p, float t, float eps) {
    const float x = (21.8745584f * (t - 273.15f)) / (t - 7.66f);
    float es = 611.2f * expf(x);
    const float h = p * 0.5f;
    if (h < es) es = h;
    return (eps * es) / (p - es);
}

__device__ __forceinline__ float nm_saturated(const NmConsts &c, const NmCell &up, const NmCell &lo, float tavg,
                                              float qtavg, float qvs, float ql, float qi, float qv, float mrdz,
                                              bool ice) {
    float cpml = c.cp + c.cpv * qv;
    cpml = cpml + c.cpl * ql;
    if (qi != 0.0f) cpml = cpml + c.cpi * qi;
    float lh, drdt, den;
    if (ice) {
        lh = c.ls1 - c.ls2 * tavg;
        drdt = 21.8745584f * (273.15f - 7.66f);
        den = (tavg - 7.66f) * (tavg - 7.66f);
    } else {
        lh = c.lv1 - c.lv2 * tavg;
        drdt = 17.67f * (273.15f - 29.65f);
        den = (tavg - 29.65f) * (tavg - 29.65f);
    }
    drdt = (drdt * qvs) / den;
    float gamma = c.g * (1.0f + qtavg);
    gamma = gamma * (1.0f + (lh * qvs) / (c.rd * tavg));
    gamma = gamma / (cpml + lh * drdt);
    float first = logf(up.t / lo.t) * mrdz;
    first = first + gamma / tavg;
    float second = tavg * drdt;
    second = second / (c.eps + qvs);
    first = first * (1.0f + second);
    float moist = logf((1.0f + up.qt) / (1.0f + lo.qt));
    moist = moist * mrdz;
    return c.g * (first - moist);
}

// grid: x over i, y over j, z over face level kf = 0..nk
__global__ void __launch_bounds__(128) moist_nm_kernel(NmArgs a) {
    const int i = blockIdx.x * 32 + threadIdx.x;
    const int j = blockIdx.y * 4 + threadIdx.y;
    const int kf = blockIdx.z;
    const int ni = a.ni, nj = a.nj, nk = a.nk;
    const bool in = i < ni && j < nj;
    int sat = 0, liq = 0, mix = 0, ice = 0;
    if (in) {
        const unsigned col = (unsigned)j * ni + i, plane = (unsigned)nj * ni;
        const unsigned m = (unsigned)kf * plane + col, f = m;
        NmCell up{}, lo{};
        if (kf < nk) {
            up = nm_cell(a, kf, m);
            a.qvci[m] = up.qvci;
            a.qt[m] = up.qt;
            a.temperature[m] = up.t;
            a.thv[m] = up.thv;
        }
        float value = 0.0f;
        if (kf >= 1 && kf < nk) {
            const unsigned l = m - plane;
            lo = nm_cell(a, kf - 1, l);
            const NmConsts &c = a.c;
            const float mrdz = a.rdz * a.mf[f];
            value = c.g * (logf(up.thv / lo.thv) * mrdz);
            const float w1 = a.c1[f], w2 = a.c2[f];
            const float pavg = w1 * a.prs[l] + w2 * a.prs[m];
            const float tavg = w1 * lo.t + w2 * up.t;
            const float qtavg = w1 * lo.qt + w2 * up.qt;
            const float qvciavg = w1 * lo.qvci + w2 * up.qvci;
            if (tavg >= 273.15f) {
                const float qvs = sat_liquid(pavg, tavg, c.eps);
                float ql = qvciavg - qvs;
                if (!(ql > 0.0f)) ql = 0.0f;
                if (ql > 1.0e-10f) {
                    float qv = qvciavg - ql;
                    if (!(qv > 0.0f)) qv = 0.0f;
                    value = nm_saturated(c, up, lo, tavg, qtavg, qvs, ql, 0.0f, qv, mrdz, false);
                    sat = liq = 1;
                }
            } else if (tavg <= 233.15f) {
                const float qvs = sat_ice(pavg, tavg, c.eps);
                float qi = qvciavg - qvs;
                if (!(qi > 0.0f)) qi = 0.0f;
                if (qi > 1.0e-10f) {
                    float qv = qvciavg - qi;
                    if (!(qv > 0.0f)) qv = 0.0f;
                    value = nm_saturated(c, up, lo, tavg, qtavg, qvs, 0.0f, qi, qv, mrdz, true);
                    sat = ice = 1;
                }
            } else {
                const float ff = (tavg - 233.15f) / (273.15f - 233.15f);
                const float qvsl = sat_liquid(pavg, tavg, c.eps), qvsi = sat_ice(pavg, tavg, c.eps);
                const float om = 1.0f - ff;
                const float qvs = ff * qvsl + om * qvsi;
                const float ex = qvciavg - qvs;
                float qi = om * ex;
                if (!(qi > 0.0f)) qi = 0.0f;
                float ql = ff * ex;
                if (!(ql > 0.0f)) ql = 0.0f;
                if (ql + qi > 1.0e-10f) {
                    float qv = (qvciavg - ql) - qi;
                    if (!(qv > 0.0f)) qv = 0.0f;
                    const float nml = nm_saturated(c, up, lo, tavg, qtavg, qvsl, ql, qi, qv, mrdz, false);
                    const float nmi = nm_saturated(c, up, lo, tavg, qtavg, qvsi, ql, qi, qv, mrdz, true);
                    value = ff * nml + om * nmi;
                    sat = mix = 1;
                }
            }
        }
        a.nm[f] = value;
        if (kf < nk) a.mask[m] = (uint8_t)sat;
    }
    if (a.counts != nullptr) {
        const int n0 = __syncthreads_count(sat), n1 = __syncthreads_count(liq);
        const int n2 = __syncthreads_count(mix), n3 = __syncthreads_count(ice);
        if (threadIdx.x == 0 && threadIdx.y == 0 && n0 > 0) {
            atomicAdd(&a.counts[0], (unsigned long long)n0);
            if (n1) atomicAdd(&a.counts[1], (unsigned long long)n1);
            if (n2) atomicAdd(&a.counts[2], (unsigned long long)n2);
            if (n3) atomicAdd(&a.counts[3], (unsigned long long)n3);
        }
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
// Whole columns leave a small plane too few warps; a chunk of levels forms the
// strains of the mass level below it again: halve until three rounds of the
// resident CTAs on 148 SMs, or at most eight levels, are left
// (256x256x80 terrain: 246 us with whole columns; 128x100x64 flat: 80 against 27).
template <bool FLAT>
void calcdef_launch(const DefArgs &p, cudaStream_t st) {
    const long long tiles =
        (long long)((p.ni + kDefOut - 1) / kDefOut) * ((p.nj + kDefRows - 2) / (kDefRows - 1));
    int chunk = p.nk - 1;
    while (chunk > 8 && tiles * ((p.nk - 2 + chunk) / chunk) < 3LL * 148 * (FLAT ? 4 : 3)) chunk = (chunk + 1) / 2;
    calcdef_march_kernel<FLAT><<<dim3((unsigned)tiles, (p.nk - 2 + chunk) / chunk), dim3(32, kDefRows), 0, st>>>(p, chunk);
}
}  // namespace

extern "C" int32_t gm1b_terrain_deformation(int32_t ni, int32_t nj, int32_t nk,
                                            const gm1b_deformation_arrays *arrays, float dx, float dy, float dz,
                                            void *stream) {
    if (arrays == nullptr || ni < 3 || nj < 3 || nk < 3) {
        gm1b_set_error("gm1b_terrain_deformation: need arrays and ni, nj, nk >= 3");
        return GM1B_ERR_ARGUMENT;
    }
    if (!(dx > 0.0f) || !(dy > 0.0f) || !(dz > 0.0f) || !isfinite(dx) || !isfinite(dy) || !isfinite(dz)) {
        gm1b_set_error("gm1b_terrain_deformation: dx, dy, dz must be finite and > 0");
        return GM1B_ERR_ARGUMENT;
    }
    const gm1b_deformation_arrays &s = *arrays;
    const void *need[] = {s.u3d, s.v3d, s.w3d, s.rho, s.rf, s.c1, s.c2, s.gz, s.rgz, s.rgzu, s.rgzv, s.gx, s.gy,
                          s.defv, s.defh};
    for (const void *q : need)
        if (q == nullptr) {
            gm1b_set_error("gm1b_terrain_deformation: a required array is NULL");
            return GM1B_ERR_ARGUMENT;
        }
    if ((size_t)(nk + 3) * (size_t)(nj + 7) * (size_t)(ni + 7) >= ((size_t)1 << 31)) {
        gm1b_set_error("gm1b_terrain_deformation: grid too large (the kernels index with 32-bit offsets)");
        return GM1B_ERR_ARGUMENT;
    }
    DefArgs p;
    p.u = s.u3d;
    p.v = s.v3d;
    p.w = s.w3d;
    p.rho = s.rho;
    p.rf = s.rf;
    p.c1 = s.c1;
    p.c2 = s.c2;
    p.gz = s.gz;
    p.rgz = s.rgz;
    p.rgzu = s.rgzu;
    p.rgzv = s.rgzv;
    p.gx = s.gx;
    p.gy = s.gy;
    p.defv = s.defv;
    p.defh = s.defh;
    p.ni = ni;
    p.nj = nj;
    p.nk = nk;
    p.rdx = 1.0f / dx;
    p.rdy = 1.0f / dy;
    p.rds = 1.0f / dz;
    p.zt = (float)nk * dz;
    p.dz = dz;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    ProfScope ps("calcdef_march_kernel", st);
    calcdef_launch<false>(p, st);
    ps.stop();
    return launch_ok("calcdef_march_kernel") ? GM1B_OK : GM1B_ERR_CUDA;
}

extern "C" int32_t gm1b_flat_deformation(int32_t ni, int32_t nj, int32_t nk, const gm1b_flat_deformation_arrays *arrays,
                                         float dx, float dy, float rdz, void *stream) {
    if (arrays == nullptr || ni < 3 || nj < 3 || nk < 3) {
        gm1b_set_error("gm1b_flat_deformation: need arrays and ni, nj, nk >= 3");
        return GM1B_ERR_ARGUMENT;
    }
    if (!(dx > 0.0f) || !(dy > 0.0f) || !(rdz > 0.0f) || !isfinite(dx) || !isfinite(dy) || !isfinite(rdz)) {
        gm1b_set_error("gm1b_flat_deformation: dx, dy, rdz must be finite and > 0");
        return GM1B_ERR_ARGUMENT;
    }
    const gm1b_flat_deformation_arrays &s = *arrays;
    const void *need[] = {s.u3d, s.v3d, s.w3d, s.rho, s.rf, s.mf, s.c1, s.c2, s.mh_profile, s.defv, s.defh};
    for (const void *q : need)
        if (q == nullptr) {
            gm1b_set_error("gm1b_flat_deformation: a required array is NULL");
            return GM1B_ERR_ARGUMENT;
        }
    if ((size_t)(nk + 3) * (size_t)(nj + 7) * (size_t)(ni + 7) >= ((size_t)1 << 31)) {
        gm1b_set_error("gm1b_flat_deformation: grid too large (the kernels index with 32-bit offsets)");
        return GM1B_ERR_ARGUMENT;
    }
    DefArgs p{};
    p.u = s.u3d;
    p.v = s.v3d;
    p.w = s.w3d;
    p.rho = s.rho;
    p.rf = s.rf;
    p.c1 = s.c1;
    p.c2 = s.c2;
    p.mf3 = s.mf;
    p.mhp = s.mh_profile;
    p.defv = s.defv;
    p.defh = s.defh;
    p.ni = ni;
    p.nj = nj;
    p.nk = nk;
    p.rdx = 1.0f / dx;
    p.rdy = 1.0f / dy;
    p.rdz = rdz;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    ProfScope ps("calcdef_flat_march_kernel", st);
    calcdef_launch<true>(p, st);
    ps.stop();
    return launch_ok("calcdef_flat_march_kernel") ? GM1B_OK : GM1B_ERR_CUDA;
}

extern "C" int32_t gm1b_moist_nm(int32_t ni, int32_t nj, int32_t nk, const gm1b_moist_nm_arrays *arrays, float dz,
                                 void *stream) {
    if (arrays == nullptr || ni < 1 || nj < 1 || nk < 2 || nk > 65534) {
        gm1b_set_error("gm1b_moist_nm: need arrays, ni >= 1, nj >= 1 and 2 <= nk <= 65534");
        return GM1B_ERR_ARGUMENT;
    }
    if ((size_t)(nk + 3) * (size_t)(nj + 7) * (size_t)(ni + 7) >= ((size_t)1 << 31)) {
        gm1b_set_error("gm1b_moist_nm: grid too large (the kernels index with 32-bit offsets)");
        return GM1B_ERR_ARGUMENT;
    }
    if (!(dz > 0.0f) || !isfinite(dz)) {
        gm1b_set_error("gm1b_moist_nm: dz must be finite and > 0");
        return GM1B_ERR_ARGUMENT;
    }
    const gm1b_moist_nm_arrays &s = *arrays;
    const void *need[] = {s.c1, s.c2, s.mf, s.pi0, s.th0, s.prs, s.pp3d, s.th3d, s.q3d, s.nm, s.temperature,
                          s.qt, s.thv, s.qvci, s.saturation_mask};
    for (const void *q : need)
        if (q == nullptr) {
            gm1b_set_error("gm1b_moist_nm: a required array is NULL");
            return GM1B_ERR_ARGUMENT;
        }
    NmArgs a;
    a.c1 = s.c1;
    a.c2 = s.c2;
    a.mf = s.mf;
    a.pi0 = s.pi0;
    a.th0 = s.th0;
    a.prs = s.prs;
    a.pp3d = s.pp3d;
    a.th3d = s.th3d;
    a.q3d = s.q3d;
    a.nm = s.nm;
    a.temperature = s.temperature;
    a.qt = s.qt;
    a.thv = s.thv;
    a.qvci = s.qvci;
    a.mask = s.saturation_mask;
    a.counts = reinterpret_cast<unsigned long long *>(s.counts);
    a.ni = ni;
    a.nj = nj;
    a.nk = nk;
    a.rdz = 1.0f / dz;
    // CM1 constants.F words and the derived latent-heat coefficients, formed
    // in binary32 as the reference forms them (cuda_moist_nm.py:179-204)
    volatile float rv = 461.5f, to = 273.15f;
    NmConsts &c = a.c;
    c.g = 9.81f;
    c.rd = 287.04f;
    c.cp = 1005.7f;
    c.cpv = 1870.0f;
    c.cpl = 4190.0f;
    c.cpi = 2106.0f;
    c.eps = c.rd / rv;
    c.reps = rv / c.rd;
    const float dl = c.cpl - c.cpv, di = c.cpi - c.cpv;
    const float tl = dl * to, ti = di * to;
    c.lv1 = 2501000.0f + tl;
    c.lv2 = dl;
    c.ls1 = 2834000.0f + ti;
    c.ls2 = di;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    ProfScope ps("moist_nm_kernel", st);
    moist_nm_kernel<<<dim3((ni + 31) / 32, (nj + 3) / 4, nk + 1), dim3(32, 4), 0, st>>>(a);
    ps.stop();
    return launch_ok("moist_nm_kernel") ? GM1B_OK : GM1B_ERR_CUDA;
}
