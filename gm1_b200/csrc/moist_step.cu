// moist_step.cu - sm_100a kernels that join the operators of the moist
// large step on the padded (ng = 3) open lane.
//
// Behaviour followed (reference file:line):
//   open-lateral halo fills bcp/bcs/bcu/bcv/bcw     src/cm1core/cuda_sound3_open_boundary.py:249-335
//   moist buoyancy, getdiv, getdivx                 src/cm1core/cuda_moist_stage_bridge.py:160-194 (kernel
//                                                   source), launchers :433-501
//   final-stage moisture pdef chain (WENO face fluxes, directional advection,
//   candidate/correction per direction, total)     src/cm1core/cuda_scalar_moist_rk.py:560-700 (kernel
//                                                   source), launcher :1336-1500
//   held-tendency composition                       src/cm1core/cuda_gm1_child_step_composer.py:547-556
//   solve3 density                                  src/cm1core/cuda_gm1_forecast.py:548 (gm1_solve3_density_v1)
//
// Design (B200): each piece is an elementwise or per-line pass with the
// reference's operation order; an open fill leaves in one launch the words of
// the reference's two ordered passes (first direction of the family, then
// the second), the halo corners among them.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "gm1b_common.cuh"
#include "weno.cuh"

namespace gm1b {
namespace {

bool launch_ok(const char *what) {
    const cudaError_t e = cudaPeekAtLastError();
    if (e != cudaSuccess) {
        cudaGetLastError();
        gm1b_set_error("%s: %s", what, cudaGetErrorString(e));
        return false;
    }
    return true;
}

unsigned grid_for(size_t work) {
    return (unsigned)std::max<size_t>(1, std::min<size_t>((work + 255) / 256, (size_t)148 * 16));
}

// ---------------------------------------------------------------------------
// open-lateral halo fills
// ---------------------------------------------------------------------------
struct FillGeom {
    float *q;
    int nx, ny;          // row length and rows per level
    int g;               // halo width (3 on the padded lane, 1 for the pressure family)
    int x0, xl, y0, yl;  // first and last live column / row
    int k0, k1;          // levels filled
    int ew_first;        // west/east pass first (all but bcv)
    int zero_w;          // bcw flag 1: zero levels 1 and nk+1 over rows y0-1..yl+1, columns x0-1..xl+1
    int nk;
};

// The reference fills in two ordered passes: the family's first direction
// over the rows (columns) y0-1..yl+1, then the second.  One launch leaves the
// same words: every halo word is a live edge word of its row or column (the
// diagonal words of the first ring: of the corner cell), except the words
// beyond the first ring beside a first-ring corner, which the first pass
// copies from the halo word the second pass then overwrites; the thread that
// overwrites it copies it first.
__device__ __forceinline__ void fill_word(const FillGeom &f, unsigned z) {
    const unsigned w = (unsigned)(f.xl - f.x0 + 1), h = (unsigned)(f.yl - f.y0 + 1), g2 = 2u * f.g;
    const unsigned na = h * g2, nb = w * g2, per = na + nb + 2 * g2;
    unsigned r = z % per;
    float *lev = f.q + ((unsigned)f.k0 + z / per) * (unsigned)f.ny * (unsigned)f.nx;
    auto word = [&](int y, int x) -> float & { return lev[(unsigned)y * (unsigned)f.nx + (unsigned)x]; };
    auto halo_x = [&](int q) { return q < f.g ? f.x0 - f.g + q : f.xl + 1 + q - f.g; };
    auto halo_y = [&](int q) { return q < f.g ? f.y0 - f.g + q : f.yl + 1 + q - f.g; };
    if (r < na) {  // west and east of the live rows
        const int q = (int)(r % g2), y = f.y0 + (int)(r / g2), x = halo_x(q);
        if (!f.ew_first && (x == f.x0 - 1 || x == f.xl + 1) && (y == f.y0 || y == f.yl)) {
            const float old = word(y, x);
            for (int t = 2; t <= f.g; ++t) {
                if (y == f.y0) word(f.y0 - t, x) = old;
                if (y == f.yl) word(f.yl + t, x) = old;
            }
        }
        word(y, x) = word(y, q < f.g ? f.x0 : f.xl);
        return;
    }
    r -= na;
    if (r < nb) {  // south and north of the live columns
        const int q = (int)(r / w), x = f.x0 + (int)(r % w), y = halo_y(q);
        if (f.ew_first && (y == f.y0 - 1 || y == f.yl + 1) && (x == f.x0 || x == f.xl)) {
            const float old = word(y, x);
            for (int t = 2; t <= f.g; ++t) {
                if (x == f.x0) word(y, f.x0 - t) = old;
                if (x == f.xl) word(y, f.xl + t) = old;
            }
        }
        word(y, x) = word(q < f.g ? f.y0 : f.yl, x);
        return;
    }
    r -= nb;  // beside the corners: the second direction's halo of the first ring
    const int q = (int)(r / 2);
    const bool hi = r % 2 != 0;
    if (f.ew_first)
        word(halo_y(q), hi ? f.xl + 1 : f.x0 - 1) = word(q < f.g ? f.y0 : f.yl, hi ? f.xl : f.x0);
    else
        word(hi ? f.yl + 1 : f.y0 - 1, halo_x(q)) = word(hi ? f.yl : f.y0, q < f.g ? f.x0 : f.xl);
}

constexpr int kMostFills = 4;
struct Fills {
    FillGeom f[kMostFills];
    unsigned words[kMostFills];  // fill_word's of each
    int n;
};

__global__ void __launch_bounds__(256) open_fill_kernel(const __grid_constant__ Fills a) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
    for (int q = 0; q < a.n; ++q) {
        const FillGeom &f = a.f[q];
        for (unsigned z = t; z < a.words[q]; z += step) fill_word(f, z);
        if (f.zero_w) {
            const unsigned rows = (unsigned)(f.yl - f.y0 + 3), cols = (unsigned)(f.xl - f.x0 + 3);
            for (unsigned z = t; z < 2 * rows * cols; z += step) {
                const int x = f.x0 - 1 + (int)(z % cols);
                const int y = f.y0 - 1 + (int)((z / cols) % rows);
                const int k = z / (rows * cols) == 0 ? 1 : f.nk + 1;
                f.q[((unsigned)k * (unsigned)f.ny + (unsigned)y) * (unsigned)f.nx + (unsigned)x] = 0.0f;
            }
        }
    }
}

// theta (th0 - 300 + th3d) and the moisture rows into their padded arrays,
// the halos of levels 1..nk as the open scalar fill leaves them (fill_word's,
// the words beyond the first ring beside its corners among them), one launch
struct PackScalars {
    const float *th0, *scalar[4];  // th3d, then the moisture rows
    float *padded[4];
};

__global__ void __launch_bounds__(256) pack_scalars_kernel(const __grid_constant__ PackScalars a, int ni, int nj) {
    const int x = blockIdx.x * 32 + threadIdx.x, y = blockIdx.y * 8 + threadIdx.y, k = blockIdx.z;
    const int px = ni + 6, py = nj + 6;
    if (x >= px || y >= py) return;
    if ((y < 3 || y > nj + 2) && (x < 2 || x > ni + 3)) return;  // left alone, or a first-ring thread's below
    const unsigned c = ((unsigned)k * nj + (unsigned)(min(max(y, 3), nj + 2) - 3)) * (unsigned)ni +
                       (unsigned)(min(max(x, 3), ni + 2) - 3);
    const unsigned d = ((unsigned)(k + 1) * py + y) * (unsigned)px + x;
    float v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = __ldg(a.scalar[q] + c);
    if ((y == 2 || y == nj + 3) && (x == 3 || x == ni + 2)) {
        // the west/east pass copied this word outward before the other overwrote it
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float old = a.padded[q][d];
            if (x == 3) a.padded[q][d - 2] = a.padded[q][d - 3] = old;
            if (x == ni + 2) a.padded[q][d + 2] = a.padded[q][d + 3] = old;
        }
    }
    const float base = __ldg(a.th0 + k) - 300.0f;
    a.padded[0][d] = base + v[0];
#pragma unroll
    for (int q = 1; q < 4; ++q) a.padded[q][d] = v[q];
}

bool fill_geometry(int kind, int ni, int nj, int nk, float *q, FillGeom &f) {
    f = FillGeom{};
    f.q = q;
    f.nk = nk;
    f.k0 = 1;
    f.k1 = nk;
    f.ew_first = 1;
    switch (kind) {
        case GM1B_FILL_PRESSURE:
            f.nx = ni + 2, f.ny = nj + 2, f.g = 1, f.x0 = 1, f.xl = ni, f.y0 = 1, f.yl = nj;
            return true;
        case GM1B_FILL_SCALAR:
            f.nx = ni + 6, f.ny = nj + 6, f.g = 3, f.x0 = 3, f.xl = ni + 2, f.y0 = 3, f.yl = nj + 2;
            return true;
        case GM1B_FILL_U:
            f.nx = ni + 7, f.ny = nj + 6, f.g = 3, f.x0 = 3, f.xl = ni + 3, f.y0 = 3, f.yl = nj + 2;
            return true;
        case GM1B_FILL_V:
            f.nx = ni + 6, f.ny = nj + 7, f.g = 3, f.x0 = 3, f.xl = ni + 2, f.y0 = 3, f.yl = nj + 3;
            f.ew_first = 0;
            return true;
        case GM1B_FILL_W:
        case GM1B_FILL_W_KEEP_ENDS:
            f.nx = ni + 6, f.ny = nj + 6, f.g = 3, f.x0 = 3, f.xl = ni + 2, f.y0 = 3, f.yl = nj + 2;
            f.k0 = 2;
            f.zero_w = kind == GM1B_FILL_W;
            return true;
        default:
            return false;
    }
}

// ---------------------------------------------------------------------------
// moist stage bridge
// ---------------------------------------------------------------------------
struct Lane {
    int ni, nj, nk;
    __device__ __forceinline__ unsigned s(int k, int y, int x) const {  // scalar / w layout, padded coordinates
        return ((unsigned)k * (nj + 6) + y) * (unsigned)(ni + 6) + x;
    }
    __device__ __forceinline__ unsigned u(int k, int y, int x) const {
        return ((unsigned)k * (nj + 6) + y) * (unsigned)(ni + 7) + x;
    }
    __device__ __forceinline__ unsigned v(int k, int y, int x) const {
        return ((unsigned)k * (nj + 7) + y) * (unsigned)(ni + 6) + x;
    }
    __device__ __forceinline__ unsigned m(int k0, int j0, int i0) const {
        return ((unsigned)k0 * nj + j0) * (unsigned)ni + i0;
    }
};

// dum8 on w levels, c1(kf) dum8(kf-1) + c2(kf) dum8(kf) (zero at the ends),
// into wten, and on a terrain column its slope part into uten and vten.  A
// thread owns the w point, west face and south face of a cell and marches a
// chunk of levels with the three columns' face words carried up.  Bound by
// memory.  A thread per w point, u face and v face formed each face word up to
// six times: 256x256x80 121 -> 68 us, 640x768x80 flat 174 -> 136.
// Inputs and the three tendencies are distinct arrays (the entry point
// refuses a call that passes one array twice), so every load may be issued
// ahead of the stores.
template <bool W_ONLY, int W>
__global__ void __launch_bounds__(256) msb_buoyancy_kernel(const float *__restrict__ dum8,
                                                          const float *__restrict__ c1, const float *__restrict__ c2,
                                                          const float *__restrict__ gxu,
                                                          const float *__restrict__ gyv, float *__restrict__ uten,
                                                          float *__restrict__ vten, float *__restrict__ wten, Lane L,
                                                          int chunk) {
    const int ni = L.ni, nj = L.nj, nk = L.nk, tiles = (ni + W - 1) / W;
    const int i = blockIdx.x % tiles * W + threadIdx.x, j = blockIdx.x / tiles * (256 / W) + threadIdx.y;
    if (i >= ni || j >= nj) return;
    const bool du = !W_ONLY && i > 0, dv = !W_ONLY && j > 0;
    const int iw = du ? i - 1 : i, js = dv ? j - 1 : j;  // neighbour cells (the own one when unused)
    const int k_lo = 1 + blockIdx.y * chunk, k_hi = min(nk, k_lo + chunk - 1);
    auto d8 = [&](int k, int jj, int ii) { return dum8[L.s(k, jj + 3, ii + 3)]; };
    auto face = [&](int kf, int jj, int ii, float below, float above) {
        if (kf == 1 || kf == nk + 1) return 0.0f;
        const unsigned p = L.m(kf - 1, jj, ii);
        return c1[p] * below + c2[p] * above;
    };
    float dc = d8(k_lo, j, i), dw = 0.0f, ds = 0.0f;
    float fc = k_lo == 1 ? 0.0f : face(k_lo, j, i, d8(k_lo - 1, j, i), dc), fw = 0.0f, fs = 0.0f, gx = 0.0f, gy = 0.0f;
    if (!W_ONLY) {
        dw = d8(k_lo, j, iw), ds = d8(k_lo, js, i);
        if (k_lo > 1) {
            fw = face(k_lo, j, iw, d8(k_lo - 1, j, iw), dw);
            fs = face(k_lo, js, i, d8(k_lo - 1, js, i), ds);
        }
        gx = gxu[((unsigned)(k_lo - 1) * nj + j) * (ni + 1) + i];
        gy = gyv[((unsigned)(k_lo - 1) * (nj + 1) + j) * ni + i];
    }
#pragma unroll(W_ONLY ? 4 : 1)
    for (int k = k_lo; k <= k_hi; ++k) {
        const bool more = k < nk;
        const float ndc = more ? d8(k + 1, j, i) : 0.0f;
        const float nfc = face(k + 1, j, i, dc, ndc);
        if (k >= 2) {
            const unsigned d = L.s(k, j + 3, i + 3);
            wten[d] = wten[d] + fc;
        }
        if (!W_ONLY) {
            const float ndw = more ? d8(k + 1, j, iw) : 0.0f, nds = more ? d8(k + 1, js, i) : 0.0f;
            const float nfw = face(k + 1, j, iw, dw, ndw), nfs = face(k + 1, js, i, ds, nds);
            const float ngx = gxu[((unsigned)k * nj + j) * (ni + 1) + i], ngy = gyv[((unsigned)k * (nj + 1) + j) * ni + i];
            if (du) {
                float t = 0.125f * ((nfc + nfw) + (fc + fw));
                t = t - 0.25f * (dc + dw);
                t = t * (gx + ngx);
                const unsigned d = L.u(k, j + 3, i + 3);
                uten[d] = uten[d] + t;
            }
            if (dv) {
                float t = 0.125f * ((nfc + nfs) + (fc + fs));
                t = t - 0.25f * (dc + ds);
                t = t * (gy + ngy);
                const unsigned d = L.v(k, j + 3, i + 3);
                vten[d] = vten[d] + t;
            }
            dw = ndw, ds = nds, fw = nfw, fs = nfs, gx = ngx, gy = ngy;
        }
        dc = ndc, fc = nfc;
    }
}

struct Getdiv {
    const float *rru, *rrv, *rrw, *rgzu, *rgzv, *dzdx, *dzdy, *gz, *thterm;
    float *div, *theta_div;
    float rdx, rdy, rdsf, dz, zt, rzt;
    // vertical column: 0 uniform; 1 terrain branch on a stretched column
    // (sigma/sigmaf/rds/rdsf, physical top zt); 2 flat column (rdz*mh, no
    // terrain w, no rgzu/rgzv) - cuda_gm1_child_stretched_moist.py:35-110
    int vmode;
    const float *sigma, *sigmaf, *rds, *rdsfp, *mh;
    float rdzm;
};

// The terrain column's vertical weights at w level kf: r1, r2 halved, and the
// height above the top.
struct SlopeWeights {
    float r1, r2, height;
};
__device__ __forceinline__ SlopeWeights slope_weights(bool pr, int kf, float dz, float rdz, float zt,
                                                      const float *sigma, const float *sigmaf, const float *rds) {
    const float sf = pr ? sigmaf[kf] : (float)(kf - 1) * dz, sm = pr ? sigma[kf - 1] : ((float)(kf - 1) - 0.5f) * dz;
    const float r2 = (sf - sm) * (pr ? rds[kf] : rdz);
    return {0.5f * (1.0f - r2), 0.5f * r2, sf - zt};
}

// getdiv on a terrain column (vmode 0 and 1).  A thread marches a chunk of a
// column's levels with the face terms and the transformed w of the level below
// carried up.  Bound by memory; 256x256x80: a thread per cell 86 us, 45 here
// (two levels a thread 58).
template <int VM, int W>
__global__ void __launch_bounds__(256) msb_getdiv_kernel(const __grid_constant__ Getdiv a, Lane L, int chunk) {
    const int ni = L.ni, nj = L.nj, nk = L.nk, tiles = (ni + W - 1) / W;
    const int i = blockIdx.x % tiles * W + threadIdx.x, j = blockIdx.x / tiles * (256 / W) + threadIdx.y;
    if (i >= ni || j >= nj) return;
    const unsigned c2d = (unsigned)j * ni + i, u2d = (unsigned)j * (ni + 1) + i;
    const float gu0 = a.rgzu[u2d], gu1 = a.rgzu[u2d + 1], gv0 = a.rgzv[c2d], gv1 = a.rgzv[c2d + ni];
    const float dzdx = a.dzdx[c2d], dzdy = a.dzdy[c2d], gz = a.gz[c2d], rzt = 1.0f / a.zt, rdz = 1.0f / a.dz;
    const int k_lo = 1 + blockIdx.y * chunk, k_hi = min(nk, k_lo + chunk - 1);
    struct Faces {
        float u0, u1, v0, v1;
    };
    auto faces = [&](int k) {
        const unsigned u = L.u(k, j + 3, i + 3), v = L.v(k, j + 3, i + 3);
        return Faces{__ldg(a.rru + u) * gu0, __ldg(a.rru + u + 1) * gu1, __ldg(a.rrv + v) * gv0,
                     __ldg(a.rrv + v + (unsigned)(ni + 6)) * gv1};
    };
    auto wt = [&](int kf, const Faces &h, const Faces &l) {  // transformed w at levels 2..nk
        const SlopeWeights s = slope_weights(VM == 1, kf, a.dz, rdz, a.zt, a.sigma, a.sigmaf, a.rds);
        const float ux = s.r2 * (h.u0 + h.u1) + s.r1 * (l.u0 + l.u1);
        const float vy = s.r2 * (h.v0 + h.v1) + s.r1 * (l.v0 + l.v1);
        float terrain = ux * dzdx + vy * dzdy;
        terrain = ((terrain * s.height) * gz) * rzt;
        return __ldg(a.rrw + L.s(kf, j + 3, i + 3)) + terrain;
    };
    Faces cur = faces(k_lo);
    float lo = k_lo == 1 ? 0.0f : wt(k_lo, cur, faces(k_lo - 1));
#pragma unroll 2
    for (int k = k_lo; k <= k_hi; ++k) {
        const Faces next = k < nk ? faces(k + 1) : cur;
        const float hi = k < nk ? wt(k + 1, next, cur) : 0.0f;
        const unsigned z = L.m(k - 1, j, i);
        const float th = __ldg(a.thterm + z);
        float d = (cur.u1 - cur.u0) * a.rdx + (cur.v1 - cur.v0) * a.rdy;
        d = d + (hi - lo) * (VM == 1 ? a.rdsfp[k] : a.rdsf);
        if (fabsf(d) < 1.0e-20f) d = 0.0f;
        a.div[z] = d;
        a.theta_div[z] = d * th;
        cur = next, lo = hi;
    }
}

// the terrain column's horizontal mass fluxes in place (vmode 1: base density
// from the padded rho0p)
template <int W>
__global__ void __launch_bounds__(256) msb_getdivx_horizontal_kernel(const float *__restrict__ rho0,
                                                                    const float *__restrict__ rgzu,
                                                                    const float *__restrict__ rgzv,
                                                                    float *__restrict__ rru, float *__restrict__ rrv,
                                                                    Lane L, int vmode,
                                                                    const float *__restrict__ rho0p, int chunk) {
    const int ni = L.ni, nj = L.nj, nk = L.nk, tiles = ni / W + 1;
    const int x = blockIdx.x % tiles * W + threadIdx.x, y = blockIdx.x / tiles * (256 / W) + threadIdx.y;
    if (x > ni || y > nj) return;
    const bool du = y < nj, dv = x < ni;
    const int xl = max(x - 1, 0), xr = min(x, ni - 1), yl = max(y - 1, 0), yr = min(y, nj - 1);
    const float gu = du ? rgzu[(unsigned)y * (ni + 1) + x] : 0.0f, gv = dv ? rgzv[(unsigned)y * ni + x] : 0.0f;
    const int k_lo = 1 + blockIdx.y * chunk, k_hi = min(nk, k_lo + chunk - 1);
#pragma unroll 4
    for (int k = k_lo; k <= k_hi; ++k) {
        const unsigned u = L.u(k, y + 3, x + 3), v = L.v(k, y + 3, x + 3), s = L.s(k, y + 3, x + 3);
        if (du) {
            const float den = vmode == 1 ? 0.5f * (rho0p[s - 1] + rho0p[s])
                                         : 0.5f * (rho0[L.m(k - 1, y, xl)] + rho0[L.m(k - 1, y, xr)]);
            rru[u] = (den * rru[u]) * gu;
        }
        if (dv) {
            const float den = vmode == 1 ? 0.5f * (rho0p[s - (unsigned)(ni + 6)] + rho0p[s])
                                         : 0.5f * (rho0[L.m(k - 1, yl, x)] + rho0[L.m(k - 1, yr, x)]);
            rrv[v] = (den * rrv[v]) * gv;
        }
    }
}

// the terrain column's vertical mass flux in place, from the horizontal ones;
// a thread marches a chunk of levels with the sums of the level below carried up
template <int W>
__global__ void __launch_bounds__(256) msb_getdivx_vertical_kernel(const float *__restrict__ rf0, const float *dzdx,
                                                                  const float *dzdy, const float *gz,
                                                                  const float *__restrict__ rru,
                                                                  const float *__restrict__ rrv,
                                                                  float *__restrict__ rrw, float dz, Lane L, int vmode,
                                                                  const float *__restrict__ sigma,
                                                                  const float *__restrict__ sigmaf,
                                                                  const float *__restrict__ rdsp, float ztop,
                                                                  int chunk) {
    const int ni = L.ni, nj = L.nj, nk = L.nk, tiles = (ni + W - 1) / W;
    const int i = blockIdx.x % tiles * W + threadIdx.x, j = blockIdx.x / tiles * (256 / W) + threadIdx.y;
    if (i >= ni || j >= nj) return;
    const bool pr = vmode == 1;
    const float rds = 1.0f / dz, zt = pr ? ztop : (float)nk * dz, rzt = 1.0f / zt;
    const unsigned c2d = (unsigned)j * ni + i;
    const float dx2 = dzdx[c2d], dy2 = dzdy[c2d], g = gz[c2d];
    const int k_lo = 2 + blockIdx.y * chunk, k_hi = min(nk, k_lo + chunk - 1);
    if (blockIdx.y == 0) rrw[L.s(1, j + 3, i + 3)] = rrw[L.s(nk + 1, j + 3, i + 3)] = 0.0f;
    auto us = [&](int k) {
        const unsigned u = L.u(k, j + 3, i + 3);
        return rru[u] + rru[u + 1];
    };
    auto vs = [&](int k) {
        const unsigned v = L.v(k, j + 3, i + 3);
        return rrv[v] + rrv[v + (unsigned)(ni + 6)];
    };
    float ul = us(k_lo - 1), vl = vs(k_lo - 1);
#pragma unroll 2
    for (int k = k_lo; k <= k_hi; ++k) {
        const SlopeWeights s = slope_weights(pr, k, dz, rds, zt, sigma, sigmaf, rdsp);
        const float uh = us(k), vh = vs(k);
        const float ux = s.r2 * uh + s.r1 * ul, vy = s.r2 * vh + s.r1 * vl;
        float terrain = ux * dx2 + vy * dy2;
        terrain = ((terrain * s.height) * g) * rzt;
        const unsigned p = L.s(k, j + 3, i + 3);
        rrw[p] = rf0[L.m(k - 1, j, i)] * rrw[p] + terrain;
        ul = uh, vl = vh;
    }
}

// The flat column's getdiv and getdivx divergences together, from the
// averaged velocities before they are scaled to mass fluxes: seven words a
// cell instead of ten in two passes.
__global__ void __launch_bounds__(256) msb_flat_divergences_kernel(Getdiv a, const float *rho0p, const float *rf0,
                                                                   float *divx, Lane L) {
    // all tiles of a level in one grid dimension, which takes any plane
    const int tiles = (L.ni + 31) / 32;
    const int i = blockIdx.x % tiles * 32 + threadIdx.x, j = blockIdx.x / tiles * 8 + threadIdx.y;
    if (i >= L.ni || j >= L.nj) return;
    for (int k = blockIdx.y + 1; k <= L.nk; k += gridDim.y) {
        const unsigned z = L.m(k - 1, j, i), u = L.u(k, j + 3, i + 3), v = L.v(k, j + 3, i + 3), w = L.s(k, j + 3, i + 3);
        const float u0 = a.rru[u], u1 = a.rru[u + 1], v0 = a.rrv[v], v1 = a.rrv[v + (unsigned)(L.ni + 6)];
        const float w0 = k == 1 ? 0.0f : a.rrw[w];
        const float w1 = k == L.nk ? 0.0f : a.rrw[w + (unsigned)(L.nj + 6) * (unsigned)(L.ni + 6)];
        const float mh = a.mh[k], r = rho0p[L.s(k, 3, 3)];
        float d = (u1 - u0) * a.rdx + (v1 - v0) * a.rdy;
        d = d + ((w1 - w0) * a.rdzm) * mh;
        if (fabsf(d) < 1.0e-30f) d = 0.0f;
        a.div[z] = d;
        a.theta_div[z] = d * a.thterm[z];
        const float m0 = k == 1 ? 0.0f : w0 * rf0[L.m(k - 1, 0, 0)], m1 = k == L.nk ? 0.0f : w1 * rf0[L.m(k, 0, 0)];
        d = (u1 * r - u0 * r) * a.rdx + (v1 * r - v0 * r) * a.rdy;
        d = d + ((m1 - m0) * a.rdzm) * mh;
        divx[z] = fabsf(d) < 1.0e-30f ? 0.0f : d;
    }
}

// the flat column's mass fluxes in place: rho0(1,1,k) u, rho0(1,1,k) v,
// rf0(1,1,k) w with the two end levels of w zero
__global__ void __launch_bounds__(256) msb_flat_mass_kernel(const float *rho0p, const float *rf0, float *rru, float *rrv,
                                                            float *rrw, Lane L) {
    const int ni = L.ni, nj = L.nj, nk = L.nk, tiles = ni / 32 + 1;
    const int x = blockIdx.x % tiles * 32 + threadIdx.x, y = blockIdx.x / tiles * 8 + threadIdx.y;
    if (x > ni || y > nj) return;
    for (int k = blockIdx.y + 1; k <= nk + 1; k += gridDim.y) {
        const unsigned u = L.u(k, y + 3, x + 3), v = L.v(k, y + 3, x + 3), w = L.s(k, y + 3, x + 3);
        const bool du = k <= nk && y < nj, dv = k <= nk && x < ni, dw = x < ni && y < nj, end = k == 1 || k == nk + 1;
        const float r = k <= nk ? rho0p[L.s(k, 3, 3)] : 0.0f, rf = end ? 0.0f : rf0[L.m(k - 1, 0, 0)];
        const float fu = du ? rru[u] : 0.0f, fv = dv ? rrv[v] : 0.0f, fw = dw && !end ? rrw[w] : 0.0f;
        if (du) rru[u] = fu * r;
        if (dv) rrv[v] = fv * r;
        if (dw) rrw[w] = end ? 0.0f : fw * rf;
    }
}

template <int W>
__global__ void __launch_bounds__(256) msb_getdivx_divergence_kernel(const float *__restrict__ rru,
                                                                    const float *__restrict__ rrv,
                                                                    const float *__restrict__ rrw,
                                                                    float *__restrict__ divx, float rdx, float rdy,
                                                                    float rdsf, Lane L, int vmode,
                                                                    const float *__restrict__ rdsfp, int chunk) {
    const int ni = L.ni, nj = L.nj, nk = L.nk, tiles = (ni + W - 1) / W;
    const int i = blockIdx.x % tiles * W + threadIdx.x, j = blockIdx.x / tiles * (256 / W) + threadIdx.y;
    if (i >= ni || j >= nj) return;
    const int k_lo = 1 + blockIdx.y * chunk, k_hi = min(nk, k_lo + chunk - 1);
    float lo = rrw[L.s(k_lo, j + 3, i + 3)];
#pragma unroll 4
    for (int k = k_lo; k <= k_hi; ++k) {
        const unsigned u = L.u(k, j + 3, i + 3), v = L.v(k, j + 3, i + 3);
        const float hi = rrw[L.s(k + 1, j + 3, i + 3)];
        float d = (rru[u + 1] - rru[u]) * rdx + (rrv[v + (unsigned)(ni + 6)] - rrv[v]) * rdy;
        d = d + (hi - lo) * (vmode == 1 ? rdsfp[k] : rdsf);
        divx[L.m(k - 1, j, i)] = fabsf(d) < 1.0e-20f ? 0.0f : d;
        lo = hi;
    }
}

// ---------------------------------------------------------------------------
// final-stage moisture pdef chain
// ---------------------------------------------------------------------------
__device__ __forceinline__ float max5abs(float a, float b, float c, float d, float e) {
    return fmaxf(fmaxf(fabsf(a), fabsf(b)), fmaxf(fabsf(c), fmaxf(fabsf(d), fabsf(e))));
}
__device__ __forceinline__ unsigned obc_side(unsigned obc, unsigned side) { return (obc >> (4u * side)) & 15u; }
__device__ __forceinline__ bool obc_owned(int i, int j, int ni, int nj, unsigned obc) {
    return obc != 0u || (i >= 3 && i + 3 < ni && j >= 3 && j + 3 < nj);
}
__device__ __forceinline__ bool inflow_lo(int i, unsigned obc, unsigned side, float m) {
    return i == 0 && obc_side(obc, side) == 2u && m >= 0.0f;
}
__device__ __forceinline__ bool inflow_hi(int i, int n, unsigned obc, unsigned side, float m) {
    return i + 1 == n && obc_side(obc, side) == 2u && m <= 0.0f;
}
// pdef.F:125-166 on a whole row: cell c in [-2, n+1] as bcs fills it (1 periodic, 2 zero gradient, 3/4 mirror)
__device__ __forceinline__ long long pdef_cell(long long c, long long n, unsigned lo, unsigned hi) {
    if (c < 0) {
        if (lo == 1u) return c + n;
        if (lo == 2u) return 0;
        return -c - 1;
    }
    if (c >= n) {
        if (hi == 1u) return c - n;
        if (hi == 2u) return n - 1;
        return 2 * n - 1 - c;
    }
    return c;
}
__device__ __forceinline__ float pdef_at(const float *d, long long base, long long stride, long long c, long long n,
                                         unsigned lo, unsigned hi) {
    return d[base + pdef_cell(c, n, lo, hi) * stride];
}
__device__ __forceinline__ float pdef_ratio(const float *d, long long base, long long stride, long long c, long long n,
                                            unsigned lo, unsigned hi) {
    const float v = pdef_at(d, base, stride, c, n, lo, hi);
    if (v >= 0.0f) return 0.0f;
    const float f1 = fmaxf(0.0f, pdef_at(d, base, stride, c - 1, n, lo, hi));
    const float f2 = fmaxf(0.0f, pdef_at(d, base, stride, c + 1, n, lo, hi));
    const float sum = f1 + f2;
    return sum > 1.0e-30f ? fmaxf(v, -sum) / sum : 0.0f;
}
__device__ __forceinline__ void pdef_row_mass(const float *d, long long base, long long stride, long long c,
                                              long long n, unsigned lo, unsigned hi, float *mass, bool *flag) {
    const float v = pdef_at(d, base, stride, c, n, lo, hi);
    if (v < 0.0f) {
        const float r = pdef_ratio(d, base, stride, c, n, lo, hi);
        if (r != 0.0f) {
            const float sum = fmaxf(0.0f, pdef_at(d, base, stride, c - 1, n, lo, hi)) +
                              fmaxf(0.0f, pdef_at(d, base, stride, c + 1, n, lo, hi));
            *mass = 0.0f - sum * r;
            *flag = true;
        }
    } else if (v > 1.0e-30f) {
        const float rl = pdef_ratio(d, base, stride, c - 1, n, lo, hi);
        const float rr = pdef_ratio(d, base, stride, c + 1, n, lo, hi);
        if (rl != 0.0f) {
            *mass = *mass + v * rl;
            *flag = true;
        }
        if (rr != 0.0f) {
            *mass = *mass + v * rr;
            *flag = true;
        }
    }
}
// interior-only repair row (tile-local launch, obc = 0)
__device__ __forceinline__ float ratio1(const float *d, long long c, long long lo, long long hi, long long stride) {
    if (c <= lo || c >= hi || d[c] >= 0.0f) return 0.0f;
    const float f1 = fmaxf(0.0f, d[c - stride]), f2 = fmaxf(0.0f, d[c + stride]);
    const float sum = f1 + f2;
    return sum > 1.0e-30f ? fmaxf(d[c], -sum) / sum : 0.0f;
}

struct Pdef {
    const float *a;      // moisture at the stage's A level, compact
    const float *s;      // the advected moisture, padded scalar layout
    const float *rho0, *gz, *rgz, *rr0, *c1, *c2, *divx;
    const float *rru, *rrv, *rrw;
    float *fx, *fy, *fz;  // face fluxes (u, v, w layouts)
    float *ax, *ay, *az, *dum, *adv;  // compact
    float dt, dx, dy, dz, rdx, rdy, rdz, rdt;
    double weps;
    unsigned obc;
    int pdefweno;
    // vertical column: 0 uniform (rdz = 1/dz); 1 terrain branch, rdsf(k);
    // 2 flat column, (x*rdz)*mh(k) with the column's rho0(k) / rr0(k) and no
    // gz or rgz (cuda_gm1_child_stretched_scalar.py:160-255, :355-470)
    int vmode;
    const float *rdsf, *mh;
};

__device__ __forceinline__ float pdef_zterm(const Pdef &p, float x, int k) {
    if (p.vmode == 2) return (x * p.rdz) * __ldg(p.mh + k);
    return x * (p.vmode == 1 ? __ldg(p.rdsf + k) : p.rdz);
}

__global__ void __launch_bounds__(256) pdef_horizontal_flux_kernel(Pdef p, Lane L) {
    const int ni = L.ni, nj = L.nj;
    const unsigned n = (unsigned)L.nk * (nj + 1) * (ni + 1);
    for (unsigned q = (unsigned)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (unsigned)gridDim.x * blockDim.x) {
        const int i = (int)(q % (ni + 1)), j = (int)((q / (ni + 1)) % (nj + 1)), k = (int)(q / ((unsigned)(ni + 1) * (nj + 1))) + 1;
        const int x = i + 3, y = j + 3;
        if (j < nj) {
            const float m = p.rru[L.u(k, y, x)];
            float s1, s2, s3, s4, s5;
            if (m >= 0.0f) {
                s1 = p.s[L.s(k, y, x - 3)], s2 = p.s[L.s(k, y, x - 2)], s3 = p.s[L.s(k, y, x - 1)];
                s4 = p.s[L.s(k, y, x)], s5 = p.s[L.s(k, y, x + 1)];
            } else {
                s1 = p.s[L.s(k, y, x + 2)], s2 = p.s[L.s(k, y, x + 1)], s3 = p.s[L.s(k, y, x)];
                s4 = p.s[L.s(k, y, x - 1)], s5 = p.s[L.s(k, y, x - 2)];
            }
            p.fx[L.u(k, y, x)] = (double)max5abs(s1, s2, s3, s4, s5) > p.weps ? m * weno5(s1, s2, s3, s4, s5, p.weps) : 0.0f;
        }
        if (i < ni) {
            const float m = p.rrv[L.v(k, y, x)];
            float s1, s2, s3, s4, s5;
            if (m >= 0.0f) {
                s1 = p.s[L.s(k, y - 3, x)], s2 = p.s[L.s(k, y - 2, x)], s3 = p.s[L.s(k, y - 1, x)];
                s4 = p.s[L.s(k, y, x)], s5 = p.s[L.s(k, y + 1, x)];
            } else {
                s1 = p.s[L.s(k, y + 2, x)], s2 = p.s[L.s(k, y + 1, x)], s3 = p.s[L.s(k, y, x)];
                s4 = p.s[L.s(k, y - 1, x)], s5 = p.s[L.s(k, y - 2, x)];
            }
            p.fy[L.v(k, y, x)] = (double)max5abs(s1, s2, s3, s4, s5) > p.weps ? m * weno5(s1, s2, s3, s4, s5, p.weps) : 0.0f;
        }
    }
}

__global__ void __launch_bounds__(256) pdef_vertical_flux_kernel(Pdef p, Lane L) {
    const int ni = L.ni, nj = L.nj, nk = L.nk;
    const unsigned n = (unsigned)(nk - 1) * nj * ni;
    const float ew = (float)p.weps;
    for (unsigned q = (unsigned)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (unsigned)gridDim.x * blockDim.x) {
        const int i = (int)(q % ni), j = (int)((q / ni) % nj), k = (int)(q / ((unsigned)ni * nj)) + 2;
        const int x = i + 3, y = j + 3;
        const float m = p.rrw[L.s(k, y, x)];
        const unsigned cm = ((unsigned)(k - 1) * nj + j) * ni + i;
        float r;
        if (k == 2) {
            r = m >= 0.0f ? p.c1[cm] * p.s[L.s(k - 1, y, x)] + p.c2[cm] * p.s[L.s(k, y, x)]
                          : upstrpd(p.s[L.s(k + 1, y, x)], p.s[L.s(k, y, x)], p.s[L.s(k - 1, y, x)], ew);
        } else if (k == nk) {
            r = m > 0.0f ? upstrpd(p.s[L.s(k - 2, y, x)], p.s[L.s(k - 1, y, x)], p.s[L.s(k, y, x)], ew)
                         : p.c1[cm] * p.s[L.s(k - 1, y, x)] + p.c2[cm] * p.s[L.s(k, y, x)];
        } else {
            const bool low = (k == 3 && (p.pdefweno ? m > 0.0f : m >= 0.0f)) || (k == nk - 1 && m < 0.0f);
            if (low) {
                r = k == 3 ? upstrpd(p.s[L.s(k - 2, y, x)], p.s[L.s(k - 1, y, x)], p.s[L.s(k, y, x)], ew)
                           : upstrpd(p.s[L.s(k + 1, y, x)], p.s[L.s(k, y, x)], p.s[L.s(k - 1, y, x)], ew);
            } else {
                float s1, s2, s3, s4, s5;
                if (m >= 0.0f) {
                    s1 = p.s[L.s(k - 3, y, x)], s2 = p.s[L.s(k - 2, y, x)], s3 = p.s[L.s(k - 1, y, x)];
                    s4 = p.s[L.s(k, y, x)], s5 = p.s[L.s(k + 1, y, x)];
                } else {
                    s1 = p.s[L.s(k + 2, y, x)], s2 = p.s[L.s(k + 1, y, x)], s3 = p.s[L.s(k, y, x)];
                    s4 = p.s[L.s(k - 1, y, x)], s5 = p.s[L.s(k - 2, y, x)];
                }
                if (p.pdefweno && (double)max5abs(s1, s2, s3, s4, s5) <= p.weps) {
                    p.fz[L.s(k, y, x)] = 0.0f;
                    continue;
                }
                r = weno5(s1, s2, s3, s4, s5, p.weps);
            }
        }
        p.fz[L.s(k, y, x)] = m * r;
    }
}

__global__ void __launch_bounds__(256) pdef_directional_kernel(Pdef p, Lane L) {
    const int ni = L.ni, nj = L.nj, nk = L.nk;
    const unsigned n = (unsigned)nk * nj * ni;
    for (unsigned q = (unsigned)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (unsigned)gridDim.x * blockDim.x) {
        const int i = (int)(q % ni), j = (int)((q / ni) % nj), k = (int)(q / ((unsigned)ni * nj)) + 1;
        const int x = i + 3, y = j + 3;
        float fw = p.fx[L.u(k, y, x)], fe = p.fx[L.u(k, y, x + 1)], fs = p.fy[L.v(k, y, x)], fn = p.fy[L.v(k, y + 1, x)];
        const float uw = p.rru[L.u(k, y, x)], ue = p.rru[L.u(k, y, x + 1)];
        const float vs = p.rrv[L.v(k, y, x)], vn = p.rrv[L.v(k, y + 1, x)];
        const bool iw = inflow_lo(i, p.obc, 0u, uw), ie = inflow_hi(i, ni, p.obc, 1u, ue);
        const bool js = inflow_lo(j, p.obc, 2u, vs), jn = inflow_hi(j, nj, p.obc, 3u, vn);
        if (iw) fw = fe;
        if (ie) fe = fw;
        if (js) fs = fn;
        if (jn) fn = fs;
        float axv = (fw - fe) * p.rdx, ayv = (fs - fn) * p.rdy;
        if (iw || ie || js || jn) {
            const float sv = p.s[L.s(k, y, x)];
            if (iw) axv = axv - (sv * (ue - uw)) * p.rdx;
            if (ie) axv = axv - (sv * (ue - uw)) * p.rdx;
            if (js) ayv = ayv - (sv * (vn - vs)) * p.rdy;
            if (jn) ayv = ayv - (sv * (vn - vs)) * p.rdy;
        }
        p.ax[q] = axv;
        p.ay[q] = ayv;
        p.az[q] = k == 1 ? pdef_zterm(p, -p.fz[L.s(2, y, x)], k)
                         : (k == nk ? pdef_zterm(p, p.fz[L.s(nk, y, x)], k)
                                    : pdef_zterm(p, p.fz[L.s(k, y, x)] - p.fz[L.s(k + 1, y, x)], k));
    }
}

// axis 0/1/2 = x/y/z candidate: dum = rho0 a + (dt (adv + (s dflux) rspacing)) gz
__global__ void __launch_bounds__(256) pdef_candidate_kernel(Pdef p, Lane L, int axis) {
    const int ni = L.ni, nj = L.nj, nk = L.nk;
    const unsigned n = (unsigned)nk * nj * ni;
    const float *dir = axis == 0 ? p.ax : axis == 1 ? p.ay : p.az;
    const float rsp = axis == 0 ? p.rdx : p.rdy;  // x and y spacing; z goes through pdef_zterm
    const bool flat = p.vmode == 2;
    for (unsigned q = (unsigned)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (unsigned)gridDim.x * blockDim.x) {
        const int i = (int)(q % ni), j = (int)((q / ni) % nj), k = (int)(q / ((unsigned)ni * nj)) + 1;
        const int x = i + 3, y = j + 3;
        float m0, m1;
        bool inflow = false;
        if (axis == 0) {
            m0 = p.rru[L.u(k, y, x)], m1 = p.rru[L.u(k, y, x + 1)];
            inflow = inflow_lo(i, p.obc, 0u, m0) || inflow_hi(i, ni, p.obc, 1u, m1);
        } else if (axis == 1) {
            m0 = p.rrv[L.v(k, y, x)], m1 = p.rrv[L.v(k, y + 1, x)];
            inflow = inflow_lo(j, p.obc, 2u, m0) || inflow_hi(j, nj, p.obc, 3u, m1);
        } else {
            m0 = p.rrw[L.s(k, y, x)], m1 = p.rrw[L.s(k + 1, y, x)];
        }
        const float dm = m1 - m0;
        const float r0a = (flat ? p.rho0[(unsigned)(k - 1) * ni * nj] : p.rho0[q]) * p.a[q];
        const float sdm = p.s[L.s(k, y, x)] * dm;
        const float inc = p.dt * (dir[q] + (axis == 2 ? pdef_zterm(p, sdm, k) : sdm * rsp));
        p.dum[q] = inflow ? r0a : (flat ? r0a + inc : r0a + inc * p.gz[(unsigned)j * ni + i]);
    }
}

__device__ __forceinline__ float zval(const float *d, long long q, int k, unsigned slab, int nk) {
    return (k < 0 || k >= nk) ? 0.0f : d[q + (long long)k * (long long)slab];
}
__device__ __forceinline__ float zratio(const float *d, long long base, int k, unsigned slab, int nk) {
    const float c = zval(d, base, k, slab, nk);
    if (c >= 0.0f) return 0.0f;
    const float f1 = fmaxf(0.0f, zval(d, base, k - 1, slab, nk)), f2 = fmaxf(0.0f, zval(d, base, k + 1, slab, nk));
    const float sum = f1 + f2;
    return sum > 1.0e-30f ? fmaxf(c, -sum) / sum : 0.0f;
}

__global__ void __launch_bounds__(256) pdef_correct_kernel(Pdef p, Lane L, int axis) {
    const int ni = L.ni, nj = L.nj, nk = L.nk;
    const unsigned n = (unsigned)nk * nj * ni, slab = (unsigned)ni * nj;
    float *dir = axis == 0 ? p.ax : axis == 1 ? p.ay : p.az;
    const float rsp = axis == 0 ? p.rdx : p.rdy;  // x and y spacing; z goes through pdef_zterm
    const bool flat = p.vmode == 2;
    const float *d = p.dum;
    for (unsigned q = (unsigned)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (unsigned)gridDim.x * blockDim.x) {
        const int i = (int)(q % ni), j = (int)((q / ni) % nj), k0 = (int)(q / slab);
        float mass = 0.0f;
        bool flag = false;
        if (axis == 2) {
            const long long base = (long long)(q - (unsigned)k0 * slab);
            const float cur = d[q];
            if (cur < 0.0f) {
                const float r = zratio(d, base, k0, slab, nk);
                if (r != 0.0f) {
                    const float sum = fmaxf(0.0f, zval(d, base, k0 - 1, slab, nk)) + fmaxf(0.0f, zval(d, base, k0 + 1, slab, nk));
                    mass = 0.0f - sum * r;
                    flag = true;
                }
            } else if (cur > 1.0e-30f) {
                const float rl = zratio(d, base, k0 - 1, slab, nk), rr = zratio(d, base, k0 + 1, slab, nk);
                if (rl != 0.0f) mass = mass + cur * rl, flag = true;
                if (rr != 0.0f) mass = mass + cur * rr, flag = true;
            }
        } else {
            const int c = axis == 0 ? i : j, nn = axis == 0 ? ni : nj;
            const long long stride = axis == 0 ? 1 : (long long)ni;
            const long long base = (long long)q - (long long)c * stride;
            if (p.obc != 0u) {
                pdef_row_mass(d, base, stride, c, nn, obc_side(p.obc, axis == 0 ? 0u : 2u),
                              obc_side(p.obc, axis == 0 ? 1u : 3u), &mass, &flag);
            } else if (c > 0 && c + 1 < nn) {
                const long long lo = base, hi = base + (long long)(nn - 1) * stride;
                if (d[q] < 0.0f) {
                    const float r = ratio1(d, (long long)q, lo, hi, stride);
                    if (r != 0.0f) {
                        const float sum = fmaxf(0.0f, d[q - stride]) + fmaxf(0.0f, d[q + stride]);
                        mass = 0.0f - sum * r;
                        flag = true;
                    }
                } else if (d[q] > 1.0e-30f) {
                    const float rl = ratio1(d, (long long)q - stride, lo, hi, stride);
                    const float rr = ratio1(d, (long long)q + stride, lo, hi, stride);
                    if (rl != 0.0f) mass = mass + d[q] * rl, flag = true;
                    if (rr != 0.0f) mass = mass + d[q] * rr, flag = true;
                }
            }
        }
        if (flag) {
            const int k = k0 + 1, x = i + 3, y = j + 3;
            const float r0 = flat ? p.rho0[(unsigned)k0 * slab] : p.rho0[q];
            float first = ((d[q] + mass) - r0 * p.a[q]) * p.rdt;
            if (!flat) first = first * p.rgz[(unsigned)j * ni + i];
            float dm;
            if (axis == 0) dm = p.rru[L.u(k, y, x + 1)] - p.rru[L.u(k, y, x)];
            else if (axis == 1) dm = p.rrv[L.v(k, y + 1, x)] - p.rrv[L.v(k, y, x)];
            else dm = p.rrw[L.s(k + 1, y, x)] - p.rrw[L.s(k, y, x)];
            const float sdm = p.s[L.s(k, y, x)] * dm;
            dir[q] = first - (axis == 2 ? pdef_zterm(p, sdm, k) : sdm * rsp);
        }
    }
}

__global__ void __launch_bounds__(256) pdef_total_kernel(Pdef p, Lane L) {
    const int ni = L.ni, nj = L.nj;
    const unsigned n = (unsigned)L.nk * nj * ni;
    for (unsigned q = (unsigned)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (unsigned)gridDim.x * blockDim.x) {
        const int i = (int)(q % ni), j = (int)((q / ni) % nj), k = (int)(q / ((unsigned)ni * nj)) + 1;
        if (!obc_owned(i, j, ni, nj, p.obc)) continue;
        float t = (p.ax[q] + p.ay[q]) + p.az[q];
        t = t + p.s[L.s(k, j + 3, i + 3)] * p.divx[q];
        p.adv[q] = p.vmode == 2 ? t * p.rr0[(unsigned)(k - 1) * ni * nj] : (t * p.rr0[q]) * p.gz[(unsigned)j * ni + i];
    }
}

// ---------------------------------------------------------------------------
// the same chain for a caller that needs only its advection: two passes and
// four words of scratch per cell (advx, advy, advz before any repair and the
// y candidate) instead of ten passes through the face fluxes, the candidates
// and the corrected rows
// ---------------------------------------------------------------------------
constexpr int kPdRows = 8;   // rows of y faces per CTA of the flux pass: 7 rows of cells
constexpr int kPdOut = 31;   // cells a warp of 32 x faces completes
constexpr int kRepOut = 28;  // cells a warp of 32 lanes completes in the repair pass
constexpr int kRepRows = 8;

// the upwind WENO flux at a face from the six points around it; nothing where
// no point exceeds the smallness
__device__ __forceinline__ float pdef_flux(float m, float s0, float s1, float s2, float s3, float s4, float s5,
                                           double weps, float small) {
    const bool pos = m >= 0.0f;
    const float a = pos ? s0 : s5, b = pos ? s1 : s4, c = pos ? s2 : s3, d = pos ? s3 : s2, e = pos ? s4 : s1;
    return max5abs(a, b, c, d, e) > small ? m * weno5(a, b, c, d, e, weps) : 0.0f;
}

// vertical flux at face f (2..nk) from levels f-3 .. f+2 (pdef_vertical_flux_kernel)
__device__ __forceinline__ float pdef_zflux(const Pdef &p, const float win[6], float m, float c1, float c2, int f,
                                            int nk, float small) {
    const float ew = (float)p.weps;
#define Q(l) win[(l) - f + 3]
    float r;
    if (f == 2) {
        r = m >= 0.0f ? c1 * Q(f - 1) + c2 * Q(f) : upstrpd(Q(f + 1), Q(f), Q(f - 1), ew);
    } else if (f == nk) {
        r = m > 0.0f ? upstrpd(Q(f - 2), Q(f - 1), Q(f), ew) : c1 * Q(f - 1) + c2 * Q(f);
    } else if (f == 3 && (p.pdefweno ? m > 0.0f : m >= 0.0f)) {
        r = upstrpd(Q(f - 2), Q(f - 1), Q(f), ew);
    } else if (f == nk - 1 && m < 0.0f) {
        r = f == 3 ? upstrpd(Q(f - 2), Q(f - 1), Q(f), ew) : upstrpd(Q(f + 1), Q(f), Q(f - 1), ew);
    } else {
        const bool pos = m >= 0.0f;
        const float a = pos ? Q(f - 3) : Q(f + 2), b = pos ? Q(f - 2) : Q(f + 1), c = pos ? Q(f - 1) : Q(f);
        const float d = pos ? Q(f) : Q(f - 1), e = pos ? Q(f + 1) : Q(f - 2);
        if (p.pdefweno && max5abs(a, b, c, d, e) <= small) return 0.0f;
        r = weno5(a, b, c, d, e, p.weps);
    }
#undef Q
    return m * r;
}

// a cell's rho0 a, the product both its candidates and its repair start from
__device__ __forceinline__ float pdef_r0a(const Pdef &p, unsigned level, unsigned q) {
    return (p.vmode == 2 ? __ldg(p.rho0 + level) : __ldg(p.rho0 + q)) * __ldg(p.a + q);
}

// Directional advection: a warp owns the x faces of one row and marches up a
// chunk of levels as the WENO scalar advection does (x fluxes by shuffle, y
// fluxes through shared memory, the vertical flux carried); the binary64
// weights bound it where there is water.  A species at 640x768x80: the chain's
// six kernels and 18 arrays 2.68 ms, 1.03 here and 0.41 in the repair.
__global__ void __launch_bounds__(32 * kPdRows, 4) pdef_advection_kernel(const __grid_constant__ Pdef p, Lane L,
                                                                          int levels_per_chunk, float small) {
    __shared__ float s_fy[2][kPdRows][32], s_vm[2][kPdRows][32];
    const int lane = threadIdx.x, ty = threadIdx.y;
    const int ni = L.ni, nj = L.nj, nk = L.nk;
    const int sx = ni + 6, sy = nj + 6, sz = sx * sy, uz = (ni + 7) * sy, vz = sx * (nj + 7), cz = ni * nj;
    const int tiles = (ni + kPdOut - 1) / kPdOut, i0 = blockIdx.x % tiles * kPdOut + lane;
    const int row = blockIdx.x / tiles * (kPdRows - 1) + ty;
    // faces and rows past the domain repeat its last ones and store nothing
    const int i = min(i0, ni), j = min(row, nj);
    const bool cell = i0 < ni && row < nj && lane < kPdOut && ty < kPdRows - 1;
    const int o = (j + 3) * sx + i + 3, ou = (j + 3) * (ni + 7) + i + 3, oc = min(j, nj - 1) * ni + min(i, ni - 1);
    const bool wo = i0 == 0 && obc_side(p.obc, 0u) == 2u, eo = i0 + 1 == ni && obc_side(p.obc, 1u) == 2u;
    const bool so = row == 0 && obc_side(p.obc, 2u) == 2u, no = row + 1 == nj && obc_side(p.obc, 3u) == 2u;
    const int k_lo = 1 + blockIdx.y * levels_per_chunk, k_hi = min(nk, k_lo + levels_per_chunk - 1);
    float win[6];  // levels k-3 .. k+2; shifted to k-2 .. k+3 for face k+1
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        const int l = k_lo - 3 + q;
        win[q] = l >= 0 && l <= nk + 1 ? __ldg(p.s + l * sz + o) : 0.0f;
    }
    auto zflux = [&](int f) {
        const bool end = f == 2 || f == nk;
        return pdef_zflux(p, win, __ldg(p.rrw + f * sz + o), end ? __ldg(p.c1 + (f - 1) * cz + oc) : 0.0f,
                          end ? __ldg(p.c2 + (f - 1) * cz + oc) : 0.0f, f, nk, small);
    };
    float zlo = 0.0f;
    if (k_lo >= 2 && cell) zlo = zflux(k_lo);
#pragma unroll 1
    for (int k = k_lo; k <= k_hi; ++k) {
        const float *pt = p.s + k * sz + o;
        float px[6], py[6];
        const float sv = win[3];
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            px[q] = q == 3 ? sv : __ldg(pt + (q - 3));
            py[q] = q == 3 ? sv : __ldg(pt + (q - 3) * sx);
        }
        const float next = k + 3 <= nk + 1 ? __ldg(pt + 3 * sz) : 0.0f;
        const float mw = __ldg(p.rru + k * uz + ou), ms = __ldg(p.rrv + k * vz + o);
        const float fx = pdef_flux(mw, px[0], px[1], px[2], px[3], px[4], px[5], p.weps, small);
        const float fy = pdef_flux(ms, py[0], py[1], py[2], py[3], py[4], py[5], p.weps, small);
        s_fy[k & 1][ty][lane] = fy;
        s_vm[k & 1][ty][lane] = ms;
        float fw = fx, fe = __shfl_down_sync(0xffffffffu, fx, 1), fs = fy;
        const float me = __shfl_down_sync(0xffffffffu, mw, 1);
        __syncthreads();
        const int up = min(ty + 1, kPdRows - 1);
        float fn = s_fy[k & 1][up][lane];
        const float mn = s_vm[k & 1][up][lane];
#pragma unroll
        for (int q = 0; q < 5; ++q) win[q] = win[q + 1];
        win[5] = next;
        if (!cell) continue;
        const float zhi = k < nk ? zflux(k + 1) : 0.0f;
        const bool iw = wo && mw >= 0.0f, ie = eo && me <= 0.0f, js = so && ms >= 0.0f, jn = no && mn <= 0.0f;
        if (iw) fw = fe;
        if (ie) fe = fw;
        if (js) fs = fn;
        if (jn) fn = fs;
        float axv = (fw - fe) * p.rdx, ayv = (fs - fn) * p.rdy;
        if (iw) axv = axv - (sv * (me - mw)) * p.rdx;
        if (ie) axv = axv - (sv * (me - mw)) * p.rdx;
        if (js) ayv = ayv - (sv * (mn - ms)) * p.rdy;
        if (jn) ayv = ayv - (sv * (mn - ms)) * p.rdy;
        const unsigned z = (unsigned)(k - 1) * (unsigned)cz + (unsigned)oc;
        p.ax[z] = axv;
        p.ay[z] = ayv;
        p.az[z] = pdef_zterm(p, k == 1 ? -zhi : k == nk ? zlo : zlo - zhi, k);
        // the y candidate, whose neighbours lie in other rows
        const float r0a = pdef_r0a(p, (unsigned)(k - 1) * (unsigned)cz, z);
        const float inc = p.dt * (ayv + (sv * (mn - ms)) * p.rdy);
        p.dum[z] = js || jn ? r0a : p.vmode == 2 ? r0a + inc : r0a + inc * __ldg(p.gz + oc);
        zlo = zhi;
    }
}

// the share a negative candidate v between lo and hi takes of each neighbour
__device__ __forceinline__ float pdef_share(float v, float lo, float hi) {
    if (v >= 0.0f) return 0.0f;
    const float sum = fmaxf(0.0f, lo) + fmaxf(0.0f, hi);
    return sum > 1.0e-30f ? fmaxf(v, -sum) / sum : 0.0f;
}

// the repair's mass of a cell from the candidates of its line, c-2 .. c+2
// (pdef_row_mass); false where there is none
__device__ __forceinline__ bool pdef_mass(float ll, float l, float v, float r, float rr, float &mass) {
    mass = 0.0f;
    bool flag = false;
    if (v < 0.0f) {
        const float s = pdef_share(v, l, r);
        if (s != 0.0f) {
            const float sum = fmaxf(0.0f, l) + fmaxf(0.0f, r);
            mass = 0.0f - sum * s;
            flag = true;
        }
    } else if (v > 1.0e-30f) {
        const float sl = pdef_share(l, ll, v), sr = pdef_share(r, v, rr);
        if (sl != 0.0f) mass = mass + v * sl, flag = true;
        if (sr != 0.0f) mass = mass + v * sr, flag = true;
    }
    return flag;
}

// Candidates, repair rows and the total in one pass: the y candidates come
// from the first pass, a warp's 32 lanes hold their row's x candidates (two
// of the boundary family's cells, or of the next tiles', on either side of the
// 28 cells it completes) and pass them by shuffle, the z candidates of levels
// k-2 .. k+2 are carried up the column.  No barrier: warps are independent.
// With the rows handed along y through shared memory instead (two halo rows
// on either side of 12, a barrier a level) it took 1.07 ms at 640x768x80.
__global__ void __launch_bounds__(32 * kRepRows, 4) pdef_repair_kernel(const __grid_constant__ Pdef p,
                                                                        const __grid_constant__ Lane L,
                                                                        int levels_per_chunk) {
    const int ni = L.ni, nj = L.nj, nk = L.nk, lane = threadIdx.x;
    const int tiles = (ni + kRepOut - 1) / kRepOut;
    const int i0 = blockIdx.x % tiles * kRepOut + lane - 2, j = blockIdx.x / tiles * kRepRows + threadIdx.y;
    if (j >= nj) return;  // whole warps
    const unsigned so = obc_side(p.obc, 2u), no = obc_side(p.obc, 3u);
    // beyond the domain the boundary family's cell; further out, any
    const int i = (int)pdef_cell(min(i0, ni + 1), ni, obc_side(p.obc, 0u), obc_side(p.obc, 1u));
    const bool own = lane >= 2 && lane < kRepOut + 2 && i0 < ni;
    const unsigned cz = (unsigned)ni * nj, sz = (unsigned)(nj + 6) * (ni + 6), uz = (unsigned)(nj + 6) * (ni + 7),
                   vz = (unsigned)(nj + 7) * (ni + 6);
    const unsigned oc = (unsigned)j * ni + i, os = (unsigned)(j + 3) * (ni + 6) + (i + 3),
                   ou = (unsigned)(j + 3) * (ni + 7) + (i + 3);
    auto yrow = [&](int c) { return (unsigned)pdef_cell(c, nj, so, no) * (unsigned)ni + (unsigned)i; };
    const unsigned ys = yrow(j - 1), yn = yrow(j + 1);
    const bool flat = p.vmode == 2;
    const float gz = flat ? 0.0f : __ldg(p.gz + oc), rgz = flat ? 0.0f : __ldg(p.rgz + oc);
    const bool wo = i == 0 && obc_side(p.obc, 0u) == 2u, eo = i + 1 == ni && obc_side(p.obc, 1u) == 2u;
    const int k_lo = 1 + blockIdx.y * levels_per_chunk, k_hi = min(nk, k_lo + levels_per_chunk - 1);
    auto step = [&](float r0a, float inc) { return flat ? r0a + inc : r0a + inc * gz; };
    // z candidates and what the levels k .. k+2 need again
    float zc[5], r0a[3], s[3], az[3], wlo = 0.0f;
    auto z_cand = [&](int k, float w0, float w1, float ra, float sv, float dir) {
        return step(ra, p.dt * (dir + pdef_zterm(p, sv * (w1 - w0), k)));
    };
    // levels k_lo-2 .. k_lo+1; the loop's first level adds k_lo+2
    zc[0] = r0a[0] = s[0] = az[0] = 0.0f;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int k = k_lo - 2 + q;
        float c = 0.0f, ra = 0.0f, sv = 0.0f, dir = 0.0f;
        if (k >= 1 && k <= nk) {
            const unsigned z = (unsigned)(k - 1) * cz + oc;
            ra = pdef_r0a(p, (unsigned)(k - 1) * cz, z);
            sv = __ldg(p.s + (unsigned)k * sz + os);
            dir = __ldg(p.az + z);
            wlo = __ldg(p.rrw + (unsigned)(k + 1) * sz + os);
            c = z_cand(k, __ldg(p.rrw + (unsigned)k * sz + os), wlo, ra, sv, dir);
        }
        zc[q + 1] = c;
        if (q >= 2) r0a[q - 1] = ra, s[q - 1] = sv, az[q - 1] = dir;
    }
#pragma unroll 1
    for (int k = k_lo; k <= k_hi; ++k) {
        const unsigned level = (unsigned)(k - 1) * cz, z = level + oc, u = (unsigned)k * uz + ou;
        const float yl = __ldg(p.dum + level + ys), yc = __ldg(p.dum + z), yr = __ldg(p.dum + level + yn);
        const float u0 = __ldg(p.rru + u), u1 = __ldg(p.rru + u + 1);
        const float ax = __ldg(p.ax + z), ay = __ldg(p.ay + z), div = __ldg(p.divx + z);
        const float rr0 = __ldg(p.rr0 + (flat ? level : z));
#pragma unroll
        for (int q = 0; q < 4; ++q) zc[q] = zc[q + 1];
        r0a[0] = r0a[1], s[0] = s[1], az[0] = az[1];
        r0a[1] = r0a[2], s[1] = s[2], az[1] = az[2];
        zc[4] = 0.0f;
        if (k + 2 <= nk) {
            const float whi = __ldg(p.rrw + (unsigned)(k + 3) * sz + os);
            r0a[2] = pdef_r0a(p, level + 2 * cz, z + 2 * cz);
            s[2] = __ldg(p.s + (unsigned)(k + 2) * sz + os);
            az[2] = __ldg(p.az + z + 2 * cz);
            zc[4] = z_cand(k + 2, wlo, whi, r0a[2], s[2], az[2]);
            wlo = whi;
        }
        const float sdx = (s[0] * (u1 - u0)) * p.rdx;
        const float xc = (wo && u0 >= 0.0f) || (eo && u1 <= 0.0f) ? r0a[0] : step(r0a[0], p.dt * (ax + sdx));
        const float xl = __shfl_up_sync(0xffffffffu, xc, 1), xr = __shfl_down_sync(0xffffffffu, xc, 1);
        float dx = ax, dy = ay, dz = az[0], mass;
        auto repaired = [&](float c, float m, float sd) {
            float first = ((c + m) - r0a[0]) * p.rdt;
            if (!flat) first = first * rgz;
            return first - sd;
        };
        // away from the edge of the water no candidate nearby is negative
        const bool fx = !(xl >= 0.0f && xc >= 0.0f && xr >= 0.0f);
        if (__any_sync(0xffffffffu, fx)) {
            const float xll = __shfl_up_sync(0xffffffffu, xc, 2), xrr = __shfl_down_sync(0xffffffffu, xc, 2);
            if (fx && pdef_mass(xll, xl, xc, xr, xrr, mass)) dx = repaired(xc, mass, sdx);
        }
        if (!(yl >= 0.0f && yc >= 0.0f && yr >= 0.0f) &&
            pdef_mass(__ldg(p.dum + level + yrow(j - 2)), yl, yc, yr, __ldg(p.dum + level + yrow(j + 2)), mass)) {
            const unsigned v = (unsigned)k * vz + os;
            dy = repaired(yc, mass, (s[0] * (__ldg(p.rrv + v + (unsigned)(ni + 6)) - __ldg(p.rrv + v))) * p.rdy);
        }
        if (!(zc[1] >= 0.0f && zc[2] >= 0.0f && zc[3] >= 0.0f) && pdef_mass(zc[0], zc[1], zc[2], zc[3], zc[4], mass)) {
            const unsigned w = (unsigned)k * sz + os;
            dz = repaired(zc[2], mass, pdef_zterm(p, s[0] * (__ldg(p.rrw + w + sz) - __ldg(p.rrw + w)), k));
        }
        if (own) {
            float t = (dx + dy) + dz;
            t = t + s[0] * div;
            p.adv[z] = flat ? t * rr0 : (t * rr0) * gz;
        }
    }
}

// ---------------------------------------------------------------------------
// held tendencies, solve3 density, scalar pack
// ---------------------------------------------------------------------------
struct Held {
    const float *th0, *pi0, *rho, *ppi, *tha, *qa, *qpten, *qtten, *qvten, *qcten;
    float *thheld, *qheld, *ppten;
};

__global__ void __launch_bounds__(256) held_compose_kernel(Held h, int ni, int nj, int nk, float dt) {
    const unsigned n = (unsigned)ni * nj * nk;
    const float rd = 287.04f, rv = 461.5f, rp00 = 1.0f / 100000.0f, rddcv = 287.04f / (1005.7f - 287.04f);
    const float tem = 0.0001f * 0.0001f, qsmall = 1.0e-14f;
    for (unsigned q = (unsigned)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (unsigned)gridDim.x * blockDim.x) {
        const int i = (int)(q % ni), j = (int)((q / ni) % nj), k = (int)(q / ((unsigned)ni * nj));
        const unsigned pp = ((unsigned)(k + 1) * (nj + 2) + (j + 1)) * (unsigned)(ni + 2) + (i + 1);
        const float ht = h.thheld[q], qvt = h.qheld[q];
        if (fabsf(dt * ht) > tem || fabsf(dt * qvt) > qsmall) {
            const float thnew = h.tha[q] + dt * ht, qvnew = h.qa[q] + dt * qvt;
            float base = (h.rho[q] * (h.th0[q] + thnew)) * (rd + rv * qvnew);
            base = base * rp00;
            const float pinew = powf(base, rddcv) - h.pi0[q];
            h.ppten[pp] = (pinew - h.ppi[q]) / dt + h.qpten[q];
        } else {
            h.ppten[pp] = h.qpten[q];
        }
        h.thheld[q] = ht + h.qtten[q];
        h.qheld[q] = qvt + h.qvten[q];
        h.qheld[n + q] = h.qheld[n + q] + h.qcten[q];
    }
}

__global__ void __launch_bounds__(256) solve3_density_kernel(const float *rho, const float *c1, const float *c2,
                                                            float *rr, float *rf, int ni, int nj, int nk) {
    const unsigned n = (unsigned)ni * nj * nk, nf = (unsigned)ni * nj * (nk + 1), plane = (unsigned)ni * nj;
    for (unsigned z = (unsigned)blockIdx.x * blockDim.x + threadIdx.x; z < nf; z += (unsigned)gridDim.x * blockDim.x) {
        if (z < n) rr[z] = 1.0f / rho[z];
        const unsigned h = z % plane;
        const int f = (int)(z / plane);
        if (f == 0) rf[z] = (1.875f * rho[h] + (-1.25f) * rho[plane + h]) + 0.375f * rho[2 * plane + h];
        else if (f == nk)
            rf[z] = (1.875f * rho[(unsigned)(nk - 1) * plane + h] + (-1.25f) * rho[(unsigned)(nk - 2) * plane + h]) +
                    0.375f * rho[(unsigned)(nk - 3) * plane + h];
        else rf[z] = c1[z] * rho[(unsigned)(f - 1) * plane + h] + c2[z] * rho[(unsigned)f * plane + h];
    }
}

__global__ void __launch_bounds__(256) pack_scalar_kernel(const float *s, float *padded, Lane L) {
    const unsigned n = (unsigned)L.nk * L.nj * L.ni;
    for (unsigned q = (unsigned)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (unsigned)gridDim.x * blockDim.x) {
        const int i = (int)(q % L.ni), j = (int)((q / L.ni) % L.nj), k = (int)(q / ((unsigned)L.ni * L.nj)) + 1;
        padded[L.s(k, j + 3, i + 3)] = s[q];
    }
}

// bc.F:1151-1178 on the physical bottom faces (cpu_bcwsfc_terrain_physical_inplace)
__global__ void __launch_bounds__(256) bcwsfc_kernel(const float *u, const float *v, float *w, const float *gz,
                                                    const float *dzdx, const float *dzdy, Lane L) {
    const unsigned n = (unsigned)L.nj * L.ni;
    for (unsigned q = (unsigned)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (unsigned)gridDim.x * blockDim.x) {
        const int i0 = (int)(q % L.ni), j0 = (int)(q / L.ni), y = j0 + 3, x = i0 + 3;
        const float ut = (u[L.u(1, y, x)] + u[L.u(1, y, x + 1)]) * dzdx[q];
        const float vt = (v[L.v(1, y, x)] + v[L.v(1, y + 1, x)]) * dzdy[q];
        w[L.s(1, y, x)] = (0.5f * (ut + vt)) * gz[q];
    }
}

// cm1_momentum_rk_bc2d_open_v1: the w(1) slab's open halo, west and east
// over every row (pass 0), then south and north over every column (pass 1)
__global__ void __launch_bounds__(256) w_level1_fill_kernel(float *w, Lane L, int pass) {
    const int nx = L.ni + 6, ny = L.nj + 6;
    const unsigned n = pass == 0 ? (unsigned)ny * 6 : (unsigned)nx * 6;
    float *s = w + (unsigned)1 * nx * ny;
    for (unsigned q = (unsigned)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (unsigned)gridDim.x * blockDim.x) {
        if (pass == 0) {
            const int y = (int)(q / 6), h = (int)(q % 6);
            const int x = h < 3 ? h : 3 + L.ni + (h - 3), sx = h < 3 ? 3 : 3 + L.ni - 1;
            s[(unsigned)y * nx + x] = s[(unsigned)y * nx + sx];
        } else {
            const int x = (int)(q % nx), h = (int)(q / nx);
            const int y = h < 3 ? h : 3 + L.nj + (h - 3), sy = h < 3 ? 3 : 3 + L.nj - 1;
            s[(unsigned)y * nx + x] = s[(unsigned)sy * nx + x];
        }
    }
}

}  // namespace
}  // namespace gm1b

using namespace gm1b;

namespace {
bool grid_ok(int ni, int nj, int nk, int mi, int mj, int mk, const char *what) {
    if (ni < mi || nj < mj || nk < mk) {
        gm1b_set_error("%s: need ni >= %d, nj >= %d, nk >= %d", what, mi, mj, mk);
        return false;
    }
    // the kernels index and count with 32-bit words
    if ((size_t)(nk + 3) * (size_t)(nj + 7) * (size_t)(ni + 7) * 2 >= ((size_t)1 << 31)) {
        gm1b_set_error("%s: a %dx%dx%d grid's padded arrays reach 2^30 words; the kernels index with 32-bit offsets",
                       what, ni, nj, nk);
        return false;
    }
    return true;
}
}  // namespace

namespace gm1b {

int32_t open_fills(int32_t ni, int32_t nj, int32_t nk, const OpenFill *fills, int n, cudaStream_t st) {
    Fills a{};
    size_t work = 0;
    for (int q = 0; q < n; ++q) {
        FillGeom &f = a.f[q];
        if (n > kMostFills || !fill_geometry(fills[q].kind, ni, nj, nk, fills[q].q, f)) return GM1B_ERR_ARGUMENT;
        const size_t per = ((size_t)(f.xl - f.x0 + 1) + (size_t)(f.yl - f.y0 + 1) + 2) * 2 * f.g;
        a.words[q] = f.k1 >= f.k0 ? (unsigned)(per * (size_t)(f.k1 - f.k0 + 1)) : 0u;
        work = std::max(work, (size_t)a.words[q]);
        if (f.zero_w) work = std::max(work, (size_t)2 * (f.yl - f.y0 + 3) * (f.xl - f.x0 + 3));
    }
    a.n = n;
    ProfScope ps("open_fill_kernel", st);
    open_fill_kernel<<<grid_for(work), 256, 0, st>>>(a);
    ps.stop();
    return launch_ok("open_fill_kernel") ? GM1B_OK : GM1B_ERR_CUDA;
}

int32_t pack_scalars_open(int32_t ni, int32_t nj, int32_t nk, const float *th0, const float *const scalar[4],
                          float *const padded[4], cudaStream_t st) {
    PackScalars a{};
    a.th0 = th0;
    for (int q = 0; q < 4; ++q) a.scalar[q] = scalar[q], a.padded[q] = padded[q];
    ProfScope ps("pack_scalars_kernel", st);
    pack_scalars_kernel<<<dim3((ni + 6 + 31) / 32, (nj + 6 + 7) / 8, nk), dim3(32, 8), 0, st>>>(a, ni, nj);
    ps.stop();
    return launch_ok("pack_scalars_kernel") ? GM1B_OK : GM1B_ERR_CUDA;
}

}  // namespace gm1b

extern "C" int32_t gm1b_open_fill(int32_t ni, int32_t nj, int32_t nk, int32_t kind, float *q, void *stream) {
    FillGeom f;
    if (q == nullptr || !grid_ok(ni, nj, nk, 2, 2, 2, "gm1b_open_fill") || !fill_geometry(kind, ni, nj, nk, q, f)) {
        if (q == nullptr || kind < 0 || kind > GM1B_FILL_W_KEEP_ENDS)
            gm1b_set_error("gm1b_open_fill: need an array and a GM1B_FILL_* kind");
        return GM1B_ERR_ARGUMENT;
    }
    const OpenFill one{kind, q};
    return open_fills(ni, nj, nk, &one, 1, static_cast<cudaStream_t>(stream));
}

namespace {
// CTAs of W x (256/W) columns, all in one grid dimension, which takes any plane
template <int W>
unsigned march_tiles(int nx, int ny) {
    return (unsigned)((nx + W - 1) / W) * (unsigned)((ny + 256 / W - 1) / (256 / W));
}

// Runs f with the width of a march's CTAs: 32 columns, or 16 where that leaves
// a third fewer CTAs, on planes up to 16 cells wide (9x200x150: buoyancy 11.7
// -> 7.8 us, the post-acoustic divergences 24.0 -> 18.1, a thread per point 8.2
// and 18.1; 12x300x60: 8.5 -> 5.9 and 18.9 -> 13.0, 7.1 and 15.3).
template <class F>
void with_tile_width(int ni, int nj, F f) {
    if (3ull * march_tiles<16>(ni, nj) <= 2ull * march_tiles<32>(ni, nj))
        f(std::integral_constant<int, 16>());
    else
        f(std::integral_constant<int, 32>());
}

int32_t buoyancy_launch(int32_t ni, int32_t nj, int32_t nk, const float *dum8, const float *c1, const float *c2,
                        const float *gxu, const float *gyv, float *uten, float *vten, float *wten, int w_only,
                        void *stream) {
    if (!dum8 || !c1 || !c2 || !gxu || !gyv || !uten || !vten || !wten ||
        !grid_ok(ni, nj, nk, 2, 2, 2, "gm1b_moist_buoyancy")) {
        if (!dum8 || !c1 || !c2 || !gxu || !gyv || !uten || !vten || !wten)
            gm1b_set_error("gm1b_moist_buoyancy: NULL array");
        return GM1B_ERR_ARGUMENT;
    }
    const void *all[8] = {dum8, c1, c2, gxu, gyv, uten, vten, wten};
    for (int x = 0; x < 8; ++x)
        for (int y = x + 1; y < 8; ++y)
            if (all[x] == all[y]) {
                gm1b_set_error("gm1b_moist_buoyancy: the eight arrays must be distinct");
                return GM1B_ERR_ARGUMENT;
            }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const Lane L{ni, nj, nk};
    ProfScope ps("msb_buoyancy_kernel", st);
    with_tile_width(ni, nj, [&](auto width) {
        constexpr int W = decltype(width)::value;
        const unsigned tiles = march_tiles<W>(ni, nj);
        const int chunk = level_chunk(tiles, nk, true);
        const dim3 grid(tiles, (nk + chunk - 1) / chunk), block(W, 256 / W);
        if (w_only)
            msb_buoyancy_kernel<true, W><<<grid, block, 0, st>>>(dum8, c1, c2, gxu, gyv, uten, vten, wten, L, chunk);
        else
            msb_buoyancy_kernel<false, W><<<grid, block, 0, st>>>(dum8, c1, c2, gxu, gyv, uten, vten, wten, L, chunk);
    });
    ps.stop();
    return launch_ok("msb_buoyancy_kernel") ? GM1B_OK : GM1B_ERR_CUDA;
}
}  // namespace

extern "C" int32_t gm1b_moist_buoyancy(int32_t ni, int32_t nj, int32_t nk, const float *dum8, const float *c1,
                                       const float *c2, const float *gxu, const float *gyv, float *uten, float *vten,
                                       float *wten, void *stream) {
    return buoyancy_launch(ni, nj, nk, dum8, c1, c2, gxu, gyv, uten, vten, wten, 0, stream);
}

// launch_cuda_gm1_flat_stretched_buoyancy (src/cm1core/cuda_gm1_child_stretched_moist.py:240):
// a flat column adds the buoyancy to wten only (solve2.F:897-906; the
// uten/vten term of :971-1008 is a terrain statement); gxu, gyv, uten and
// vten may be NULL
extern "C" int32_t gm1b_moist_buoyancy_flat(int32_t ni, int32_t nj, int32_t nk, const float *dum8, const float *c1,
                                            const float *c2, float *wten, void *stream) {
    // the w-only launch never reads or writes the u/v arrays; distinct stand-ins keep the aliasing check meaningful
    if (!dum8 || !c1 || !c2 || !wten) {
        gm1b_set_error("gm1b_moist_buoyancy_flat: NULL array");
        return GM1B_ERR_ARGUMENT;
    }
    static float standin[4];
    return buoyancy_launch(ni, nj, nk, dum8, c1, c2, standin, standin + 1, standin + 2, standin + 3, wten, 1, stream);
}

namespace {
int32_t post_acoustic_launch(int32_t ni, int32_t nj, int32_t nk, const gm1b_post_acoustic_arrays *a, float dx,
                             float dy, float dz, const gm1b_momentum_column *c, void *stream) {
    if (a == nullptr || !grid_ok(ni, nj, nk, 2, 2, 2, "gm1b_post_acoustic_flux")) {
        if (a == nullptr) gm1b_set_error("gm1b_post_acoustic_flux: NULL arrays");
        return GM1B_ERR_ARGUMENT;
    }
    const void *need[] = {a->rru, a->rrv, a->rrw, a->rgzu, a->rgzv, a->dzdx, a->dzdy, a->gz, a->rho0_3d, a->rf0,
                          a->thterm, a->divergence, a->theta_divergence_term, a->divx};
    for (const void *q : need)
        if (q == nullptr) {
            gm1b_set_error("gm1b_post_acoustic_flux: NULL array");
            return GM1B_ERR_ARGUMENT;
        }
    if (!(dx > 0.0f) || !(dy > 0.0f) || !(dz > 0.0f)) {
        gm1b_set_error("gm1b_post_acoustic_flux: dx, dy, dz must be > 0");
        return GM1B_ERR_ARGUMENT;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const Lane L{ni, nj, nk};
    const float rdx = 1.0f / dx, rdy = 1.0f / dy, rdsf = 1.0f / dz;
    const int vmode = c == nullptr ? 0 : (c->flat ? 2 : 1);
    const float zt = vmode == 1 ? c->ztop : (float)nk * dz;
    Getdiv g{a->rru, a->rrv, a->rrw, a->rgzu, a->rgzv, a->dzdx, a->dzdy, a->gz, a->thterm, a->divergence,
             a->theta_divergence_term, rdx, rdy, rdsf, dz, zt, 0.0f, vmode,
             c ? c->sigma : nullptr, c ? c->sigmaf : nullptr, c ? c->rds : nullptr, c ? c->rdsf : nullptr,
             c ? c->mh : nullptr, c ? c->rdz : 0.0f};
    if (vmode == 2) {
        const dim3 block(32, 8);
        {
            ProfScope ps("msb_flat_divergences_kernel", st);
            msb_flat_divergences_kernel<<<dim3((ni + 31) / 32 * ((nj + 7) / 8), std::min(nk, 65535)), block, 0, st>>>(
                g, c->rho0_padded, a->rf0, a->divx, L);
            ps.stop();
        }
        if (!launch_ok("msb_flat_divergences_kernel")) return GM1B_ERR_CUDA;
        {
            ProfScope ps("msb_flat_mass_kernel", st);
            msb_flat_mass_kernel<<<dim3((ni / 32 + 1) * (nj / 8 + 1), std::min(nk + 1, 65535)), block, 0, st>>>(
                c->rho0_padded, a->rf0, a->rru, a->rrv, a->rrw, L);
            ps.stop();
        }
        return launch_ok("msb_flat_mass_kernel") ? GM1B_OK : GM1B_ERR_CUDA;
    }
    int32_t result = GM1B_ERR_CUDA;
    with_tile_width(ni, nj, [&](auto width) {
        constexpr int W = decltype(width)::value;
        const unsigned tiles = march_tiles<W>(ni, nj), faces = march_tiles<W>(ni + 1, nj + 1);
        const int chunk = level_chunk(tiles, nk, true);
        const dim3 grid(tiles, (nk + chunk - 1) / chunk), block(W, 256 / W);
        {
            ProfScope ps("msb_getdiv_kernel", st);
            if (vmode == 1)
                msb_getdiv_kernel<1, W><<<grid, block, 0, st>>>(g, L, chunk);
            else
                msb_getdiv_kernel<0, W><<<grid, block, 0, st>>>(g, L, chunk);
            ps.stop();
        }
        if (!launch_ok("msb_getdiv_kernel")) return;
        {
            ProfScope ps("msb_getdivx_horizontal_kernel", st);
            msb_getdivx_horizontal_kernel<W><<<dim3(faces, grid.y), block, 0, st>>>(
                a->rho0_3d, a->rgzu, a->rgzv, a->rru, a->rrv, L, vmode, c ? c->rho0_padded : nullptr, chunk);
            ps.stop();
        }
        if (!launch_ok("msb_getdivx_horizontal_kernel")) return;
        {
            ProfScope ps("msb_getdivx_vertical_kernel", st);
            msb_getdivx_vertical_kernel<W><<<grid, block, 0, st>>>(a->rf0, a->dzdx, a->dzdy, a->gz, a->rru, a->rrv,
                                                                  a->rrw, dz, L, vmode, g.sigma, g.sigmaf, g.rds, zt,
                                                                  chunk);
            ps.stop();
        }
        if (!launch_ok("msb_getdivx_vertical_kernel")) return;
        {
            ProfScope ps("msb_getdivx_divergence_kernel", st);
            msb_getdivx_divergence_kernel<W><<<grid, block, 0, st>>>(a->rru, a->rrv, a->rrw, a->divx, rdx, rdy, rdsf, L,
                                                                    vmode, g.rdsfp, chunk);
            ps.stop();
        }
        if (launch_ok("msb_getdivx_divergence_kernel")) result = GM1B_OK;
    });
    return result;
}
}  // namespace

extern "C" int32_t gm1b_post_acoustic_flux(int32_t ni, int32_t nj, int32_t nk, const gm1b_post_acoustic_arrays *a,
                                           float dx, float dy, float dz, void *stream) {
    return post_acoustic_launch(ni, nj, nk, a, dx, dy, dz, nullptr, stream);
}

extern "C" int32_t gm1b_post_acoustic_flux_column(int32_t ni, int32_t nj, int32_t nk,
                                                  const gm1b_post_acoustic_arrays *a, float dx, float dy,
                                                  const gm1b_momentum_column *column, void *stream) {
    if (column == nullptr || (column->flat != 0 && column->flat != 1) || column->rho0_padded == nullptr ||
        (column->flat ? (column->mh == nullptr || !(column->rdz > 0.0f))
                      : (column->sigma == nullptr || column->sigmaf == nullptr || column->rds == nullptr ||
                         column->rdsf == nullptr || !(column->ztop > 0.0f)))) {
        gm1b_set_error("gm1b_post_acoustic_flux_column: need the padded base density and a flat column (mh, rdz > 0) "
                       "or a terrain column (sigma, sigmaf, rds, rdsf, ztop > 0)");
        return GM1B_ERR_ARGUMENT;
    }
    // dz forms only the uniform reciprocals, which a stretched column never reads
    return post_acoustic_launch(ni, nj, nk, a, dx, dy, 1.0f, column, stream);
}

namespace {
// the operator's arguments; `whole` for the chain that leaves every row,
// false for its advection alone (fx, fy and fz unused)
int32_t pdef_args(int32_t ni, int32_t nj, int32_t nk, const gm1b_pdef_chain_arrays *a, float dttmp, float dx, float dy,
                  float dz, double weps, uint32_t lateral_obc, int32_t pdefweno, const gm1b_vertical_column *column,
                  bool whole, Pdef &p, const char *what) {
    if (a == nullptr || !grid_ok(ni, nj, nk, 2, 2, 4, what)) {
        if (a == nullptr) gm1b_set_error("%s: NULL arrays", what);
        return GM1B_ERR_ARGUMENT;
    }
    if (column != nullptr && ((column->flat != 0 && column->flat != 1) ||
                              (column->flat ? (column->mh == nullptr || !(column->rdz > 0.0f) || !isfinite(column->rdz))
                                            : column->rdsf == nullptr))) {
        gm1b_set_error("%s: need a flat column (mh, rdz > 0) or a terrain column (rdsf)", what);
        return GM1B_ERR_ARGUMENT;
    }
    const void *need[] = {a->scalar_a, a->scalar_padded, a->rho0_3d, a->gz, a->rgz, a->rr0, a->c1, a->c2, a->divx,
                          a->rru, a->rrv, a->rrw, a->advx, a->advy, a->advz, a->candidate, a->advection};
    const void *rows[] = {a->fx, a->fy, a->fz};
    bool null = false;
    for (const void *q : need) null = null || q == nullptr;
    for (const void *q : rows) null = null || (whole && q == nullptr);
    if (null) {
        gm1b_set_error("%s: NULL array", what);
        return GM1B_ERR_ARGUMENT;
    }
    for (int s = 0; s < 4; ++s) {
        const unsigned v = (lateral_obc >> (4 * s)) & 15u;
        if (v > 4) {
            gm1b_set_error("%s: lateral side codes must be 0..4", what);
            return GM1B_ERR_ARGUMENT;
        }
    }
    if (!(dttmp > 0.0f) || !(dx > 0.0f) || !(dy > 0.0f) || !(dz > 0.0f)) {
        gm1b_set_error("%s: dttmp, dx, dy, dz must be > 0", what);
        return GM1B_ERR_ARGUMENT;
    }
    p = Pdef{};
    p.a = a->scalar_a, p.s = a->scalar_padded, p.rho0 = a->rho0_3d, p.gz = a->gz, p.rgz = a->rgz, p.rr0 = a->rr0;
    p.c1 = a->c1, p.c2 = a->c2, p.divx = a->divx, p.rru = a->rru, p.rrv = a->rrv, p.rrw = a->rrw;
    p.fx = a->fx, p.fy = a->fy, p.fz = a->fz, p.ax = a->advx, p.ay = a->advy, p.az = a->advz;
    p.dum = a->candidate, p.adv = a->advection;
    p.vmode = column == nullptr ? 0 : column->flat ? 2 : 1;
    p.dt = dttmp, p.dx = dx, p.dy = dy, p.dz = dz;
    p.rdx = 1.0f / dx, p.rdy = 1.0f / dy, p.rdz = column == nullptr ? 1.0f / dz : column->rdz, p.rdt = 1.0f / dttmp;
    p.weps = weps, p.obc = lateral_obc, p.pdefweno = pdefweno ? 1 : 0;
    p.rdsf = column ? column->rdsf : nullptr, p.mh = column ? column->mh : nullptr;
    return GM1B_OK;
}

int32_t pdef_chain_launch(const Pdef &p, const Lane &L, cudaStream_t st) {
    const int ni = L.ni, nj = L.nj, nk = L.nk;
    const size_t n = (size_t)ni * nj * nk;
#define TOS_LAUNCH(name, work, ...)                                    \
    do {                                                               \
        ProfScope ps(#name, st);                                       \
        name<<<grid_for(work), 256, 0, st>>>(__VA_ARGS__);             \
        ps.stop();                                                     \
        if (!launch_ok(#name)) return GM1B_ERR_CUDA;                   \
    } while (0)
    TOS_LAUNCH(pdef_horizontal_flux_kernel, (size_t)nk * (nj + 1) * (ni + 1), p, L);
    TOS_LAUNCH(pdef_vertical_flux_kernel, (size_t)(nk - 1) * nj * ni, p, L);
    TOS_LAUNCH(pdef_directional_kernel, n, p, L);
    for (int axis = 0; axis < 3; ++axis) {
        TOS_LAUNCH(pdef_candidate_kernel, n, p, L, axis);
        TOS_LAUNCH(pdef_correct_kernel, n, p, L, axis);
    }
    TOS_LAUNCH(pdef_total_kernel, n, p, L);
#undef TOS_LAUNCH
    return GM1B_OK;
}

// levels per chunk of a marching pass: halve until two rounds of `warps` on
// each of 148 SMs, or at most four levels, are left
int march_chunk(long long row_warps, int nk, int warps) {
    int chunk = nk;
    while (chunk > 4 && row_warps * ((nk + chunk - 1) / chunk) < 2LL * 148 * warps) chunk = (chunk + 1) / 2;
    return chunk;
}
}  // namespace

extern "C" int32_t gm1b_pdef_moisture_chain(int32_t ni, int32_t nj, int32_t nk, const gm1b_pdef_chain_arrays *a,
                                            float dttmp, float dx, float dy, float dz, double weps,
                                            uint32_t lateral_obc, int32_t pdefweno, void *stream) {
    Pdef p;
    const int32_t r = pdef_args(ni, nj, nk, a, dttmp, dx, dy, dz, weps, lateral_obc, pdefweno, nullptr, true, p,
                                "gm1b_pdef_moisture_chain");
    return r != GM1B_OK ? r : pdef_chain_launch(p, Lane{ni, nj, nk}, static_cast<cudaStream_t>(stream));
}

extern "C" int32_t gm1b_pdef_moisture_chain_column(int32_t ni, int32_t nj, int32_t nk,
                                                   const gm1b_pdef_chain_arrays *a, float dttmp, float dx, float dy,
                                                   double weps, uint32_t lateral_obc, int32_t pdefweno,
                                                   const gm1b_vertical_column *column, void *stream) {
    if (column == nullptr) {
        gm1b_set_error("gm1b_pdef_moisture_chain_column: need a flat column (mh, rdz > 0) or a terrain column (rdsf)");
        return GM1B_ERR_ARGUMENT;
    }
    Pdef p;
    const int32_t r = pdef_args(ni, nj, nk, a, dttmp, dx, dy, 1.0f, weps, lateral_obc, pdefweno, column, true, p,
                                "gm1b_pdef_moisture_chain_column");
    return r != GM1B_OK ? r : pdef_chain_launch(p, Lane{ni, nj, nk}, static_cast<cudaStream_t>(stream));
}

extern "C" int32_t gm1b_pdef_moisture_advection(int32_t ni, int32_t nj, int32_t nk, const gm1b_pdef_chain_arrays *a,
                                                float dttmp, float dx, float dy, float dz, double weps,
                                                uint32_t lateral_obc, int32_t pdefweno,
                                                const gm1b_vertical_column *column, void *stream) {
    for (int s = 0; s < 4; ++s)
        if (((lateral_obc >> (4 * s)) & 15u) == 0u) {
            gm1b_set_error("gm1b_pdef_moisture_advection: lateral code 0x%x: each side is 1..4", lateral_obc);
            return GM1B_ERR_ARGUMENT;
        }
    Pdef p;
    const int32_t r = pdef_args(ni, nj, nk, a, dttmp, dx, dy, column ? 1.0f : dz, weps, lateral_obc, pdefweno, column,
                                false, p, "gm1b_pdef_moisture_advection");
    if (r != GM1B_OK) return r;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const Lane L{ni, nj, nk};
    // largest float <= weps: x > weps exactly when x > small, for every float x
    float small = (float)weps;
    if ((double)small > weps) small = nextafterf(small, -INFINITY);
    {
        const int tiles = (ni + kPdOut - 1) / kPdOut, rows = (nj + kPdRows - 2) / (kPdRows - 1);
        const int chunk = march_chunk((long long)tiles * nj, nk, 32);
        ProfScope ps("pdef_advection_kernel", st);
        pdef_advection_kernel<<<dim3(tiles * rows, (nk + chunk - 1) / chunk), dim3(32, kPdRows), 0, st>>>(p, L, chunk,
                                                                                                         small);
        ps.stop();
    }
    if (!launch_ok("pdef_advection_kernel")) return GM1B_ERR_CUDA;
    {
        const int tiles = (ni + kRepOut - 1) / kRepOut, rows = (nj + kRepRows - 1) / kRepRows;
        const int chunk = march_chunk((long long)tiles * nj, nk, 32);
        ProfScope ps("pdef_repair_kernel", st);
        pdef_repair_kernel<<<dim3(tiles * rows, (nk + chunk - 1) / chunk), dim3(32, kRepRows), 0, st>>>(p, L, chunk);
        ps.stop();
    }
    return launch_ok("pdef_repair_kernel") ? GM1B_OK : GM1B_ERR_CUDA;
}

extern "C" int32_t gm1b_held_compose(int32_t ni, int32_t nj, int32_t nk, const gm1b_held_arrays *a, float dt,
                                     void *stream) {
    if (a == nullptr || !grid_ok(ni, nj, nk, 1, 1, 1, "gm1b_held_compose") || !(dt > 0.0f)) {
        if (a == nullptr || !(dt > 0.0f)) gm1b_set_error("gm1b_held_compose: need arrays and dt > 0");
        return GM1B_ERR_ARGUMENT;
    }
    Held h{a->th0, a->pi0, a->rho, a->ppi, a->tha, a->qa, a->qpten, a->qtten, a->qvten, a->qcten,
           a->thheld, a->qheld, a->ppten};
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    ProfScope ps("held_compose_kernel", st);
    held_compose_kernel<<<grid_for((size_t)ni * nj * nk), 256, 0, st>>>(h, ni, nj, nk, dt);
    ps.stop();
    return launch_ok("held_compose_kernel") ? GM1B_OK : GM1B_ERR_CUDA;
}

extern "C" int32_t gm1b_solve3_density(int32_t ni, int32_t nj, int32_t nk, const float *rho, const float *c1,
                                       const float *c2, float *rr, float *rf, void *stream) {
    if (!rho || !c1 || !c2 || !rr || !rf || !grid_ok(ni, nj, nk, 1, 1, 3, "gm1b_solve3_density")) {
        if (!rho || !c1 || !c2 || !rr || !rf) gm1b_set_error("gm1b_solve3_density: NULL array");
        return GM1B_ERR_ARGUMENT;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    ProfScope ps("solve3_density_kernel", st);
    solve3_density_kernel<<<grid_for((size_t)ni * nj * (nk + 1)), 256, 0, st>>>(rho, c1, c2, rr, rf, ni, nj, nk);
    ps.stop();
    return launch_ok("solve3_density_kernel") ? GM1B_OK : GM1B_ERR_CUDA;
}

extern "C" int32_t gm1b_pack_scalar(int32_t ni, int32_t nj, int32_t nk, const float *scalar, float *padded,
                                    void *stream) {
    if (!scalar || !padded || !grid_ok(ni, nj, nk, 1, 1, 1, "gm1b_pack_scalar")) {
        if (!scalar || !padded) gm1b_set_error("gm1b_pack_scalar: NULL array");
        return GM1B_ERR_ARGUMENT;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    ProfScope ps("pack_scalar_kernel", st);
    pack_scalar_kernel<<<grid_for((size_t)ni * nj * nk), 256, 0, st>>>(scalar, padded, Lane{ni, nj, nk});
    ps.stop();
    return launch_ok("pack_scalar_kernel") ? GM1B_OK : GM1B_ERR_CUDA;
}

extern "C" int32_t gm1b_bcwsfc(int32_t ni, int32_t nj, int32_t nk, const float *u3d, const float *v3d, float *w3d,
                               const float *gz, const float *dzdx, const float *dzdy, void *stream) {
    if (!u3d || !v3d || !w3d || !gz || !dzdx || !dzdy || !grid_ok(ni, nj, nk, 1, 1, 1, "gm1b_bcwsfc")) {
        if (!u3d || !v3d || !w3d || !gz || !dzdx || !dzdy) gm1b_set_error("gm1b_bcwsfc: NULL array");
        return GM1B_ERR_ARGUMENT;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    ProfScope ps("bcwsfc_kernel", st);
    bcwsfc_kernel<<<grid_for((size_t)ni * nj), 256, 0, st>>>(u3d, v3d, w3d, gz, dzdx, dzdy, Lane{ni, nj, nk});
    ps.stop();
    return launch_ok("bcwsfc_kernel") ? GM1B_OK : GM1B_ERR_CUDA;
}

extern "C" int32_t gm1b_w_level1_fill(int32_t ni, int32_t nj, int32_t nk, float *w3d, void *stream) {
    if (!w3d || !grid_ok(ni, nj, nk, 1, 1, 1, "gm1b_w_level1_fill")) {
        if (!w3d) gm1b_set_error("gm1b_w_level1_fill: NULL array");
        return GM1B_ERR_ARGUMENT;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    for (int pass = 0; pass < 2; ++pass) {
        ProfScope ps("w_level1_fill_kernel", st);
        w_level1_fill_kernel<<<grid_for((size_t)(std::max(ni, nj) + 6) * 6), 256, 0, st>>>(w3d, Lane{ni, nj, nk}, pass);
        ps.stop();
        if (!launch_ok("w_level1_fill_kernel")) return GM1B_ERR_CUDA;
    }
    return GM1B_OK;
}

// ---------------------------------------------------------------------------
// step status: the failure words the reference reads back after a step and
// refuses on (satadj non-convergence, cuda_cartesian_finish.py:638-639; the
// advective Courant stop, gm1_runtime.py:518-549), folded on the device into
// one accumulator so a captured step needs no host read.
// acc: [0] non-converged satadj cells (sum), [1] largest fallout sub-step
// count, [2] blown-up fall columns (sum), [3] largest Courant number (float
// bits; a NaN stays), [4] folds of a Courant number, [5] folds of Kessler words.
// ---------------------------------------------------------------------------
namespace gm1b {
namespace {
__global__ void step_status_fold_kernel(const int32_t *kessler_status, const float *courant, int32_t *acc) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    if (kessler_status != nullptr) {
        acc[0] += kessler_status[0];
        acc[1] = max(acc[1], kessler_status[1]);
        acc[2] += kessler_status[2];
        acc[5] += 1;
    }
    if (courant != nullptr) {
        const float c = *courant;
        const float prev = __int_as_float(acc[3]);
        if (acc[4] == 0 || c != c || (prev == prev && c > prev)) acc[3] = __float_as_int(c);
        acc[4] += 1;
    }
}
}  // namespace
}  // namespace gm1b

extern "C" int32_t gm1b_step_status_fold(const int32_t *kessler_status, const float *courant, int32_t *acc,
                                         void *stream) {
    if (acc == nullptr) {
        gm1b_set_error("gm1b_step_status_fold: NULL accumulator");
        return GM1B_ERR_ARGUMENT;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    ProfScope ps("step_status_fold_kernel", st);
    step_status_fold_kernel<<<1, 32, 0, st>>>(kessler_status, courant, acc);
    ps.stop();
    return launch_ok("step_status_fold_kernel") ? GM1B_OK : GM1B_ERR_CUDA;
}
