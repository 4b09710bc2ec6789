"""The column solves' shared sweep where pivots leave the short reciprocal's
range (2^-125 .. 2^125): it forms such a chunk of rows a second time, with the
rows of the other lanes of the warp.  A level's own vertical factor, which
scales its row of the matrix alone, is made huge at some levels; against the
oracle, every float32 word identical."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

LONG = 2.0 ** 125


def _dev(d):
    return {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in d.items()}


def _same(got, want, names):
    torch.cuda.synchronize()
    for n in names:
        assert np.isfinite(want[n]).all(), n
        assert np.array_equal(got[n].cpu().numpy().view(np.uint32), want[n].view(np.uint32)), n


def _spike(x, size, seed, share=0.2):
    """Scale a share of the words of x up to about ``size``."""
    rng = np.random.default_rng(seed)
    at = rng.random(x.shape) < share
    x[at] = (np.float32(size) * rng.uniform(0.5, 1.0, int(at.sum()))).astype(np.float32)


def _rare(diagonal):
    """Some rows' diagonals lie beyond the short range, some warps' all within."""
    rare = diagonal > LONG
    assert rare.any() and not rare.all()


@pytest.mark.parametrize("flat", [False, True])
@pytest.mark.parametrize("ni,nj,nk", [(33, 8, 8), (64, 7, 19), (7, 9, 40)])
def test_turbt(ni, nj, nk, flat):
    from gm1_b200 import tke_evolution as te
    from oracle import tke_evolution as orc
    from tests.golden.make_golden import tke_evolution_fixture

    a = tke_evolution_fixture(ni, nj, nk, seed=ni + nk)
    _spike(a["mf"], 3e35, nk)
    d = _dev(a)
    g = dict(ni=ni, nj=nj, nk=nk, dx=500.0, dy=450.0, dt=2.0)
    w = lambda n: a[n].astype(np.float64)  # noqa: E731
    c = 2.0 * w("mf")[1:nk] / w("rf")[1:nk]
    up = (w("kmv")[1:nk] + w("kmv")[2:]) * w("mh")[1:] * w("rho")[1:]
    down = (w("kmv")[:nk - 1] + w("kmv")[1:nk]) * w("mh")[:-1] * w("rho")[:-1]
    _rare(c * (up + down))
    if flat:
        orc.tke_diffusion_flat(a, rdz=1.0, **g)
        te.launch_cuda_flat_tke_diffusion(d, rdz=1.0, **g)
    else:
        orc.tke_diffusion(a, dz=1.0, **g)
        te.launch_cuda_tke_diffusion(d, dz=1.0, **g)
    _same(d, a, ("tketen",))


@pytest.mark.parametrize("flat,factor,size,names", [
    (True, "mh", 1.2e34, ("uten", "vten")), (False, "mh", 5e33, ("uten", "vten")),
    (True, "mf", 7e34, ("wten",)), (False, "mf", 3e34, ("wten",))])
@pytest.mark.parametrize("ni,nj,nk", [(33, 4, 8), (31, 5, 18)])
def test_stress_solves(ni, nj, nk, flat, factor, size, names):
    """mh scales the rows of turbu and turbv, mf those of turbw."""
    from gm1_b200 import stress
    from oracle import stress as ost
    from tests.test_stress_gpu import _inputs
    from tests.test_stress_terrain_gpu import _stress_inputs

    g = dict(ni=ni, nj=nj, nk=nk, dx=100.0, dy=90.0, dt=16.0 if factor == "mh" else 1.0)
    a = _inputs(ni, nj, nk, nk)[0] if flat else _stress_inputs(ni, nj, nk, nk)
    for n in ("u3d", "v3d", "w3d"):
        a[n] *= np.float32(0.01)
    # whole levels, so that both cells of a wind's column scale alike
    a[factor][np.random.default_rng(nk).permutation(np.arange(1, nk - 1))[:nk // 3]] *= np.float32(size)
    w = lambda n: a[n].astype(np.float64)  # noqa: E731
    if factor == "mh":  # a u column's cells
        pair = lambda n: w(n)[:, :, 1:] + w(n)[:, :, :-1]  # noqa: E731
        face = (pair("kmv") * pair("mf") * pair("rf"))[1:nk]
        _rare(0.0625 * g["dt"] * (face[:-1] + face[1:]) * (pair("mh") * 2.0 / pair("rho"))[1:nk - 1])
    else:
        mass = w("mh") * w("rho") * (w("kmh")[:-1] + w("kmh")[1:])
        _rare(g["dt"] * (mass[:-1] + mass[1:]) * (w("mf") / w("rf"))[1:nk])
    d = _dev(a)
    if flat:
        ost.flat_momentum_stress(a, rdz=1.0, **g)
        stress.launch_cuda_flat_momentum_stress(d, rdz=1.0, **g)
    else:
        grid = dict(ni=ni, nj=nj, nk=nk)
        ost.terrain_strain(a, **grid, dx=g["dx"], dy=g["dy"], dz=1.0)
        ost.terrain_gettau(a, **grid)
        ost.terrain_momentum_stress(a, dz=1.0, **g)
        stress.launch_cuda_terrain_strain(d, **grid, dx=g["dx"], dy=g["dy"], dz=1.0)
        stress.launch_cuda_terrain_stress(d, dz=1.0, **g)
    _same(d, a, names)


@pytest.mark.parametrize("ni,nj,nk,size", [(33, 3, 9, 1.5e34), (5, 4, 40, 3e34)])
def test_acoustic_column_pass(ni, nj, nk, size):
    """The flat column's mf(k) scales the row of w level k; little wind and
    pressure keep the right sides finite beside it."""
    from gm1_b200 import terrain_open as tos
    from gm1_b200.momentum import StretchedMomentumColumn
    from oracle import terrain_open as orc
    from tests.golden.make_golden import terrain_open_fixture
    from tests.test_oracle_momentum import _padded_rho0

    a, m = terrain_open_fixture(ni, nj, nk, ni + nk)
    for names, scale in ((("ppterm",), 1e3), (("ppi", "pp3d", "ppx", "ppten", "ppd"), 1e-3),
                         (("ua", "u3d", "va", "v3d", "wa", "w3d", "uten", "vten", "wten", "radbcw", "radbce", "radbcs",
                           "radbcn"), 1e-4)):
        for n in names:
            a[n] *= np.float32(scale)
    rng = np.random.default_rng(nk)
    mh, mf = rng.uniform(0.3, 3.0, nk + 2).astype(np.float32), rng.uniform(0.3, 3.0, nk + 3).astype(np.float32)
    mf[rng.permutation(np.arange(2, nk))[:nk // 3]] *= np.float32(size)
    d, md = _dev(a), _dev(m)
    for n in tos.COLUMN_DIAGNOSTIC_NAMES:
        d[n] = torch.zeros(1, device="cuda")
    md["rho0_padded"] = torch.from_numpy(_padded_rho0(m["rho0_3d"], ni, nj, nk)).cuda()
    vertical = StretchedMomentumColumn(True, None, mh=torch.from_numpy(mh).cuda(), mf=torch.from_numpy(mf).cuda(),
                                       rdz=0.01)
    kw = dict(ni=ni, nj=nj, nk=nk, nrk=1, dt=2.0, nsound=4, dx=450.0, dy=520.0)
    orc.terrain_open_stage_flat(a, m, {"mh": mh, "mf": mf, "rdz": 0.01}, **kw)
    _rare(np.abs(a["tri_pivot"][2:nk + 1, 1:nj + 1, 1:ni + 1]))
    tos.launch_cuda_gm1_child_psolver3_open_stage(
        d, md, vertical=vertical, compiled=tos.compile_cuda_psolver3_terrain_open(retain_column_diagnostics=False), **kw)
    _same(d, a, [n for n in tos.COMPARE_OUTPUT_NAMES if not n.startswith("tri_")])
