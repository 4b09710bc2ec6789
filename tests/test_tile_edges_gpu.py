"""The marching kernels at the sizes where their tiles can go wrong: the
edges of the 31- and 32-wide tiles and of the 4-, 7- and 8-row blocks, runs
of levels that do not divide the column, the shortest columns.  Against the
oracle, every float32 word identical."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _dev(d):
    return {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in d.items()}


def _differ(got, want, names):
    torch.cuda.synchronize()
    return [n for n in names if not np.array_equal(got[n].cpu().numpy().view(np.uint32), want[n].view(np.uint32))]


def _t(x):
    return torch.from_numpy(np.array(x, dtype=np.float32)).cuda()


def _profiles(nk):
    rng = np.random.default_rng(nk)
    return dict(mh=rng.uniform(0.3, 3.0, nk + 2).astype(np.float32), mf=rng.uniform(0.3, 3.0, nk + 3).astype(np.float32),
                rdz=float(np.float32(1.0) / np.float32(100.0)))


@pytest.mark.parametrize("column", ["uniform", "terrain", "flat"])
@pytest.mark.parametrize("ni,nj,nk", [(31, 4, 4), (32, 3, 7), (33, 5, 8), (64, 3, 9), (65, 4, 17), (3, 3, 160)])
def test_compact_acoustic_stage(column, ni, nj, nk):
    """The column pass that marches runs of levels, without diagnostics."""
    from gm1_b200 import terrain_open as tos
    from gm1_b200.momentum import StretchedMomentumColumn
    from gm1_b200.vertical import uniform_vertical_levels
    from oracle import terrain_open as orc
    from tests.golden.make_golden import terrain_open_fixture
    from tests.test_oracle_momentum import _padded_rho0

    a, m = terrain_open_fixture(ni, nj, nk, 40 + ni + nk)
    ref = {k: v.copy() for k, v in a.items()}
    dev, mdev = _dev(a), _dev(m)
    kw = dict(ni=ni, nj=nj, nk=nk, dt=2.0, nsound=6, dx=450.0, dy=520.0)
    compiled = tos.compile_cuda_psolver3_terrain_open(retain_column_diagnostics=False)
    for n in tos.COLUMN_DIAGNOSTIC_NAMES:
        dev[n] = torch.zeros(1, device="cuda")
    rho0p = _padded_rho0(m["rho0_3d"], ni, nj, nk)
    mdev["rho0_padded"] = _t(rho0p)
    if column == "flat":
        p = _profiles(nk)
        vertical = StretchedMomentumColumn(True, None, mh=_t(p["mh"]), mf=_t(p["mf"]), rdz=p["rdz"])
    elif column == "terrain":
        lv = uniform_vertical_levels(nk, 210.0)
        p = {"sigma": lv.sigma, "sigmaf": lv.sigmaf, "rds": lv.rds, "rdsf": lv.rdsf, "ztop": lv.ztop_m, "rho0p": rho0p}
        vertical = StretchedMomentumColumn(False, None, **{n: _t(p[n]) for n in ("sigma", "sigmaf", "rds", "rdsf")},
                                           ztop=lv.ztop_m)
    for nrk in (1, 2, 3):
        if column == "uniform":
            orc.terrain_open_stage(ref, m, nrk=nrk, dz=210.0, **kw)
            tos.launch_cuda_psolver3_terrain_open_stage(dev, mdev, nrk=nrk, dz=210.0, compiled=compiled, **kw)
        else:
            (orc.terrain_open_stage_flat if column == "flat" else orc.terrain_open_stage_column)(ref, m, p, nrk=nrk, **kw)
            tos.launch_cuda_gm1_child_psolver3_open_stage(dev, mdev, nrk=nrk, vertical=vertical, compiled=compiled, **kw)
        names = [n for n in tos.COMPARE_OUTPUT_NAMES if not n.startswith("tri_")] + ["scalar"]
        assert _differ(dev, ref, names) == [], nrk


@pytest.mark.parametrize("nrk", [1, 3])
@pytest.mark.parametrize("ni,nj,nk,chunk", [(30, 8, 8, None), (31, 13, 9, 4), (32, 14, 11, 5), (61, 15, 8, 1),
                                            (62, 9, 21, None), (8, 8, 40, 7), (124, 8, 8, None), (248, 9, 9, 5)])
def test_scalar_advection(ni, nj, nk, chunk, nrk):
    """Open sides with the face fluxes written, each word of the tendency and
    the fluxes (the warps' shared faces among them)."""
    from gm1_b200.advection import launch_cuda_scalar_advection5, padded_shapes
    from oracle import advection as adv

    rng = np.random.default_rng(ni + nk)
    sh = padded_shapes(ni, nj, nk)
    f = lambda s, lo, hi: rng.uniform(lo, hi, s).astype(np.float32)  # noqa: E731
    h = {"scalar": f(sh["scalar"], -1, 1), "rru": f(sh["u"], -9, 9), "rrv": f(sh["v"], -9, 9), "rrw": f(sh["w"], -2, 2),
         "c1": f(sh["face"], 0.3, 0.7), "c2": f(sh["face"], 0.3, 0.7), "rr0": f(sh["cell"], 0.8, 3.0),
         "gz": f((nj, ni), 0.8, 1.2), "divx": f(sh["cell"], -1e-3, 1e-3), "tendency": np.zeros(sh["cell"], np.float32),
         "flux_x": np.zeros(sh["u"], np.float32), "flux_y": np.zeros(sh["v"], np.float32),
         "flux_z": np.zeros(sh["w"], np.float32)}
    h["scalar"][:, :, : ni // 2] = 0.0  # whole stencils of zeros, and edges of them
    d = _dev(h)
    kw = dict(ni=ni, nj=nj, nk=nk, nrk=nrk, dx=400.0, dy=350.0, dz=150.0, weps=1.0e-20)
    adv.scalar_advection5(h, lateral_obc=0x2222, **kw)
    launch_cuda_scalar_advection5(
        d["scalar"], {k: d[k] for k in ("rru", "rrv", "rrw")}, {k: d[k] for k in ("c1", "c2", "rr0", "gz")}, d["divx"],
        d["tendency"], {q: d["flux_" + q] for q in "xyz"}, lateral_sides=(2, 2, 2, 2), levels_per_chunk=chunk, **kw)
    assert _differ(d, h, ("tendency", "flux_x", "flux_y", "flux_z")) == []


@pytest.mark.parametrize("sides", [(2, 2, 2, 2), (1, 1, 1, 1)])
@pytest.mark.parametrize("ni,nj,nk", [(30, 7, 8), (31, 8, 9), (32, 9, 10), (62, 11, 13), (63, 12, 33),
                                      (33, 800, 9), (32, 1200, 17)])
def test_momentum_advection(ni, nj, nk, sides):
    from gm1_b200 import momentum as mom
    from oracle import momentum as orc
    from tests.golden.make_golden import momentum_fixture
    from tests.test_oracle_momentum import OUTS

    a, m, _ = momentum_fixture(ni, nj, nk, 7 * ni + nk)
    kw = dict(ni=ni, nj=nj, nk=nk, dx=500.0, dy=450.0, dz=150.0, lateral_sides=sides)
    dev = _dev({**a, **m})
    out = mom.launch_cuda_terrain_open_momentum_advection5(dev, dev, nrk=1, **kw)
    ref = {**a, **m, "divx": np.zeros((nk, nj, ni), np.float32)}
    orc.momentum_advection5(ref, **kw)
    assert _differ({**dev, "divx": out.divx}, ref, OUTS) == []


@pytest.mark.parametrize("ni,nj,nk", [(31, 8, 2), (33, 9, 3), (33, 800, 9), (32, 1200, 17), (2, 17, 2), (15, 33, 5),
                                      (16, 32, 24), (17, 32, 24), (48, 16, 9), (33, 64, 40), (9, 500, 33), (16, 4000, 9)])
def test_column_marches(ni, nj, nk):
    """Buoyancy and the post-acoustic divergences, which march one, two, four
    or eight levels a thread, in CTAs of 32 and of 16 columns."""
    from gm1_b200 import moist_ops as mo
    from oracle import moist_step as om
    from tests.golden.make_golden import moist_piece_fixture

    g = dict(ni=ni, nj=nj, nk=nk)
    a = moist_piece_fixture(ni, nj, nk, 3 * ni + nk)
    for n in ("divergence", "theta_divergence_term"):
        a[n] = np.zeros((nk, nj, ni), np.float32)
    d = _dev(a)
    names = ("dum8", "c1", "c2", "gxu", "gyv", "uten", "vten", "wten")
    om.moist_buoyancy(*(a[n] for n in names), **g)
    mo.moist_buoyancy(*(d[n] for n in names), **g)
    assert _differ(d, a, ("uten", "vten", "wten")) == []
    om.moist_buoyancy_flat(a["dum8"], a["c1"], a["c2"], a["wten"], **g)
    mo.moist_buoyancy_flat(d["dum8"], d["c1"], d["c2"], d["wten"], **g)
    om.post_acoustic_flux(a, **g, dx=400.0, dy=350.0, dz=180.0)
    mo.post_acoustic_flux(d, **g, dx=400.0, dy=350.0, dz=180.0)
    assert _differ(d, a, ("wten", "rru", "rrv", "rrw", "divergence", "theta_divergence_term", "divx")) == []


def test_column_marches_of_more_chunks_than_a_grid_takes():
    """2x2 columns whose chunks of eight levels exceed a grid dimension's
    65535: the whole column against the same columns cut in two."""
    from gm1_b200 import moist_ops as mo

    ni, nj, nk, cut = 2, 2, 524300, 262144
    g = torch.Generator(device="cuda").manual_seed(1)
    r = lambda *s: torch.rand(*s, generator=g, device="cuda")  # noqa: E731
    a = {"dum8": r(nk + 2, 8, 8), "c1": r(nk + 1, 2, 2), "c2": r(nk + 1, 2, 2), "wten": r(nk + 3, 8, 8)}
    parts = []
    for lo, hi in ((1, cut + 1), (cut, nk)):  # two levels in common: the faces at either end are not formed
        p = {n: a[n][lo - 1:hi + k].contiguous() for n, k in (("dum8", 2), ("c1", 1), ("c2", 1), ("wten", 3))}
        mo.moist_buoyancy_flat(*p.values(), ni=ni, nj=nj, nk=hi - lo + 1)
        parts.append(p["wten"])
    mo.moist_buoyancy_flat(*a.values(), ni=ni, nj=nj, nk=nk)
    want = torch.cat((parts[0][:cut + 1], parts[1][2:]))
    assert torch.equal(a["wten"], want)


@pytest.mark.parametrize("flat", [False, True])
@pytest.mark.parametrize("ni,nj,nk", [(30, 7, 8), (31, 8, 9), (32, 14, 11), (62, 15, 12), (7, 9, 40),
                                      (124, 7, 8), (248, 8, 9), (30, 147, 23), (30, 148, 23)])
def test_tke_stages(ni, nj, nk, flat):
    from gm1_b200 import tke_evolution as te
    from oracle import tke_evolution as orc
    from tests.golden.make_golden import tke_evolution_fixture

    a = tke_evolution_fixture(ni, nj, nk, seed=ni + nk)
    dev = _dev(a)
    ws, p = torch.empty_like(dev["tke3d"]), _profiles(nk)
    kw = dict(ni=ni, nj=nj, nk=nk, dx=500.0, dy=450.0, dt=2.0)
    for nrk in (1, 2, 3):
        nxt = np.zeros_like(a["tke3d"])
        if flat:
            orc.tke_rk_stage_flat(a, p["mf"], a["tke3d"], nxt, nrk=nrk, rdz=p["rdz"], **kw)
            te.launch_cuda_flat_tke_rk_stage(dev, mf_profile=_t(p["mf"]), workspace=ws, nrk=nrk, rdz=p["rdz"], **kw)
        else:
            orc.tke_rk_stage(a, a["tke3d"], nxt, nrk=nrk, dz=150.0, **kw)
            te.launch_cuda_tke_rk_stage(dev, workspace=ws, nrk=nrk, dz=150.0, **kw)
        a["tke3d"] = nxt
        assert _differ(dev, a, ("tke3d",)) == [], nrk


@pytest.mark.parametrize("ni,nj,nk", [(31, 7, 8), (32, 8, 9), (33, 7, 10), (7, 7, 17), (8, 9, 201)])
def test_flat_tke_diffusion(ni, nj, nk):
    from gm1_b200 import tke_evolution as te
    from oracle import tke_evolution as orc
    from tests.golden.make_golden import tke_evolution_fixture

    a = tke_evolution_fixture(ni, nj, nk, seed=3 * ni + nk)
    dev = _dev(a)
    kw = dict(ni=ni, nj=nj, nk=nk, dx=500.0, dy=450.0, rdz=_profiles(nk)["rdz"], dt=2.0)
    orc.tke_diffusion_flat(a, **kw)
    te.launch_cuda_flat_tke_diffusion(dev, **kw)
    assert _differ(dev, a, ("tketen",)) == []


@pytest.mark.parametrize("ni,nj,nk", [(31, 7, 8), (32, 8, 9), (33, 7, 10), (7, 7, 17), (8, 9, 201),
                                      (7, 1332, 8), (33, 666, 9), (31, 1340, 10), (7, 1331, 9), (7, 1332, 64),
                                      (7, 1332, 65)])
def test_terrain_tke_diffusion(ni, nj, nk):
    """Columns to a CTA, the eight warps' and the three warps' runs of levels."""
    from gm1_b200 import tke_evolution as te
    from oracle import tke_evolution as orc
    from tests.golden.make_golden import tke_evolution_fixture

    a = tke_evolution_fixture(ni, nj, nk, seed=3 * ni + nk)
    dev = _dev(a)
    kw = dict(ni=ni, nj=nj, nk=nk, dx=500.0, dy=450.0, dz=150.0, dt=2.0)
    orc.tke_diffusion(a, **kw)
    te.launch_cuda_tke_diffusion(dev, **kw)
    assert _differ(dev, a, ("tketen",)) == []


@pytest.mark.parametrize("ni,nj,nk,numq", [(31, 3, 7, 2), (32, 4, 8, 3), (33, 3, 9, 4), (64, 3, 17, 5), (3, 5, 200, 6),
                                           (3, 1332, 4, 1), (31, 1331, 5, 1), (33, 666, 7, 1), (4, 1332, 40, 1),
                                           (4, 1332, 41, 1)])
def test_flat_turbulence_columns(ni, nj, nk, numq):
    """Runs of levels of the stress and scalar solves, and the scalars'
    groups of four."""
    from gm1_b200 import stress
    from oracle import stress as ost
    from tests.test_stress_gpu import _inputs, _turbs_inputs

    g = dict(ni=ni, nj=nj, nk=nk, dx=100.0, dy=90.0, dt=0.6)
    a, rdz = _inputs(ni, nj, nk, ni + nk)
    rng = np.random.default_rng(nk)
    for n in ost.TAU_NAMES:
        a[n][:] = rng.normal(0.0, 1.0, a[n].shape)
    d = _dev(a)
    ost.flat_momentum_stress(a, **g, rdz=rdz)
    stress.launch_cuda_flat_momentum_stress(d, **g, rdz=rdz)
    assert _differ(d, a, ost.TENDENCY_NAMES) == []
    a, dz = _turbs_inputs(ni, nj, nk, numq, ni + nk)
    d = _dev(a)
    d["workspace"] = stress.scalar_turbulence_workspace(ni, nj, nk, numq, d["tha"].device)
    ost.flat_scalar_turbulence(a, **g, numq=numq, dz=dz)
    stress.launch_cuda_flat_scalar_turbulence(d, **g, numq=numq, dz=dz)
    assert _differ(d, a, ("thten1", "qten")) == []


@pytest.mark.parametrize("ni,nj,nk,numq", [(31, 3, 7, 2), (32, 8, 8, 3), (33, 7, 9, 4), (64, 3, 17, 5), (3, 5, 200, 6)])
def test_terrain_turbulence_columns(ni, nj, nk, numq):
    from gm1_b200 import stress
    from oracle import stress as ost
    from tests.test_stress_terrain_gpu import _stress_inputs, _turbs_inputs

    g = dict(ni=ni, nj=nj, nk=nk, dx=1000.0, dy=900.0, dz=250.0)
    a = _stress_inputs(ni, nj, nk, ni + nk)
    rng = np.random.default_rng(nk)
    for n in ost.STRAIN_NAMES:
        a[n][:] = rng.normal(0.0, 1.0, a[n].shape)
    d = _dev(a)
    ost.terrain_gettau(a, ni=ni, nj=nj, nk=nk)
    ost.terrain_momentum_stress(a, **g, dt=5.0)
    stress.launch_cuda_terrain_stress(d, **g, dt=5.0)
    assert _differ(d, a, ("uten", "vten", "wten")) == []
    a = _turbs_inputs(ni, nj, nk, ni + nk)
    d = _dev(a)
    d["workspace"] = stress.terrain_scalar_turbulence_workspace(ni, nj, nk, numq, d["tha"].device)
    ost.terrain_scalar_turbulence(a, **g, numq=numq, dt=5.0)
    stress.launch_cuda_terrain_scalar_turbulence(d, **g, numq=numq, dt=5.0)
    assert _differ(d, a, ("thten1", "qten")) == []


@pytest.mark.parametrize("ni,nj,nk", [(31, 3, 1), (32, 2, 7), (33, 5, 8), (65, 2, 9), (5, 3, 296), (5, 3, 297)])
def test_kessler_columns(ni, nj, nk):
    """Columns in shared memory (up to 296 levels) and a thread per column:
    the sub-step counts and the level-ordered sums are the oracle's."""
    from oracle import kessler as ko
    from tests.golden.make_golden import kessler_fixture
    from tests.test_kessler_gpu import run_gpu
    from tests.kessler_common import assert_budgets_close, assert_fields_close

    dz = 100.0 if nk < 100 else 20.0
    meta = dict(ni=ni, nj=nj, nk=nk, dx=1000.0, dy=1000.0, dz=dz, dt=0.2 * dz, eqtset=2)
    inputs = kessler_fixture(ni, nj, nk, dz, ni + nk)
    want = {k: v.copy() for k, v in inputs.items()}
    nfall = np.zeros((nj, ni), np.int32)
    ko.kessler_driver(want, **meta, nfall=nfall)
    got, _, nf, _ = run_gpu(inputs, meta)
    assert np.array_equal(nf, nfall)
    assert_fields_close(want, got)
    assert np.array_equal(got["asq"].view(np.uint64), want["asq"].view(np.uint64))
    assert_budgets_close(want["qbudget"], got["qbudget"])


@pytest.mark.parametrize("flat", [False, True])
@pytest.mark.parametrize("ni,nj,nk", [(31, 7, 9), (32, 8, 10), (30, 6, 18), (3, 3, 3), (63, 15, 20)])
def test_deformation(ni, nj, nk, flat):
    """Runs of levels of the strains' march."""
    from gm1_b200 import closure
    from oracle import closure as orc
    from tests.golden.make_golden import deformation_fixture

    a = deformation_fixture(ni, nj, nk, seed=3 * ni + nk)
    dx, dy, dz = (float(x) for x in a.pop("_spacing"))
    g = dict(ni=ni, nj=nj, nk=nk, dx=dx, dy=dy)
    if flat:
        p = _profiles(nk)
        a["mf"] = np.random.default_rng(nk).uniform(0.3, 3.0, (nk + 1, nj, ni)).astype(np.float32)
        a["mh_profile"] = p["mh"]
        a = {n: a[n] for n in orc.FLAT_DEFORMATION_INPUTS + ("defv", "defh")}
        dev = _dev(a)
        orc.flat_calcdef(a, **g, rdz=p["rdz"])
        mh = dev.pop("mh_profile")
        closure.launch_cuda_flat_deformation(dev, mh_profile=mh, **g, rdz=p["rdz"])
    else:
        dev = _dev(a)
        orc.calcdef(a, **g, dz=dz)
        closure.launch_cuda_terrain_deformation(dev, **g, dz=dz)
    assert _differ(dev, a, ("defv", "defh")) == []


@pytest.mark.parametrize("column", ["uniform", "terrain", "flat"])
@pytest.mark.parametrize("obc,pdefweno", [(0x2222, 0), (0x2222, 1), (0x1111, 1), (0x3443, 0)])
@pytest.mark.parametrize("ni,nj,nk", [(29, 7, 4), (30, 8, 5), (31, 9, 6), (61, 14, 9), (5, 15, 33), (62, 7, 5),
                                      (124, 8, 4)])
def test_pdef_advection_is_the_chains(ni, nj, nk, obc, pdefweno, column):
    """The two-pass moisture advection against the chain's, with negative
    candidates on every axis and dry air beside the water."""
    from gm1_b200 import moist_ops as mo
    from gm1_b200.advection import StretchedColumn
    from tests.test_oracle_moist_step import chain_arrays

    a = chain_arrays(ni, nj, nk, ni + nk)
    rng = np.random.default_rng(nk)
    dry = rng.random(a["scalar_a"].shape) < 0.4
    a["scalar_a"][dry] = 0.0
    a["scalar_padded"][1:nk + 1, 3:nj + 3, 3:ni + 3][dry] = 0.0
    one = _dev(a)
    two = {k: v.clone() for k, v in one.items()}
    kw = dict(ni=ni, nj=nj, nk=nk, dttmp=2.0, dx=400.0, dy=300.0, weps=1e-20, lateral_obc=obc, pdefweno=pdefweno)
    p = _profiles(nk)
    if column == "uniform":
        mo.pdef_moisture_chain(one, dz=200.0, **kw)
        mo.pdef_moisture_advection(two, dz=200.0, **kw)
    else:
        col = StretchedColumn(True, mh=_t(p["mh"]), rdz=p["rdz"]) if column == "flat" else \
            StretchedColumn(False, rdsf=_t(np.abs(p["mf"]) / 100.0))
        mo.pdef_moisture_chain_column(one, col, **kw)
        mo.pdef_moisture_advection(two, col, **kw)
    torch.cuda.synchronize()
    want = {k: v.cpu().numpy() for k, v in one.items()}
    assert np.count_nonzero(want["candidate"] < 0.0) > 0
    assert _differ(two, want, ("advection",)) == []


@pytest.mark.parametrize("nrk", [1, 3])
@pytest.mark.parametrize("ni,nj,nk", [(8, 8, 8), (9, 33, 9), (34, 9, 12), (65, 10, 17), (28, 44, 9), (42, 42, 9),
                                      (43, 43, 9)])
def test_advection_adjoint_in_one_pass(ni, nj, nk, nrk):
    """An output that overlaps the tendency adjoint takes the two passes over
    the face scratch: the fifth-order words are those of the one pass; and the
    edge cells sum the carrier adjoint's words."""
    from gm1_b200 import adjoint as adj
    from tests.test_adjoint_gpu import _flow, warm_rain_case

    state, fr, g = warm_rain_case(ni=ni, nj=nj, nk=nk, seed=ni + nk)
    flow = _flow(fr, g)
    s, rng = _t(state["qv"]), np.random.default_rng(nj)
    lam = _t(rng.standard_normal((nk, nj, ni)))
    got = adj.advection_tendency_adjoint(flow, s, lam, nrk)
    in_place = lam.clone()
    assert torch.equal(adj.advection_tendency_adjoint(flow, s, in_place, nrk, out=in_place), got)
    padded = adj.advection_carrier_adjoint(flow, adj._carrier(flow, s), lam, nrk)
    assert torch.equal(padded[1:-1, 4:-4, 4:-4], got[:, 1:-1, 1:-1])
    west = padded[1:-1, 4:-4, :4].double().sum(-1)
    # four float32 words of at most the largest one's size
    assert torch.allclose(west, got[:, 1:-1, 0].double(), rtol=0.0, atol=float(padded.abs().max()) * 2.0 ** -21)


@pytest.mark.parametrize("name", ["c1", "c2"])
@pytest.mark.parametrize("running", [False, True])
def test_advection_adjoint_over_its_face_weights(name, running):
    """An output over c1 or c2, which the cells beside the column's ends read
    at their neighbours' levels, takes the two passes."""
    import dataclasses

    from gm1_b200 import adjoint as adj
    from tests.test_adjoint_gpu import _flow, warm_rain_case

    ni, nj, nk = 34, 9, 12
    state, fr, g = warm_rain_case(ni=ni, nj=nj, nk=nk, seed=3)
    flow = _flow(fr, g)
    s, lam = _t(state["qv"]), _t(np.random.default_rng(4).standard_normal((nk, nj, ni)))
    got = adj.advection_tendency_adjoint(flow, s, lam, 1)
    over = flow.fields[name].clone()
    flow = dataclasses.replace(flow, fields={**flow.fields, name: over})
    if running:
        adj.advection_tendency_adjoint(flow, s, lam, 1, accumulate=torch.zeros_like(lam), running_sum=over[:nk])
    else:
        adj.advection_tendency_adjoint(flow, s, lam, 1, out=over[:nk])
    assert torch.equal(over[:nk], got)


def _columns(nk, rho0p):
    """The terrain and the flat stretched column: the profiles for the oracle
    and their device form."""
    from gm1_b200.momentum import StretchedMomentumColumn
    from gm1_b200.vertical import uniform_vertical_levels

    lv, p = uniform_vertical_levels(nk, 150.0), _profiles(nk)
    names = ("sigma", "sigmaf", "rds", "rdsf")
    shape = (nk, rho0p.shape[1] - 6, rho0p.shape[2] - 6)
    rr0 = np.random.default_rng(nk).uniform(0.8, 1.4, shape).astype(np.float32)
    terrain = {"flat": False, "rho0p": rho0p, **{n: getattr(lv, n) for n in names}, "ztop": lv.ztop_m, "mh": lv.mh,
               "mf": lv.mf, "rr0": rr0, "rdz": p["rdz"]}
    flat = {"flat": True, "rho0p": rho0p, **dict.fromkeys(names), "ztop": 0.0, "mh": p["mh"], "mf": p["mf"], "rr0": rr0,
            "rdz": p["rdz"]}
    return {"terrain": (terrain, StretchedMomentumColumn(False, _t(rho0p), ztop=lv.ztop_m,
                                                         **{n: _t(terrain[n]) for n in names})),
            "flat": (flat, StretchedMomentumColumn(True, _t(rho0p), mh=_t(p["mh"]), mf=_t(p["mf"]), rr0=_t(rr0),
                                                   rdz=p["rdz"]))}


@pytest.mark.parametrize("column", ["terrain", "flat"])
@pytest.mark.parametrize("sides", [(2, 2, 2, 2), (1, 1, 3, 2)])
@pytest.mark.parametrize("ni,nj,nk", [(30, 7, 8), (31, 8, 9), (33, 9, 21), (62, 13, 10), (32, 1200, 9)])
def test_momentum_advection_on_a_column(ni, nj, nk, sides, column):
    from gm1_b200 import momentum as mom
    from oracle import momentum as orc
    from tests.golden.make_golden import momentum_fixture
    from tests.test_oracle_momentum import OUTS, _padded_rho0

    a, m, _ = momentum_fixture(ni, nj, nk, 7 * ni + nk)
    ref = {**a, **m, "divx": np.zeros((nk, nj, ni), np.float32)}
    host, vertical = _columns(nk, _padded_rho0(m["rho0_3d"], ni, nj, nk))[column]
    d = _dev(ref)
    kw = dict(ni=ni, nj=nj, nk=nk, dx=500.0, dy=450.0, lateral_sides=sides)
    orc.momentum_advection5_column(ref, host, **kw)
    mom.launch_cuda_gm1_child_stretched_momentum5(d, d, vertical, nrk=1, divx=d["divx"], **kw)
    assert _differ(d, ref, OUTS) == []


@pytest.mark.parametrize("column", ["terrain", "flat"])
@pytest.mark.parametrize("ni,nj,nk", [(31, 8, 4), (33, 9, 5), (2, 17, 4), (16, 32, 24), (33, 800, 9), (9, 500, 33)])
def test_post_acoustic_marches_on_a_column(ni, nj, nk, column):
    from gm1_b200 import moist_ops as mo
    from oracle import moist_step as om
    from tests.golden.make_golden import moist_piece_fixture
    from tests.test_oracle_momentum import _padded_rho0

    a = moist_piece_fixture(ni, nj, nk, 3 * ni + nk)
    for n in ("divergence", "theta_divergence_term"):
        a[n] = np.zeros((nk, nj, ni), np.float32)
    host, vertical = _columns(nk, _padded_rho0(a["rho0_3d"], ni, nj, nk))[column]
    d = _dev(a)
    om.post_acoustic_flux_column(a, host, ni=ni, nj=nj, nk=nk, dx=400.0, dy=350.0)
    mo.post_acoustic_flux_column(d, vertical, ni=ni, nj=nj, nk=nk, dx=400.0, dy=350.0)
    assert _differ(d, a, ("rru", "rrv", "rrw", "divergence", "theta_divergence_term", "divx")) == []


@pytest.mark.parametrize("column", ["terrain", "flat"])
@pytest.mark.parametrize("nrk", [1, 3])
@pytest.mark.parametrize("ni,nj,nk,chunk", [(30, 8, 8, None), (31, 13, 9, 4), (32, 14, 11, 5), (62, 9, 21, None)])
def test_scalar_advection_on_a_column(ni, nj, nk, chunk, nrk, column):
    from gm1_b200.advection import (StretchedColumn, launch_cuda_gm1_child_stretched_scalar_advection5, padded_shapes)
    from oracle import advection as adv

    rng = np.random.default_rng(ni + nk)
    sh, p = padded_shapes(ni, nj, nk), _profiles(nk)
    f = lambda s, lo, hi: rng.uniform(lo, hi, s).astype(np.float32)  # noqa: E731
    h = {"scalar": f(sh["scalar"], -1, 1), "rru": f(sh["u"], -9, 9), "rrv": f(sh["v"], -9, 9), "rrw": f(sh["w"], -2, 2),
         "c1": f(sh["face"], 0.3, 0.7), "c2": f(sh["face"], 0.3, 0.7), "rr0": f(sh["cell"], 0.8, 3.0),
         "gz": f((nj, ni), 0.8, 1.2), "divx": f(sh["cell"], -1e-3, 1e-3), "tendency": np.zeros(sh["cell"], np.float32),
         **{"flux_" + q: np.zeros(sh[s], np.float32) for q, s in zip("xyz", "uvw")}}
    d = _dev(h)
    kw = dict(ni=ni, nj=nj, nk=nk, nrk=nrk, dx=400.0, dy=350.0, weps=1.0e-20)
    flat = column == "flat"
    profile = p["mh"] if flat else p["mf"] / np.float32(100.0)
    adv.scalar_advection5_column(h, flat=flat, profile=profile, rdz=p["rdz"], lateral_obc=0x2222, **kw)
    launch_cuda_gm1_child_stretched_scalar_advection5(
        d["scalar"], d, d, d["divx"], d["tendency"], None if chunk else {q: d["flux_" + q] for q in "xyz"},
        StretchedColumn(True, mh=_t(profile), rdz=p["rdz"]) if flat else StretchedColumn(False, rdsf=_t(profile)),
        lateral_sides=(2, 2, 2, 2), levels_per_chunk=chunk, write_fluxes=chunk is None, **kw)
    assert _differ(d, h, ("tendency",) if chunk else ("tendency", "flux_x", "flux_y", "flux_z")) == []
