"""Branches that only launches of many columns or rows reach, against the oracle: tracers in the semi-implicit kernel of
four columns per warp, hybrid coordinates in the fixer reduction of larger grids, and the flux, kinetic-energy
and height prologues of the register-split FP64 FFT (one-layer models of several members).  First and last
member; tolerances: those of the same steps with one member (test_gpu_models, test_gpu_tracers)."""
import numpy as np
import pytest

from jgcm import configs
from test_gpu_models import MIXED_TOL, _compare
from test_gpu_tracers import _synth, _tracer_fields
from test_gpu_transforms import _meshes

pytestmark = pytest.mark.gpu


def _developed(orc, om, params, **kw):
    omod = orc.Model(om, params, **kw)
    omod.spectral_initialize_fields(configs.hs_temperature_noise(om), True)
    configs.add_hs_flow(orc, om, omod)
    return omod


@pytest.mark.parametrize("nd,members", [(9, 56), (20, 58)])
def test_tracers_in_many_members(jg, orc, nd, members):
    """from 100 (mode, member) columns per SM on; the last warp ragged"""
    gm, om = _meshes(jg, orc, 21, 32, 64, nd, "fp32")
    assert 275 * members >= 100 * jg.device_info()["sm_count"]
    params = configs.PARAMS["hs_t21l10"]
    omod = _developed(orc, om, params, num_tracers=2)
    one = jg.Model(gm, params, num_tracers=2)
    configs.copy_state(omod, one, "held_suarez")
    spe = _tracer_fields(om, omod)
    grid = _synth(orc, om, spe)
    for md in (one, omod):
        md.set("spe_tracers_c", spe)
        md.set("spe_tracers_p", spe)
        md.set("grid_tracers_c", grid)
    ens = jg.Model(gm, params, members=members, num_tracers=2)
    for e in range(members):
        ens.copy_member(e, one)
    ens.step(3)
    omod.step(3)
    for e in (0, members - 1):
        one.copy_member(0, ens, e)
        _compare(one, omod, "held_suarez", MIXED_TOL["fp32"])
        for f in ("spe_tracers_c", "spe_tracers_p", "grid_tracers_c", "grid_tracers_p"):
            a, b = one.get(f), omod.get(f)
            for i in range(2):
                assert configs.rel_l2(a[..., i], b[..., i]) < 1e-5, (e, f, i)


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-10), ("fp32", MIXED_TOL["fp32"])])
@pytest.mark.parametrize("N,nlat,nlon,nd,members", [(21, 32, 64, 20, 9), (31, 48, 128, 13, 3)])
def test_hybrid_coordinates_in_members(jg, orc, N, nlat, nlon, nd, members, prec, tol):
    """more than three blocks of 32 columns per SM"""
    assert (nlon // 32) * nlat * members > 3 * jg.device_info()["sm_count"]
    params = configs.PARAMS["hs_t21l20"]
    gm, om = _meshes(jg, orc, N, nlat, nlon, nd, prec)
    omod = _developed(orc, om, params, vert_coord="hybrid")
    one = jg.Model(gm, params, vert_coord="hybrid")
    configs.copy_state(omod, one, "held_suarez")
    ens = jg.Model(gm, params, members=members, vert_coord="hybrid")
    for e in range(members):
        ens.copy_member(e, one)
    ens.step(3)
    omod.step(3)
    for e in (0, members - 1):
        one.copy_member(0, ens, e)
        _compare(one, omod, "held_suarez", tol)


@pytest.mark.parametrize("kind,members", [("barotropic", {64: 40, 128: 11, 256: 8}), ("shallow_water", {64: 20, 128: 6, 256: 5})])
@pytest.mark.parametrize("N,nlat,nlon", [(21, 36, 64), (42, 64, 128), (63, 96, 256)])
def test_one_layer_members_fp64(jg, orc, kind, members, N, nlat, nlon):
    """two warps or more per SM in the FFT of the step's fluxes (2 or 4 fields a member)"""
    E = members[nlon]
    rows = (2 if kind == "barotropic" else 4) * E * nlat
    assert rows * (4 if nlon == 64 else 8) >= 64 * jg.device_info()["sm_count"]
    params = dict(configs.PARAMS["barotropic_t42" if kind == "barotropic" else "sw_t85"], dt=600,
                  kappa_m=1.0 / (20 * 86400.0), kappa_t=1.0 / (10 * 86400.0))
    gm, om = _meshes(jg, orc, N, nlat, nlon, 1, "fp64")
    one, omod = jg.Model(gm, params), orc.Model(om, params)
    if kind == "barotropic":
        configs.init_barotropic_rh4(orc, om, omod)
    else:
        configs.init_shallow_water_jet(orc, om, omod)
        omod.set("grid_h_eq", np.asfortranarray(omod.get("grid_ps_c") * 1.01))
    configs.copy_state(omod, one, kind)
    ens = jg.Model(gm, params, members=E)
    for e in range(E):
        ens.copy_member(e, one)
    ens.step(4)
    omod.step(4)
    for e in (0, E - 1):
        one.copy_member(0, ens, e)
        _compare(one, omod, kind, 1e-10)
