"""Every transform entry point at the edges of the launch rules: one column, column counts that fill no
tile, latitude counts that are no power of two (and whose half is no multiple of a 16-byte chunk), rows
of one m that do not divide into the row chunks.

Tolerances: the transforms' own (tests/test_gpu_transforms.py): FP64 1e-12, FP32 5e-6 relative L2.
"""
import numpy as np
import pytest

from jgcm import configs
from test_gpu_models import MIXED_TOL, _compare
from test_hs_adjoint import _rand_like, _rms
from test_gpu_transforms import TOL, _grid, _meshes, _spec

pytestmark = pytest.mark.gpu

CASES = [(5, 10, 16, 1), (7, 12, 16, 3), (21, 36, 64, 5), (31, 48, 128, 13), (42, 64, 128, 1), (63, 96, 256, 7),
         (85, 128, 256, 1), (106, 160, 512, 2)]
# enough rows for the register-split FFTs at every length, column counts that leave a ragged last tile
MANY = [(31, 48, 64, 61), (42, 64, 128, 41), (63, 96, 256, 27), (106, 160, 512, 9), (170, 256, 1024, 5),
        (85, 128, 256, 61)]  # the last: the tiled synthesis, too


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("case", CASES + MANY)
def test_transforms(jg, orc, case, prec):
    N, nlat, nlon, nd = case
    gm, om = _meshes(jg, orc, N, nlat, nlon, nd, prec)
    for nlev in sorted({nd, 1}):
        s, s2, g, g2 = _spec(om, nlev, 3, False), _spec(om, nlev, 4, False), _grid(om, nlev, 5), _grid(om, nlev, 6)
        calls = [("Trans_Spherical_To_Grid", (s,), "g"), ("Trans_Grid_To_Spherical", (g,), "s"),
                 ("UV_Grid_From_Vor_Div", (s, s2), "gg"), ("Vor_Div_From_Grid_UV", (g, g2), "ss"),
                 ("Compute_Gradients", (s,), "gg"), ("Trans_Spherical_To_Grid_Adjoint", (g,), "s"),
                 ("Trans_Grid_To_Spherical_Adjoint", (s,), "g")]
        for name, ins, outs in calls:
            a = [gm.grid(nlev) if o == "g" else gm.spectral(nlev) for o in outs]
            b = [om.grid(nlev) if o == "g" else om.spectral(nlev) for o in outs]
            getattr(jg, name)(gm, *ins, *a)
            getattr(orc, name)(om, *ins, *b)
            for x, y in zip(a, b):
                assert configs.rel_l2(x, y) < TOL[prec], (name, nlev)


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-10), ("fp32", 5e-5)])
@pytest.mark.parametrize("N,nlat,nlon", [(21, 36, 64), (42, 64, 128), (63, 96, 256)])
def test_one_layer_steps(jg, orc, N, nlat, nlon, prec, tol):
    """Barotropic steps (the fused leapfrog epilogue behind the split rows) against the oracle, at the
    barotropic step tolerances."""
    params = dict(configs.PARAMS["barotropic_t42"], dt=1200)
    gm, om = _meshes(jg, orc, N, nlat, nlon, 1, prec)
    gmod, omod = jg.Model(gm, params), orc.Model(om, params)
    configs.init_barotropic_rh4(orc, om, omod)
    configs.copy_state(omod, gmod, "barotropic")
    gmod.step(6)
    omod.step(6)
    for f in configs.PROGNOSTIC["barotropic"]:
        assert configs.rel_l2(gmod.get(f), omod.get(f)) < tol, f


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-10), ("fp32", MIXED_TOL["fp32"])])
@pytest.mark.parametrize("N,nlat,nlon,nd,members", [(21, 40, 64, 7, 1), (31, 48, 128, 13, 1), (31, 48, 128, 13, 29),
                                                    (42, 64, 128, 20, 11), (63, 96, 256, 9, 1), (63, 96, 256, 9, 17),
                                                    (21, 40, 64, 7, 60), (31, 48, 128, 17, 30), (21, 32, 64, 32, 61),
                                                    (42, 64, 128, 20, 18)])
def test_held_suarez_steps(jg, orc, N, nlat, nlon, nd, members, prec, tol):
    """Held-Suarez steps on latitude counts that are no power of two, alone and as ensembles large enough
    for the tiled Legendre kernels, whose column tiles straddle members, and for the semi-implicit kernel of
    four columns per warp (every number of levels per lane, a ragged last warp): the first and last members
    against the oracle, at the step tolerances."""
    if prec == "fp64" and members > 1:
        members = 3
    params = configs.PARAMS["hs_t21l20"]
    gm, om = _meshes(jg, orc, N, nlat, nlon, nd, prec)
    omod, one = orc.Model(om, params), jg.Model(gm, params)
    configs.init_held_suarez(orc, om, omod)
    configs.add_hs_flow(orc, om, omod)
    configs.copy_state(omod, one, "held_suarez")
    ens = jg.Model(gm, params, members=members)
    for e in range(members):
        ens.copy_member(e, one)
    ens.step(3)
    omod.step(3)
    for e in {0, members - 1}:
        one.copy_member(0, ens, e)
        _compare(one, omod, "held_suarez", tol)


# the step adjoint's own tolerances (tests/test_hs_adjoint.py, ten levels); FP32 x sqrt(32 / 10) for the
# roundings of up to 32 levels' sums
@pytest.mark.parametrize("prec,tol", [("fp64", 1e-10), ("fp32", 2e-4 * 1.8)])
@pytest.mark.parametrize("N,nlat,nlon,nd", [(21, 36, 64, 3), (21, 32, 64, 8), (21, 32, 64, 9), (31, 48, 128, 20),
                                            (21, 32, 64, 25), (21, 32, 64, 32)])
def test_step_adjoint_levels(jg, orc, N, nlat, nlon, nd, prec, tol):
    """Every number of levels per lane of the reverse column kernel, its first and last level counts, and the
    transposed alpha operators at sizes that leave a ragged last block."""
    params = dict(configs.PARAMS["hs_t21l10"], dt=900)
    gm, om = _meshes(jg, orc, N, nlat, nlon, nd, prec)
    omod = orc.Model(om, params)
    configs.init_held_suarez(orc, om, omod)
    configs.add_hs_flow(orc, om, omod)
    orc.set_state(omod, orc.get_state(omod))
    omod.step(3)
    fields, _ = orc.get_state(omod)
    orc.set_state(omod, (fields, False))
    rng = np.random.default_rng(21)
    ybar = {k: _rand_like(rng, v, 1.0 / _rms(v)) for k, v in fields.items()}
    xb_o, pb_o = orc.HS_Step_Adjoint(omod, ybar)
    gmod = jg.Model(gm, params)
    for k in orc.STATE_FIELDS:
        gmod.set(k, fields[k])
    gmod.update_init_step()
    xb_g, pb_g = jg.HS_Step_Adjoint(gmod, ybar)
    for k in orc.STATE_FIELDS:
        assert configs.rel_l2(xb_g[k], xb_o[k]) < tol, k
    for p, x, y in zip(orc.HS_PARAMS, pb_g, pb_o):
        assert abs(x - y) <= tol * abs(y) + 1e-30, p


def _shifted(a):
    """a copy of `a` whose data start 8 bytes past a 16-byte boundary (FP64 arrays need no more)"""
    raw = np.zeros(a.nbytes // 8 + 3)
    off = 1 if raw.ctypes.data % 16 == 0 else 2
    b = raw[off:off + a.nbytes // 8].view(a.dtype).reshape(a.shape, order="F")
    b[...] = a
    assert b.ctypes.data % 16 == 8 and b.flags.f_contiguous
    return b


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("case", [(7, 12, 16, 3), (42, 64, 128, 1), (42, 64, 128, 20)])
def test_host_arrays_off_the_pair_alignment(jg, orc, case, prec):
    """Arrays that the kernels do not read or write in place (8 bytes off a 16-byte boundary) give the
    results of those that they do, bit for bit; so does a fresh output whose pages nobody has touched."""
    N, nlat, nlon, nd = case
    gm, om = _meshes(jg, orc, N, nlat, nlon, nd, prec)
    s, g = _spec(om, nd, 3, False), _grid(om, nd, 5)
    for name, ins, outs in (("UV_Grid_From_Vor_Div", (s, 2 * s), (gm.grid(nd), gm.grid(nd))),
                            ("Vor_Div_From_Grid_UV", (g, 2 * g), (gm.spectral(nd), gm.spectral(nd))),
                            ("Add_Horizontal_Advection", (s, g, 2 * g), (g.copy(order="F"),))):
        off = [_shifted(x) for x in outs]
        getattr(jg, name)(gm, *[np.asfortranarray(x) for x in ins], *outs)
        getattr(jg, name)(gm, *[_shifted(x) for x in ins], *off)
        for a, b in zip(outs, off):
            assert np.array_equal(a, b), name


def test_packed_state_off_the_pair_alignment(jg):
    params = configs.PARAMS["hs_t21l10"]
    mesh = configs.make_mesh(jg, "hs_t21l10", precision="fp32")
    md = jg.Model(mesh, params)
    configs.init_held_suarez(jg, mesh, md)
    a, b = md.get_state(), _shifted(np.zeros(md.state_size()))
    md.get_state(out=b)
    assert np.array_equal(a, b)
    md.set_state(2.0 * a)
    md.set_state(b)
    assert np.array_equal(md.get_state(), a)
