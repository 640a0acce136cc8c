"""The height gradients that a shallow-water step keeps for the next one are dropped when the state changes.

Steps (single, graphs of three and an ensemble's window graphs) with changes in between: another spe_lnps_c, another
spe_lnps_n (which the next step advects), Update_Init_Step!'s flag, members copied in.  The oracle gets the same
sequence; its advected height is spe_lnps_n throughout, which the library reads only after it was set, so a
new spe_lnps_c is set in both there.  Tolerance: the one-layer models' own after about six steps (FP64 1e-10, FP32
5e-5), four times that for the 25 steps here.
"""
import numpy as np
import pytest

from jgcm import configs
from test_gpu_models import _compare
from test_gpu_transforms import _meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,tol", [("fp64", 4e-10), ("fp32", 2e-4)])
@pytest.mark.parametrize("N,nlat,nlon", [(31, 48, 128), (42, 64, 128)])
def test_changes_between_steps(jg, orc, N, nlat, nlon, prec, tol):
    params = dict(configs.PARAMS["sw_t85"], dt=600)
    gm, om = _meshes(jg, orc, N, nlat, nlon, 1, prec)
    md, omod = jg.Model(gm, params), orc.Model(om, params)
    configs.init_shallow_water_jet(orc, om, omod)
    configs.copy_state(omod, md, "shallow_water")

    def both(n):
        md.step(n)
        omod.step(n)
        _compare(md, omod, "shallow_water", tol)

    def height(seed):  # the oracle's height with its waves changed by several per cent
        rng = np.random.default_rng(seed)
        s = omod.get("spe_lnps_c")
        f = 1.0 + 0.1 * rng.standard_normal(s.shape)
        f[0, 0] = 1.0
        return s * f

    both(5)
    x = height(1)
    md.set("spe_lnps_c", x)
    omod.set("spe_lnps_c", x)
    omod.set("spe_lnps_n", x)
    both(4)
    x = height(2)
    md.set("spe_lnps_n", x)
    omod.set("spe_lnps_n", x)
    both(4)
    md.set_init_step(True)
    orc.set_init_step(omod, True)
    both(3)
    x = height(3)
    en = jg.Ensemble([md], 2 * params["dt"])
    md.set("spe_lnps_c", x)
    omod.set("spe_lnps_c", x)
    omod.set("spe_lnps_n", x)
    en.step(2)
    omod.step(4)
    _compare(md, omod, "shallow_water", tol)
    en.close()
    # members: an ensemble past its first step takes the state, gradients of another one in hand
    ens = jg.Model(gm, params, members=3)
    fresh = jg.Model(gm, params)
    first = orc.Model(om, params)
    configs.init_shallow_water_jet(orc, om, first)
    configs.copy_state(first, fresh, "shallow_water")
    for e in range(3):
        ens.copy_member(e, fresh)
    ens.step(4)
    for e in (1, 2):
        ens.copy_member(e, md)
    ens.step(5)
    omod.step(5)
    first.step(9)
    for e, ref in ((0, first), (1, omod), (2, omod)):
        md.copy_member(0, ens, e)
        _compare(md, ref, "shallow_water", tol)
