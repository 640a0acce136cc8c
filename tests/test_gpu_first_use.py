"""Buffers that a call allocates (zero-filled) are complete before the mesh's stream uses them: the first packed
read-out of a fresh model, through its staging buffer, holds the model's fields, and the first semi-implicit steps
on a fresh model agree with later ones, bit for bit."""
import numpy as np
import pytest

from jgcm import configs
from test_gpu_ragged_sizes import _shifted

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_first_read_out(jg, prec):
    mesh = jg.Spectral_Spherical_Mesh(85, 86, 128, 256, 20, 6371.0e3, precision=prec)
    for _ in range(4):
        md = jg.Model(mesh, configs.PARAMS["hs_t42l20"])
        md.spectral_initialize_fields(None, True)
        out = _shifted(np.zeros(md.state_size()))
        md.get_state(out=out)  # the staging buffer is allocated by this call
        got = jg.unpack_state(mesh, out)
        for k in ("spe_vor_c", "spe_t_p", "grid_u_p", "grid_t_c", "grid_vor", "grid_div"):
            assert np.array_equal(got[k], md.get(k)), k


def test_first_semi_implicit_steps(jg):
    mesh = configs.make_mesh(jg, "hs_t42l20", precision="fp64")
    rng = np.random.default_rng(4)
    ins = {k: mesh.spectral(1 if "lnps" in k else 20) for k in jg.SI_IN}
    for a in ins.values():
        a[...] = rng.standard_normal(a.shape)
    ref = None
    for _ in range(4):
        md = jg.Model(mesh, configs.PARAMS["hs_t42l20"])
        for _ in range(2):
            out = jg.Semi_Implicit_Step(md, ins)
            ref = ref or out
            for k in jg.SI_OUT:
                assert out[k].any() and np.array_equal(out[k], ref[k]), k
