"""The semi-implicit step and its adjoint on host arrays that the kernels read and write in place, on arrays 8 bytes off
a pair (copied through the staging buffer, one after another) and with outputs over inputs: the same bits."""
import ctypes as C

import numpy as np
import pytest

from jgcm import configs
from test_gpu_ragged_sizes import _shifted

pytestmark = pytest.mark.gpu


def _run(fn, md, ins, outs):
    a = (C.c_void_p * len(ins))(*[x.ctypes.data for x in ins])
    b = (C.c_void_p * len(outs))(*[x.ctypes.data for x in outs])
    assert fn(md._h, a, b) == 0


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_semi_implicit_arrays(jg, prec):
    mesh = jg.Spectral_Spherical_Mesh(31, 32, 48, 128, 13, 6371.0e3, precision=prec)
    md = jg.Model(mesh, configs.PARAMS["hs_t42l20"])
    md.update_init_step()  # (a first step does not depend on vor_p: its cotangent would be zero)
    rng = np.random.default_rng(2)

    def arrays(names, zero=False):
        out = []
        for k in names:
            a = mesh.spectral(1 if "lnps" in k else 13)
            if not zero:
                a[...] = rng.standard_normal(a.shape) + 1j * rng.standard_normal(a.shape)
            out.append(a)
        return out

    L = jg.lib()
    for fn, i, o in ((L.jgcm_model_semi_implicit_step, jg.SI_IN, jg.SI_OUT),
                     (L.jgcm_model_semi_implicit_step_adjoint, jg.SI_OUT, jg.SI_IN)):
        ins = arrays(i)
        ref, off = arrays(o, True), [_shifted(x) for x in arrays(o, True)]
        _run(fn, md, ins, ref)
        assert all(np.isfinite(x).all() and x.any() for x in ref)
        _run(fn, md, [_shifted(x) for x in ins], off)
        mixed = arrays(o, True)
        _run(fn, md, [x if k % 2 else _shifted(x) for k, x in enumerate(ins)], mixed)
        over = [x.copy(order="F") for x in ins]  # each output over the first free input of its size
        free = list(range(len(over)))
        outs = []
        for k in o:
            n = 1 if "lnps" in k else 13
            j = next((j for j in free if over[j].shape[2] == n), None)
            outs.append(over[j] if j is not None else mesh.spectral(n))
            if j is not None:
                free.remove(j)
        _run(fn, md, over, outs)
        for k in range(len(o)):
            for got in (off[k], mixed[k], outs[k]):
                assert np.array_equal(ref[k], got), (o[k])
