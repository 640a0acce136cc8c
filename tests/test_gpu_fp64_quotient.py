"""FP64 winds and gradients are quotients by cos(lat), rounded once, whichever inverse FFT forms them.

Zonally symmetric fields pass the FFTs exactly (one coefficient, sums with zeros), so a launch of many columns
(register-split kernel) has to give the bits of a launch of one level (shared-memory kernel).  The latitude counts
are those whose synthesis tiles divide a block: others (160: three columns) form their inputs in code of their own,
with roundings of its own."""
import numpy as np
import pytest

from test_gpu_transforms import _meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,nlat,nlon,nd", [(21, 32, 64, 40), (42, 64, 128, 20), (63, 96, 256, 13), (106, 256, 512, 5)])
def test_many_levels_as_one(jg, orc, N, nlat, nlon, nd):
    gm, _ = _meshes(jg, orc, N, nlat, nlon, nd, "fp64")
    rng = np.random.default_rng(9)
    vor, div = gm.spectral(nd), gm.spectral(nd)
    vor[0, :N + 1], div[0, :N + 1] = rng.standard_normal((2, N + 1, nd))
    u, v = gm.grid(nd), gm.grid(nd)
    for name, ins in (("UV_Grid_From_Vor_Div", (vor, div)), ("Compute_Gradients", (vor,))):
        getattr(jg, name)(gm, *ins, u, v)
        for k in (0, nd // 2, nd - 1):
            a, b = gm.grid(1), gm.grid(1)
            getattr(jg, name)(gm, *[np.asfortranarray(x[:, :, k:k + 1]) for x in ins], a, b)
            assert np.abs(a).max() + np.abs(b).max() > 0
            assert np.array_equal(u[:, :, k:k + 1], a) and np.array_equal(v[:, :, k:k + 1], b), (name, k)
