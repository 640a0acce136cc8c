"""Transforms whose output array is, or holds, an input array (C callers may): the arrays are read and written in
place, and every call has to give what it gives on arrays apart, bit for bit."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _call(jg, name, mesh, *args):
    f = getattr(jg.lib(), name)
    assert f(mesh._h, *[a if isinstance(a, int) else C.c_void_p(a.ctypes.data) for a in args]) == 0, jg.lib().jgcm_last_error()


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("N,nlat,nlon,nd", [(5, 10, 16, 3), (42, 64, 128, 20), (85, 128, 256, 13)])
def test_outputs_over_inputs(jg, N, nlat, nlon, nd, prec):
    mesh = jg.Spectral_Spherical_Mesh(N, N + 1, nlat, nlon, nd, 6371.0e3, precision=prec)
    rng = np.random.default_rng(3)
    ng, ns = nlon * nlat * nd, 2 * (N + 1) * (N + 2) * nd

    def arrays():  # a field twice as long as a grid (a Fourier array), another grid, a spectrum as long as a grid
        r = np.random.default_rng(3)
        return r.standard_normal(2 * ng), r.standard_normal(max(ng, ns)), r.standard_normal(max(ng, ns))

    for off in (0, 2 * (ng // 4), ng):  # the field at the start, in the middle and at the end of the output
        a, _, _ = arrays()
        out = np.zeros(2 * ng)
        _call(jg, "jgcm_trans_grid_to_fourier", mesh, a[off:off + ng].copy(), nd, out)
        _call(jg, "jgcm_trans_grid_to_fourier", mesh, a[off:], nd, a)
        assert np.array_equal(a, out), off
    for name, args in (("jgcm_trans_grid_to_spherical", "a b"), ("jgcm_trans_spherical_to_grid", "a b"),
                       ("jgcm_trans_spherical_to_grid_adjoint", "a b"), ("jgcm_trans_grid_to_spherical_adjoint", "a b"),
                       ("jgcm_vor_div_from_grid_uv", "bc de"), ("jgcm_uv_grid_from_vor_div", "bc de")):
        _, b, c = arrays()
        x, y = np.zeros(max(ng, ns)), np.zeros(max(ng, ns))
        if len(args) == 3:
            _call(jg, name, mesh, b.copy(), nd, x)
            _call(jg, name, mesh, b, nd, b)
            n = ng if name.endswith(("to_grid", "spherical_adjoint")) else ns
            assert np.array_equal(b[:n], x[:n]), name
        else:
            _call(jg, name, mesh, b.copy(), c.copy(), nd, x, y)
            _call(jg, name, mesh, b, c, nd, c, b)  # crossed
            n = ng if name.startswith("jgcm_uv") else ns
            assert np.array_equal(c[:n], x[:n]) and np.array_equal(b[:n], y[:n]), name
