"""jgcm_trans_spherical_to_grid_noalloc on device grids that start off a pair of values.

The inverse FFTs in registers store two values at a time; a grid that starts one value off that boundary has
to take the kernel that stores single values.  One size for each of them: a warp per row, split in registers,
a row per thread, and a row shorter than a warp's.  Tolerances: the transforms' own (FP64 1e-12, FP32 5e-6).
"""
import numpy as np
import pytest

from jgcm import configs
from test_zz_no_alloc import DeviceBuffer, _entry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-12), ("fp32", 5e-6)])
@pytest.mark.parametrize("N,nlat,nlon,nd", [(42, 64, 128, 1), (42, 64, 128, 20), (21, 320, 64, 61), (63, 96, 256, 13),
                                            (5, 10, 16, 3)])
def test_grid_off_a_pair(jg, N, nlat, nlon, nd, prec, tol):
    mesh = jg.Spectral_Spherical_Mesh(N, N + 1, nlat, nlon, nd, 6371.0e3, precision=prec)
    rng = np.random.default_rng(5)
    s = rng.standard_normal((N + 1, N + 2, nd)) + 1j * rng.standard_normal((N + 1, N + 2, nd))
    s = np.asfortranarray(s * (np.arange(N + 2)[None, :, None] >= np.arange(N + 1)[:, None, None]))
    ref = mesh.grid(nd)
    jg.Trans_Spherical_To_Grid(mesh, s, ref)
    cdt, rdt = (np.complex128, np.float64) if prec == "fp64" else (np.complex64, np.float32)
    ts, n = np.dtype(rdt).itemsize, nlon * nlat * nd
    d_s, d_g = DeviceBuffer(s.size * 2 * ts), DeviceBuffer((n + 2) * ts)
    try:
        d_s.upload(np.ascontiguousarray(s).astype(cdt))
        f = _entry(jg)
        for off in (0, 1):
            d_g.poison()
            assert f(mesh._h, d_s.ptr, nd, d_g.ptr.value + off * ts, None) == 0, jg.lib().jgcm_last_error()
            assert jg.lib().jgcm_mesh_synchronize(mesh._h) == 0, jg.lib().jgcm_last_error()
            out = d_g.download((n + 2,), rdt)
            assert np.isnan(out[:off]).all() and np.isnan(out[off + n:]).all()
            got = out[off:off + n].astype(np.float64).reshape(nd, nlat, nlon).transpose(2, 1, 0)
            assert configs.rel_l2(got, ref) < tol, off
        # an array that is not aligned to its own values is an error, before anything is queued
        assert f(mesh._h, d_s.ptr, nd, d_g.ptr.value + 2, None) == -1
        assert f(mesh._h, d_s.ptr.value + ts, nd, d_g.ptr, None) == -1
        assert b"aligned" in jg.lib().jgcm_last_error()
    finally:
        d_s.free()
        d_g.free()
