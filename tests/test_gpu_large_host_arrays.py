"""Results of more than 16 MiB: in pageable memory they go through the copy engine, in pinned memory the kernels
write them in place.  Both give the same bits, for every call with a grid result and for a packed state."""
import ctypes as C

import numpy as np
import pytest

from jgcm import configs
from test_zz_no_alloc import cudart

pytestmark = pytest.mark.gpu


class Pinned:
    """FP64 arrays in page-locked memory, freed together"""

    def __init__(self):
        self.ptrs = []

    def array(self, shape, dtype=np.float64):
        rt, p = cudart(), C.c_void_p()
        rt.cudaMallocHost.argtypes = [C.POINTER(C.c_void_p), C.c_size_t]
        n = int(np.prod(shape)) * np.dtype(dtype).itemsize
        assert rt.cudaMallocHost(C.byref(p), n) == 0
        self.ptrs.append(p)
        a = np.frombuffer((C.c_char * n).from_address(p.value), dtype=dtype).reshape(shape, order="F")
        a[...] = 0
        return a

    def free(self):
        rt = cudart()
        rt.cudaFreeHost.argtypes = [C.c_void_p]
        for p in self.ptrs:
            rt.cudaFreeHost(p)


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_grids(jg, prec):
    N, nlat, nlon, nd = 106, 160, 512, 30
    mesh = jg.Spectral_Spherical_Mesh(N, N + 1, nlat, nlon, nd, 6371.0e3, precision=prec)
    rng = np.random.default_rng(1)
    s = np.asfortranarray(rng.standard_normal((N + 1, N + 2, nd)) + 1j * rng.standard_normal((N + 1, N + 2, nd)))
    g, g2, dh = (np.asfortranarray(rng.standard_normal((nlon, nlat, nd))) for _ in range(3))
    assert g.nbytes > 16 << 20
    pin = Pinned()
    try:
        for name, ins, outs in (("Trans_Spherical_To_Grid", (s,), 1), ("UV_Grid_From_Vor_Div", (s, 2 * s), 2),
                                ("Compute_Gradients", (s,), 2), ("Add_Horizontal_Advection", (s, g, g2), 1),
                                ("Trans_Grid_To_Spherical_Adjoint", (s,), 1), ("Trans_Grid_To_Fourier", (g,), 1)):
            dt = np.complex128 if name.endswith("Fourier") else np.float64
            a = [np.zeros(g.shape, dtype=dt, order="F") for _ in range(outs)]
            b = [pin.array(g.shape, dt) for _ in range(outs)]
            if name.startswith("Add"):
                a[0][...] = dh
                b[0][...] = dh
            getattr(jg, name)(mesh, *ins, *a)
            getattr(jg, name)(mesh, *ins, *b)
            for x, y in zip(a, b):
                assert np.isfinite(x).all() and x.any() and np.array_equal(x, y), name
    finally:
        pin.free()


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_state(jg, prec):
    mesh = jg.Spectral_Spherical_Mesh(63, 64, 96, 256, 13, 6371.0e3, precision=prec)
    md = jg.Model(mesh, configs.PARAMS["hs_t42l20"])
    configs.init_held_suarez(jg, mesh, md)
    pin = Pinned()
    try:
        a, b = md.get_state(), pin.array(md.state_size())
        assert a.nbytes > 16 << 20
        md.get_state(out=b)
        assert a.any() and np.array_equal(a, b)
        md.set_state(2.0 * a)
        assert np.array_equal(md.get_state(), 2.0 * a)
        md.set_state(b)
        assert np.array_equal(md.get_state(), a)
    finally:
        pin.free()
