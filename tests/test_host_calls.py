"""The host-pointer transforms leave the caller's arrays alone once they return, in failure too (CPU).

Their kernels read and write the arrays in place, so a call that returns with work in flight would let a
program free memory that the device still reads or writes.  The entry points are compiled over stand-ins
(native/host_calls.cu) that record what is queued and fail on request; nothing runs on a device.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))

# entry point -> its array arguments ('a'), the level count ('n') where it stands
CALLS = {"jgcm_trans_spherical_to_grid": "ana", "jgcm_trans_grid_to_spherical": "ana",
         "jgcm_trans_spherical_to_grid_adjoint": "ana", "jgcm_trans_grid_to_spherical_adjoint": "ana",
         "jgcm_trans_grid_to_fourier": "ana", "jgcm_vor_div_from_grid_uv": "aanaa",
         "jgcm_uv_grid_from_vor_div": "aanaa", "jgcm_compute_gradients": "anaa",
         "jgcm_add_horizontal_advection": "aaana", "jgcm_apply_laplacian": "an",
         "jgcm_area_weighted_global_mean": "aa"}


@pytest.fixture(scope="module")
def stub(built, tmp_path_factory):
    import build_lib

    so = str(tmp_path_factory.mktemp("native") / "libhostcalls.so")
    wrap = [f"-Xlinker=--wrap={f}" for f in ("cudaStreamSynchronize", "cudaGetLastError", "cudaMemcpyAsync")]
    cmd = [build_lib.NVCC] + build_lib.ARCH + build_lib.FLAGS + ["-Xcompiler", "-fvisibility=default", "-shared",
           "-o", so, os.path.join(HERE, "native", "host_calls.cu")] + wrap
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = C.CDLL(so)
    lib.stub_mesh.restype = C.c_void_p
    lib.stub_events.restype = C.c_char_p
    return lib


def _call(stub, name, mesh, fail_at, null=None, nlev=3):
    f = getattr(stub, name)
    arrays, args, k = [], [C.c_void_p(mesh)], 0
    for c in CALLS[name]:
        if c == "n":
            args.append(C.c_int(nlev))
            continue
        arrays.append(np.zeros(2 * 16 * 10 * 3))
        args.append(C.c_void_p(None if k == null else arrays[-1].ctypes.data))
        k += 1
    stub.stub_begin(fail_at)
    status = f(*args)
    return status, stub.stub_events().decode()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("name", sorted(CALLS))
def test_arguments_are_checked_before_anything_is_queued(stub, name, precision):
    mesh = stub.stub_mesh(precision)
    for null in range(CALLS[name].count("a")):
        assert _call(stub, name, mesh, 0, null=null) == (-1, ""), null
    if "n" in CALLS[name]:
        assert _call(stub, name, mesh, 0, nlev=2) == (-1, "")
    assert _call(stub, name, None, 0) == (-1, "")


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("name", sorted(CALLS))
def test_a_failing_call_waits_for_what_it_queued(stub, name, precision):
    """whichever launch or copy fails: a synchronisation follows the last thing queued"""
    mesh = stub.stub_mesh(precision)
    status, events = _call(stub, name, mesh, 0)
    assert status == 0 and events.endswith("s") and "q" in events
    for k in range(1, events.count("q") + 1):
        status, ev = _call(stub, name, mesh, k)
        assert status == -2 and ev == "q" * (k - 1) + "s", (k, ev)
