"""The host-pointer transforms leave the caller's arrays alone once they return, in failure too (CPU).

Their kernels read and write the arrays in place, so a call that returned with work in flight would let a
program free memory that the device still reads or writes.  The entry points are compiled over stand-ins
(native/host_calls.cu) that record what is queued and fail on request.  The stand-ins run in a process of their
own that sees no CUDA device: nothing can be launched, whatever machine this runs on.
"""
import ctypes as C
import json
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))

# entry point -> its array arguments ('a'), the level count ('n') where it stands
CALLS = {"jgcm_trans_spherical_to_grid": "ana", "jgcm_trans_grid_to_spherical": "ana",
         "jgcm_trans_spherical_to_grid_adjoint": "ana", "jgcm_trans_grid_to_spherical_adjoint": "ana",
         "jgcm_trans_grid_to_fourier": "ana", "jgcm_vor_div_from_grid_uv": "aanaa",
         "jgcm_uv_grid_from_vor_div": "aanaa", "jgcm_compute_gradients": "anaa",
         "jgcm_add_horizontal_advection": "aaana", "jgcm_apply_laplacian": "an",
         "jgcm_area_weighted_global_mean": "aa"}


def _run(so):
    """every call of both precisions: {"name/precision": {what: [status, events]}}"""
    lib = C.CDLL(so)
    lib.stub_mesh.restype = C.c_void_p
    lib.stub_events.restype = C.c_char_p

    def call(name, mesh, fail_at=0, null=None, nlev=3):
        arrays, args = [], [C.c_void_p(mesh)]
        for c in CALLS[name]:
            if c == "n":
                args.append(C.c_int(nlev))
                continue
            arrays.append((C.c_double * (2 * 16 * 10 * 3))())
            args.append(C.c_void_p(None if len(arrays) - 1 == null else C.addressof(arrays[-1])))
        lib.stub_begin(fail_at)
        return [getattr(lib, name)(*args), lib.stub_events().decode()]

    out = {}
    for precision in (0, 1):
        mesh = lib.stub_mesh(precision)
        for name, args in CALLS.items():
            good = call(name, mesh)
            r = {"good": good, "bad": [call(name, mesh, null=k) for k in range(args.count("a"))] + [call(name, None)],
                 "failing": [call(name, mesh, fail_at=k) for k in range(1, good[1].count("q") + 1)]}
            if "n" in args:
                r["bad"].append(call(name, mesh, nlev=2))
            out[f"{name}/{precision}"] = r
    return out


@pytest.fixture(scope="module")
def results(built, tmp_path_factory):
    import build_lib

    so = str(tmp_path_factory.mktemp("native") / "libhostcalls.so")
    wrap = [f"-Xlinker=--wrap={f}" for f in ("cudaStreamSynchronize", "cudaGetLastError", "cudaMemcpyAsync")]
    cmd = [build_lib.NVCC] + build_lib.ARCH + build_lib.FLAGS + ["-Xcompiler", "-fvisibility=default", "-shared", "-o", so,
           os.path.join(HERE, "native", "host_calls.cu")] + wrap
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([sys.executable, os.path.abspath(__file__), so], capture_output=True, text=True,
                       env=dict(os.environ, CUDA_VISIBLE_DEVICES=""))
    assert r.returncode == 0, r.stderr
    return json.loads(r.stdout)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("name", sorted(CALLS))
def test_arguments_are_checked_before_anything_is_queued(results, name, precision):
    for r in results[f"{name}/{precision}"]["bad"]:
        assert r == [-1, ""]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("name", sorted(CALLS))
def test_a_failing_call_waits_for_what_it_queued(results, name, precision):
    """whichever launch or copy fails: a synchronisation follows the last thing queued"""
    r = results[f"{name}/{precision}"]
    assert r["good"][0] == 0 and r["good"][1].strip("q") == "s" and r["failing"]
    for k, f in enumerate(r["failing"]):
        assert f == [-2, "q" * k + "s"], k


if __name__ == "__main__":
    print(json.dumps(_run(sys.argv[1])))
