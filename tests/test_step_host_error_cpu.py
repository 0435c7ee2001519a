"""mhdgb_step_host with page-locked arrays when one of its launches fails: the descriptor on the device must
not keep pointing at the caller's U_out, which the program may free before its next step.  The
library's own objects run on a stand-in for the CUDA runtime (fake_cudart.cpp)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from mhdturbulence_gb300 import _lib, build

HERE = os.path.dirname(os.path.abspath(__file__))
DP = C.POINTER(C.c_double)


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    build.build(driver=False)
    d = tmp_path_factory.mktemp("fake")
    so, obj = str(d / "libmhdgb_fake.so"), str(d / "fake_cudart.o")
    subprocess.run([build.nvcc(), "-O1", "-std=c++17", "-Xcompiler", "-fPIC", "-x", "c++", "-c",
                    os.path.join(HERE, "fake_cudart.cpp"), "-o", obj], check=True)
    objs = [os.path.join(build.OUT, os.path.splitext(u)[0] + ".o") for u, _ in build.UNITS]
    if not all(os.path.exists(o) for o in objs):
        build.build(force=True, driver=False)
    # (symbols bound inside the library: another CUDA runtime may be loaded in this process)
    subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-o", so, *objs, obj, "-lpthread"], check=True)
    lib = C.CDLL(so)
    lib.fake_host_u.restype = C.c_void_p
    lib.mhdgb_last_error.restype = C.c_char_p
    return lib


@pytest.mark.parametrize("precision", ["fp64", "fp64_exact", "mixed"])
@pytest.mark.parametrize("nsteps", [1, 3])
@pytest.mark.parametrize("kernel", [None, "k_recover", "k_fused_step"])
def test_a_failed_launch_leaves_no_pointer_to_the_output(fake, kernel, nsteps, precision):
    cfg = _lib.Config()
    fake.mhdgb_config_default(C.byref(cfg))
    cfg.nx = cfg.ny = cfg.nz = 8
    cfg.precision = {"fp64": 0, "fp64_exact": 1, "mixed": 2}[precision]
    h = C.c_void_p()
    assert fake.mhdgb_create(C.byref(cfg), C.byref(h)) == 0
    U = [np.zeros((13, 13, 10, 13)) for _ in range(2)]
    fake.fake_reset((kernel or "").encode())
    rc = fake.mhdgb_step_host(h, *(u.ctypes.data_as(DP) for u in U), nsteps, None, None)
    assert (rc != 0) == (kernel is not None), (rc, fake.mhdgb_last_error(h))
    assert fake.fake_host_u() is None
    assert fake.mhdgb_destroy(h) == 0
