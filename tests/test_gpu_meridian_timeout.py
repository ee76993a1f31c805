"""A resident streamfunction solve whose wait for a table copy gives up ends with
GB_TIMEOUT, its copies landed and psi as it was, and the context goes on working.
The wait is made to run out by a build of meridian.cu whose waits take no poll
(every copy does arrive; its tables are just not waited for)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def impatient(gblib, tmp_path_factory):
    from codesthesis_dir_gb300 import _build, lib
    out = tmp_path_factory.mktemp("impatient")
    obj, so = str(out / "meridian.o"), str(out / "libimpatient.so")
    src = os.path.join(_build.CSRC, "meridian.cu")
    subprocess.run([_build.nvcc(), *_build.ARCH, *_build.COMMON, "-DMER_POLLS=0", "-c", src, "-o", obj], check=True)
    rest = [os.path.join(_build.OUT, os.path.basename(s)[:-3] + ".o") for s in _build._sources() if s != src]
    subprocess.run([_build.nvcc(), *_build.ARCH, "-shared", "-Xlinker", "-Bsymbolic", "-o", so, obj, *rest, "-lcudart_static", "-ldl", "-lrt", "-lpthread"], check=True)
    L = C.CDLL(so, mode=os.RTLD_LOCAL)
    for name, res, args in lib.SIGNATURES:
        fn = getattr(L, name)
        fn.restype, fn.argtypes = res, args
    return L


@pytest.mark.parametrize("nr,nz", [(64, 64), (128, 96)])
def test_wait_gives_up(gblib, impatient, nr, nz):
    from codesthesis_dir_gb300 import axi, lib
    rng = np.random.default_rng(1)
    rhs = np.asfortranarray(rng.standard_normal((nr + 1, nz + 1)))

    def solve(L):
        p, h, n = lib.AxiParams(), C.c_void_p(), C.c_int()
        L.gb_axi_default_params(C.byref(p), nr, nz)
        p.smoother, p.precision = lib.SMOOTHER_ZEBRA, lib.PRB_MIXED
        assert L.gb_axi_create(C.byref(p), C.byref(h), C.byref(n)) == 0
        assert L.gb_axi_set_field(h, lib.AXI_FIELD_ID["omegn"], rhs.ctypes.data, nr + 1) == 0
        psi = np.zeros((nr + 1, nz + 1), order="F")
        status = L.gb_axi_poisson(h, C.byref(n))
        assert L.gb_axi_get_field(h, lib.AXI_FIELD_ID["phi"], psi.ctypes.data, nr + 1) == 0
        L.gb_axi_destroy(h)
        return status, psi

    st, want = solve(gblib)
    assert st == lib.GB_OK and np.abs(want).max() > 0
    st, psi = solve(impatient)
    assert st == lib.GB_TIMEOUT and not psi.any()
    st, again = solve(gblib)
    assert st == lib.GB_OK
    np.testing.assert_array_equal(again, want)
