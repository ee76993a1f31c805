"""A cluster launch's result cannot be dropped: the build's own flags refuse it
(an error while a stream is captured would otherwise leave a step without its
solve)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "codesthesis_dir_gb300", "csrc")

CALLS = {
    "cl_launch": ('#include "cluster.cuh"', "cl_launch(k, 1, 1, 32, 0, s)"),
    "mer_launch": ('#include "meridian.cuh"', "mer_launch(MerDev(), 1, s)"),
    "mer_launch_many": ('#include "meridian.cuh"', "mer_launch_many(nullptr, 1, 0, 1, 0, s)"),
    "gb_str_launch_device": ('#include "gbcommon.cuh"\n#include "str_internal.cuh"',
                             "gb_str_launch_device(nullptr, nullptr, nullptr, nullptr, nullptr, 0, 0., 1, 1, 0, s)"),
    "prb_launch_mg": ('#include "prb_internal.cuh"', "prb_launch_mg(nullptr, 1, 1, s)"),
    "prb_mg_launch_eqs": ('#include "prb_internal.cuh"', "prb_mg_launch_eqs(nullptr, 0, 1, 0, 1, 0, s)"),
    "prb_resident_launch": ('#include "prb_internal.cuh"', "prb_resident_launch(nullptr, 0, 1, 0, 1, 0, s)"),
}


def _compiles(tmp_path, include, body):
    from codesthesis_dir_gb300 import _build
    src = tmp_path / "t.cu"
    src.write_text("%s\n__global__ void k() {}\nint f(cudaStream_t s) { %s return 0; }\n" % (include, body))
    cmd = [_build.nvcc(), *_build.ARCH, *_build.COMMON, "-c", str(src), "-o", str(tmp_path / "t.o")]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode:
        assert "unused-result" in r.stderr, r.stderr
    return r.returncode == 0


@pytest.mark.parametrize("call", CALLS)
def test_dropped_launch_result_does_not_compile(tmp_path, call):
    include, expr = CALLS[call]
    assert _compiles(tmp_path, include, "auto r = %s; (void)r;" % expr)
    assert not _compiles(tmp_path, include, expr + ";")
