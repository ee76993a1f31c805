"""The 3D line phases' staging rule (r3d_stage.cuh), compiled for the host: for
every line length and every number of lines up to a chunk's the staged lines
stay inside their area, or, where one line alone is longer than it, inside
both areas with the factors not staged."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "codesthesis_dir_gb300", "csrc")

SOURCE = r"""
#include "r3d_stage.cuh"
#include "banded.cuh"
#include <cstdio>
int main()
{
    long bad = 0, full = 0;
    for (int f64 = 0; f64 <= 1; ++f64)
        for (int dir = 0; dir < 3; ++dir)
            for (int n = 3; n <= (dir == 2 ? 16384 : 4096); ++n) {
                if (f64 && n > R3_MAX_ROWS) continue;
                // the longest table a line may have: pentadiagonal or, along phi, periodic
                const int len = dir == 2 ? (f64 ? 7 * n : 4) : (int)(f64 ? pdma_fac_len(n) : pdma32_len(n));
                const int words = R3_CHUNK_BYTES / (f64 ? 8 : 4), room = R3_FAC_BYTES / (f64 ? 8 : 4);
                const int chunk = r3_chunk(f64, dir, n, len);
                if (chunk < 1 || chunk > R3_THREADS) ++bad;
                for (int nl = 1; nl <= chunk; ++nl) {
                    const long need = r3_stage_words(f64, n, nl);
                    if (need <= words) continue;
                    if (chunk > 1 || need > words + room || (f64 && len <= room)) {
                        if (bad++ < 5) std::printf("f64 %d dir %d n %d nl %d of %d: %ld words\n", f64, dir, n, nl, chunk, need);
                    }
                }
                // and a chunk leaves no room for two lines more
                if (dir != 1 && chunk + 2 < R3_THREADS && r3_stage_words(f64, n, chunk + 2) <= words) ++full;
            }
    std::printf("bad %ld, not full %ld\n", bad, full);
    return bad || full;
}
"""


def test_chunks_fit_their_area(tmp_path):
    from codesthesis_dir_gb300 import _build
    src, exe = tmp_path / "stage.cu", tmp_path / "stage"
    src.write_text(SOURCE)
    subprocess.run([_build.nvcc(), *_build.ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-I", CSRC, "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_lines_longer_than_the_buffer_are_refused(gblib):
    """An FP64 ring one step too long is refused before anything is allocated;
    mixed ones (FP32 lines) of the same length fit, as does the longest FP64 one."""
    import ctypes as C

    from codesthesis_dir_gb300 import lib

    params = gblib.gb_r3d_default_params.argtypes[0]._type_   # the binding's, also after a reload of lib

    def create(np_, precision):
        p, h = params(), C.c_void_p()
        gblib.gb_r3d_default_params(C.byref(p), 4, 4, np_)
        p.precision = precision
        st = gblib.gb_r3d_create(C.byref(p), C.byref(h), None)
        if st == 0:
            gblib.gb_r3d_destroy(h)
        return st

    longest = 96 * 1024 // 8
    assert create(longest + 8, lib.PRB_FP64) == lib.GB_ERR_INVALID
    assert create(16384, lib.PRB_FP64) == lib.GB_ERR_INVALID
    assert create(longest, lib.PRB_FP64) != lib.GB_ERR_INVALID
    assert create(16384, lib.PRB_MIXED) != lib.GB_ERR_INVALID
