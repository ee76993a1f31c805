"""The grid barrier's arithmetic (gridsync.cuh), compiled for the host: the
blocks that arrive between two multiples of the grid size all wait for the
next one, whatever the count has grown to; around 2^32, where a 32-bit count
would start again in the middle of a barrier, as at its start."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include "gridsync.cuh"
#include <type_traits>
static_assert(sizeof(*GridSync::count) == 8, "the count must not wrap during a launch");
int main()
{
    int bad = 0;
    const unsigned grids[] = {1, 2, 152, 303, 304};
    for (unsigned b : grids)
        for (unsigned long long barrier : {0ull, 1ull, (1ull << 32) / b - 1, (1ull << 32) / b, (1ull << 32) / b + 1, 1ull << 40})
            for (unsigned k = 0; k < b; ++k)
                if (grid_barrier_end(barrier * b + k, b, barrier * b) != (barrier + 1) * b) ++bad;
    return bad != 0;
}
"""


def test_barriers_end_at_multiples_of_the_grid(tmp_path):
    from codesthesis_dir_gb300 import _build
    src, exe = tmp_path / "barrier.cu", tmp_path / "barrier"
    src.write_text(SOURCE)
    csrc = os.path.join(ROOT, "codesthesis_dir_gb300", "csrc")
    subprocess.run([_build.nvcc(), *_build.ARCH, "-std=c++17", "-I", csrc, "-o", str(exe), str(src)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
