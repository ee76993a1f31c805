"""The cluster size of a gang's resident streamfunction solves (mer_plan_many,
host code, compiled with its kernels but not run): it grows to what the largest
solve needs, never beyond what every solve can have, and a solve that does not
fit even then is named, not launched."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "codesthesis_dir_gb300", "csrc")

SOURCE = r"""
#include "meridian.cu"
#include <cstring>
static MerDev solve(int n1, int n2)
{
    MerDev d;
    memset(&d, 0, sizeof(d));
    d.nlev = 2;
    for (int l = 1; l <= 2; ++l) {
        d.lev[l].n1 = n1 / l;
        d.lev[l].n2 = n2 / l;
        d.lev[l].fac_z_step = (int)tdma32_len(n2 / l - 1);
    }
    return d;
}
#define CHECK(x) do { if (!(x)) return __LINE__; } while (0)
int main()
{
    size_t smem;
    char fits[2];
    MerDev d[2] = {solve(32, 32), solve(256, 256)};
    CHECK(mer_plan(d[0], 1) && !mer_plan(d[1], 1) && mer_plan(d[1], 16));
    int c = mer_plan_many(d, 2, 1, 16, &smem, fits);
    CHECK(c > 1 && c <= 16 && fits[0] && fits[1]);
    CHECK(smem <= MER_SMEM_MAX && smem >= 4 * (size_t)d[0].smem_floats && smem >= 4 * (size_t)d[1].smem_floats);
    c = mer_plan_many(d, 2, 1, 1, &smem, fits);
    CHECK(c == 1 && fits[0] && !fits[1] && smem == 4 * (size_t)d[0].smem_floats);
    c = mer_plan_many(d, 1, 4, 16, &smem, fits);
    CHECK(c == 4 && fits[0]);
    return 0;
}
"""


def test_gang_cluster_size(tmp_path):
    from codesthesis_dir_gb300 import _build
    src, exe = tmp_path / "plan.cu", tmp_path / "plan"
    src.write_text(SOURCE)
    subprocess.run([_build.nvcc(), *_build.ARCH, *_build.COMMON, "-o", str(exe), str(src)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
