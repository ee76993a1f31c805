"""The streamfunction solve on a cluster (meridian.cu, axi.cu, str.cu) at the
sizes where its layouts change: lines of 32, 64, 128, 256 and 512 rows and one
more or less, more CTAs than rows, n1 != n2 both ways, grids too long for the
resident cycles, both line orders.

The FP64 solve is bit-identical to the oracle (test_gpu_axi_parity.py,
test_gpu_str_parity.py).  The mixed solve stops at the same residual bound, so
A (psi_mixed - psi_fp64) is below 2 tolcon everywhere.  The operator on the
0.5 x 0.5 section has |A^-1| <= 0.5^2 / 8 in the maximum norm (the uniform one
obeys a maximum principle; the stretched one's one-sided points make it only
nearly so: a factor 4 is allowed), which bounds the difference."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOLCON = 1e-8
BOUND = 2 * TOLCON * 0.5 ** 2 / 8


def _solve(nr, nz, precision, smoother, stretch, rhs):
    from codesthesis_dir_gb300 import axi
    grid = axi.stretched_grid(nr, nz, 0.5, 1.0, 0.5, stretch) if stretch else None
    g = axi.AXI(nr, nz, tolcon=TOLCON, smoother=smoother, precision=precision, grid=grid)
    g.set("omegn", rhs)
    sweeps = g.poisson()
    phi = g.get("phi")
    g.close()
    return phi, sweeps


def _check(nr, nz, smoother, stretch):
    rng = np.random.default_rng(nr * 1000 + nz)
    r = np.linspace(0.0, 1.0, nr + 1)[:, None]
    z = np.linspace(0.0, 1.0, nz + 1)[None, :]
    rhs = sum(rng.standard_normal() * np.sin(a * np.pi * r) * np.sin(b * np.pi * z) for a in (1, 2, 5) for b in (1, 3, 4))
    p64, s64 = _solve(nr, nz, 0, smoother, stretch, rhs)
    p32, s32 = _solve(nr, nz, 1, smoother, stretch, rhs)
    assert 0 < s64 < 10000 and 0 < s32 < 10000
    assert np.abs(p64).max() > 1e-4
    assert np.abs(p32 - p64).max() <= (4 if stretch else 1) * BOUND


@pytest.mark.parametrize("nr,nz", [(4, 4), (8, 36), (32, 34), (34, 64), (66, 32), (64, 130), (130, 128), (256, 64),
                                   (258, 32), (64, 258), (512, 32), (16, 514)])
def test_uniform(nr, nz):
    _check(nr, nz, 1, 0.0)


@pytest.mark.parametrize("nr,nz", [(8, 8), (32, 36), (68, 32), (64, 132), (256, 64), (64, 260)])
def test_stretched(nr, nz):
    _check(nr, nz, 1, 1.0)


@pytest.mark.parametrize("stretch", [0.0, 1.0])
def test_reference_line_order(stretch):
    _check(32, 24, 0, stretch)
