"""The uniform grid's FP32 quotients (mer_quot) where they are formed the other
way: operands too small or too large for the corrections, and a divisor out of
range on every point.  Equal, bit for bit, to the plain restatement of
test_gpu_mixed_serial_order.py, which divides; both sides do IEEE operations
(denormals included), so there is no tolerance."""
import numpy as np
import pytest

from test_gpu_mixed_serial_order import _solve

pytestmark = pytest.mark.gpu


# (zmax, scale): right-hand sides whose corrections lie around 2^-95 and below, or
# above 2^95; a spacing hz with hz^2 above 2^24 or below 2^-24 (with a scale that
# keeps the corrections inside the floats)
@pytest.mark.parametrize("zmax,scale", [(0.5, 1.0), (0.5, 1e-26), (0.5, 1e-30), (0.5, 1e31), (4e5, 1.0), (2e-3, 1.0), (2e-3, 1e-24)])
@pytest.mark.parametrize("nr,nz", [(10, 14), (34, 66)])
def test_equals_division(gblib, nr, nz, zmax, scale):
    from codesthesis_dir_gb300 import axi
    rng = np.random.default_rng(nr * 1000 + nz)
    rhs = np.zeros((nr + 1, nz + 1))
    rhs[1:-1, 1:-1] = scale * rng.standard_normal((nr - 1, nz - 1))
    want, cycles, tolcon = _solve(nr, nz, 0.5, 1.0, zmax, rhs, 0.7, 2)
    g = axi.AXI(nr, nz, r0=0.5, rmax=1.0, zmax=zmax, tolcon=tolcon, smoother=1, precision=1, nrel=2)
    g.set("omegn", rhs)
    assert g.poisson() == cycles > 0
    np.testing.assert_array_equal(g.get("phi"), want)
    g.close()
