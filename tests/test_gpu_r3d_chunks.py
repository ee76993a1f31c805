"""3D FP64 line phases whose blocks fill a chunk of staged lines and go on to a
second one, the sizes where an even number of lines takes the row pitch of the
next odd number: bit for bit the oracle's step.  128 x 64 x 256 (a block of the
w and v solves' half grid has 54 r-lines of 128 rows, 108 z-lines of 63 and 27
phi-lines of 256) and 64 x 64 x 384 (14 phi-lines of 384).  And phi-lines longer
than the staging area, up to the longest that a solve takes; their mixed solve
stops at the same residual bound (the derivation stands in test_gpu_r3d_lines.py)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ["A", "Ap", "B", "Bp", "C", "Cp", "th", "thp", "uel", "vel", "wel", "uelp", "velp", "welp"]


@pytest.mark.parametrize("nr,nz,np_", [(128, 64, 256), (64, 64, 384), (4, 4, 5640), (4, 4, 12288)])
def test_step_equals_oracle(oracle, gblib, nr, nz, np_):
    from codesthesis_dir_gb300 import lib, r3d
    prm = dict(dt=1e-5, r0=0.5, rmax=1.0, zmax=0.5, Ra=1e5, Re=100.0, Pr=0.7)
    tolcon = 1e3   # one cycle a solve
    o = oracle.OracleR3D(nr, nz, np_, *prm.values(), mode=lib.SMOOTHER_ZEBRA, tolcon=tolcon)
    o.initial(3, 5e-2)
    rng = np.random.default_rng(3)
    for n in ("A", "B", "C"):
        o.field(n)[...] = rng.standard_normal(o.shape)
        o.field(n + "p")[...] = o.field(n)
    g = r3d.R3D(nr, nz, np_, smoother=lib.SMOOTHER_ZEBRA, tolcon=tolcon, **prm)
    for n in FIELDS:
        g.set(n, np.array(o.field(n)))
    st, nu_o, sw_o = o.step()
    assert st == 0
    nu, sw = g.step(1)
    np.testing.assert_array_equal(sw[0], sw_o)
    assert nu[0] == nu_o
    assert np.abs(np.array(o.field("wel"))).max() > 0
    for n in FIELDS:
        np.testing.assert_array_equal(g.get(n), np.array(o.field(n)), err_msg=n)
    g.close()


@pytest.mark.parametrize("comp", [1, 2, 3])
def test_longest_mixed_rings(gblib, comp):
    from test_gpu_r3d_lines import _solve
    a, _, sa = _solve(4, 4, 12288, comp, 0, 1, 1e-3)
    b, _, sb = _solve(4, 4, 12288, comp, 1, 1, 1e-3)
    assert sa > 0 and sb > 0
    assert np.abs(a - b).max() <= 4 * 2 * 1e-3 * 0.5 ** 2 / 8
