"""The 3D annulus's line phases at the sizes where their layouts change: line
lengths around 32, 64, 128, 256 and 512 rows in each direction, one and
several levels, fewer lines than blocks and lines longer than the staging
buffers.

FP64 (two-colour and reference order) equals the oracle bit for bit.  The mixed
solve stops at the same residual bound as the FP64 solve of the same
equation, so the residual of their difference is below twice the bound (plus
the REAL*4 literal's part, 3e-8 |psi| / h^2, which is below it here); on the
unit-size domain |A^-1| <= 0.5^2 / 8 in the maximum norm (r- and z-gaps 0.5,
Dirichlet walls; the one-sided wall rows make that approximate: a factor 4)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(4, 4, 16), (8, 8, 8), (16, 12, 24), (36, 8, 16), (8, 68, 16), (12, 8, 136), (8, 8, 264), (8, 12, 520), (136, 8, 8), (8, 264, 8)]
FIELDS = {1: ("wel", "welp", "wrh"), 2: ("vel", "velp", "vrh"), 3: ("uel", "uelp", "urh")}


def _random(shape, seed, comp):
    nr, nz = shape[0] - 2, shape[1] - 2
    rng = np.random.default_rng(seed)
    a = np.zeros(shape, order="F")
    ii, jj = (nr - 1 if comp == 3 else nr), (nz - 1 if comp == 1 else nz)
    a[1:ii + 1, 1:jj + 1, 1:] = rng.standard_normal((ii, jj, shape[2] - 1))
    a[:, :, 0] = a[:, :, -1]
    return a


def _solve(nr, nz, np_, comp, precision, smoother, tolcon):
    from codesthesis_dir_gb300 import r3d
    g = r3d.R3D(nr, nz, np_, Ra=1e5, Re=100.0, Pr=0.7, smoother=smoother, precision=precision, tolcon=tolcon)
    psi, psip, rhs = FIELDS[comp]
    g.set(rhs, _random(g.shape, 5, comp))
    g.set(psi, 1e-3 * _random(g.shape, 6, comp))
    g.set(psip, 1e-3 * _random(g.shape, 7, comp))
    sweeps = g.poisson(comp)
    out = g.get(psi), g.get(psip), sweeps
    g.close()
    return out


@pytest.mark.parametrize("smoother", [0, 1], ids=["lex", "zebra"])
@pytest.mark.parametrize("nr,nz,np_", SIZES)
def test_fp64_equals_oracle(oracle, gblib, nr, nz, np_, smoother):
    from codesthesis_dir_gb300 import lib
    if smoother == lib.SMOOTHER_LEX and max(nr, nz, np_) > 140:
        pytest.skip("the reference order's wavefronts at these lengths are covered by the shorter ones")
    for comp in (1, 2, 3):
        o = oracle.OracleR3D(nr, nz, np_, 1e-5, 0.5, 1.0, 0.5, 1e5, 100.0, 0.7, mode=smoother, tolcon=1e-3)
        psi, psip, rhs = FIELDS[comp]
        shape = np.array(o.field(psi)).shape
        o.field(rhs)[...] = _random(shape, 5, comp)
        o.field(psi)[...] = 1e-3 * _random(shape, 6, comp)
        o.field(psip)[...] = 1e-3 * _random(shape, 7, comp)
        st, sw = o.poisson(comp)
        assert st == 0
        a, b, sweeps = _solve(nr, nz, np_, comp, 0, smoother, 1e-3)
        assert sweeps == sw
        np.testing.assert_array_equal(a, np.array(o.field(psi)))
        np.testing.assert_array_equal(b, np.array(o.field(psip)))


@pytest.mark.parametrize("nr,nz,np_", SIZES)
def test_mixed_meets_the_same_bound(gblib, nr, nz, np_):
    for comp in (1, 2, 3):
        a, _, sa = _solve(nr, nz, np_, comp, 0, 1, 1e-3)
        b, _, sb = _solve(nr, nz, np_, comp, 1, 1, 1e-3)
        assert sa > 0 and sb > 0
        assert np.abs(a - b).max() <= 4 * 2 * 1e-3 * 0.5 ** 2 / 8
