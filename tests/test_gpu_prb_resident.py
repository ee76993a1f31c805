"""The velocity solves on one CTA, on a cluster of 8 and on the largest
cluster, in shared memory or (lines or grids too long for it) on global
memory: the same bits, at line lengths around the layouts' edges (32, 64,
128, 256, 512 rows), more CTAs than lines, few and many levels, every
operator (layer, annulus, tank).  The FP64 solve on one of them equals the
oracle (test_gpu_prb_parity.py, test_gpu_annulus_parity.py, test_gpu_tank.py)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (nr, np, variant, tolcon): the tolerance is far above the residual's rounding
# floor eps |A| |psi| of each grid (at most 1e-16 * 4 nr^2 * 1)
LAYER, ANNULUS, TANK = 0, 1, 4
CASES = [(8, 16, LAYER), (16, 64, LAYER), (32, 32, LAYER), (34, 8, LAYER), (66, 16, LAYER), (128, 256, LAYER), (130, 16, LAYER),
         (256, 32, LAYER), (260, 16, LAYER), (520, 16, LAYER), (16, 32, ANNULUS), (96, 64, ANNULUS), (136, 400, ANNULUS),
         (16, 32, TANK), (64, 96, TANK), (128, 256, TANK)]


def _solve(nr, np_, variant, precision, spread):
    from codesthesis_dir_gb300 import lib, prb
    r0 = 0.5 if variant == ANNULUS else 0.0
    g = prb.PRB(nr, np_, dt=1e-5, r0=r0, rmax=1.0, xx=2.0, Ra=1e5, Pr=1.0, Re=100.0 if variant == ANNULUS else 0.0,
                tolcon=1e-6, maxsweeps=60, smoother=lib.SMOOTHER_ZEBRA, precision=precision, variant=variant)
    if spread:
        g.set_solve_spread(spread)
    rng = np.random.default_rng(nr + 7 * np_ + variant)
    shape = (nr + 2, g.ncol)
    for name, amp in (("vrh", 1.0), ("urh", 1.0), ("vel", 1e-3), ("uel", 1e-3), ("velp", 1e-3), ("uelp", 1e-3)):
        a = np.zeros(shape)
        a[1:-1] = amp * rng.standard_normal((nr, g.ncol))
        g.set(name, a)
    out = []
    for solve, fields in (("poisson2", ("vel", "velp")), ("poisson3", ("uel", "uelp"))):
        try:
            out.append(getattr(g, solve)())
        except lib.GBError as e:   # the sweep limit: fields as the solve leaves them
            assert e.status == lib.GB_MAXSWEEPS
            out.append(-1)
        out += [g.get(n) for n in fields]
    g.close()
    return out


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
@pytest.mark.parametrize("nr,np_,variant", CASES)
def test_same_bits_on_every_cluster_size(nr, np_, variant, precision):
    if precision and variant == TANK:
        pytest.skip("the tank runs in FP64")
    one = _solve(nr, np_, variant, precision, 1)
    assert np.abs(one[1]).max() > 0
    for spread in (8, 0):
        for a, b in zip(one, _solve(nr, np_, variant, precision, spread)):
            np.testing.assert_array_equal(a, b)
