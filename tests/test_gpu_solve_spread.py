"""gb_prb_set_solve_spread changes the clusters of an instance's solves between
steps and, with 0, gives the default back; the bits stay those of an instance
without a call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
def test_default_spread_can_be_asked_for_again(gblib, precision):
    from codesthesis_dir_gb300 import initial, lib, prb
    out = []
    for spreads in ((None, None, None), (8, 1, 0)):
        g = prb.PRB(32, 64, dt=1e-5, r0=0.0, rmax=1.0, xx=2.0, Ra=1e5, Pr=1.0, smoother=lib.SMOOTHER_ZEBRA, precision=precision)
        for name, a in initial.initial_fields(32, 64, 0.0, 1.0, 0, 1, 3, 1e-3).items():
            g.set(name, a)
        got = []
        for s in spreads:
            if s is not None:
                g.set_solve_spread(s)
            got += [*g.step(2)]
        out.append(got + [g.get(n) for n in ("C", "th", "vel", "uel")])
        for bad in (-1, 2, 16):
            assert gblib.gb_prb_set_solve_spread(g._h, bad) == lib.GB_ERR_INVALID
        g.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
