"""The FP32 register tiles (op_tile32) where their layout changes: grids whose
last tile ends on the domain's edge, before it and one column after it, several
tiles both ways, every halo (0 to 6: sweeps per pass 0, 1 and 2, with and
without the restriction) and the three ways of storing (into the level, added
to an FP64 and to a float-pair solution).  Bit for bit the oracle's solutions
and cycle counts (the operations are the same and in the same order)."""
import numpy as np
import pytest

from test_gpu_batch_parity import make_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [1, 2])
@pytest.mark.parametrize("nu1,nu2,inner,local_n,fuse", [(2, 2, 1, 33, 2), (1, 1, 3, 65, 2), (2, 0, 2, 65, 2), (3, 4, 1, 129, 1)])
def test_matches_oracle(oracle, gblib, precision, nu1, nu2, inner, local_n, fuse):
    from codesthesis_dir_gb300.batch import BatchPoisson
    sizes = [1025, 65, 129, 257, 33, 513]
    f = make_batch(sizes, 23)
    st_o, psi_o, cyc_o, _ = oracle.batch_solve(sizes, f, nu1=nu1, nu2=nu2, precision=precision, inner=inner)
    t = dict(nu1=nu1, nu2=nu2, inner=inner, local_n=local_n, fuse=fuse, exec=0)
    st, psi, cyc, _ = BatchPoisson(sizes, precision=precision, tuning=t).solve_host(f)
    assert st == st_o
    np.testing.assert_array_equal(cyc, cyc_o)
    np.testing.assert_array_equal(psi, psi_o)
