"""Batches whose problems are all small enough for one block each (or a cluster
that repeats one block's cycles) are solved whole in one launch (k_local_solve): bit for bit the oracle's solutions and
cycle counts at every size from one interior point to the largest such problem,
in each precision, and the same endings as the level-by-level solve (cycle
limit, right-hand sides of zero and with a NaN)."""
import numpy as np
import pytest

from test_gpu_batch_parity import make_batch

pytestmark = pytest.mark.gpu

MODES = [(0, 1), (1, 1), (1, 3), (2, 1), (2, 4)]


@pytest.mark.parametrize("precision,inner", MODES)
@pytest.mark.parametrize("sizes", [[3], [5, 3], [9], [17, 9, 17], [33], [65, 3, 33, 5, 17, 9, 65], [65, 5, 33] * 8, [17, 3, 65] * 16,
                                   [9, 33, 17] * 32])   # eight, four, two and one CTA per problem
def test_matches_oracle(oracle, gblib, precision, inner, sizes):
    from codesthesis_dir_gb300.batch import BatchPoisson
    f = make_batch(sizes, 31)
    _, psi_o, cyc_o, rr_o = oracle.batch_solve(sizes, f, precision=precision, inner=inner)
    bp = BatchPoisson(sizes, precision=precision, inner=inner)
    st, psi, cyc, rr = bp.solve_host(f)
    assert st == 0 and bp.last_launches() == 1
    np.testing.assert_array_equal(cyc, cyc_o)
    np.testing.assert_array_equal(psi, psi_o)
    # the norm's sum runs in another order: 65^2 terms, each rounding 2^-53
    np.testing.assert_allclose(rr, rr_o, rtol=65 ** 2 * 2.0 ** -53 + 1e-9, atol=1e-25)


@pytest.mark.parametrize("precision,inner", MODES)
def test_endings_match_the_level_by_level_solve(gblib, precision, inner):
    """The persistent mode runs the operations level by level."""
    from codesthesis_dir_gb300.batch import BatchPoisson
    sizes = [65, 33, 17]
    f = make_batch(sizes, 4)
    f[65 * 65:65 * 65 + 33 * 33] = 0.0
    out = []
    for mode in (0, 1):
        bp = BatchPoisson(sizes, precision=precision, inner=inner, exec_mode=mode, max_cycles=2, rtol=1e-14)
        st, psi, cyc, _ = bp.solve_host(f)
        g = f.copy()
        g[-17 * 8] = np.nan
        out.append((st, psi, cyc, bp.solve_host(g)[0]))
    assert out[0][0] == out[1][0] == 1 and out[0][3] == out[1][3] != 0
    assert out[0][2][1] == 0
    np.testing.assert_array_equal(out[0][1], out[1][1])
    np.testing.assert_array_equal(out[0][2], out[1][2])
