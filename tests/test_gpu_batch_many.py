"""Batches of many small problems: as many as are still solved whole, one launch,
and one more, solved level by level; bit for bit the oracle's solutions and cycle
counts either way."""
import numpy as np
import pytest

from test_gpu_batch_parity import make_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,inner", [(0, 1), (1, 2), (2, 1)])
def test_either_side_of_the_rule(oracle, gblib, precision, inner):
    import torch
    from codesthesis_dir_gb300.batch import BatchPoisson
    most = 40 * torch.cuda.get_device_properties(0).multi_processor_count
    sizes = ([9, 3, 5, 17] * (most // 4 + 1))[:most + 1]
    f = make_batch(sizes, 5)
    _, psi_o, cyc_o, _ = oracle.batch_solve(sizes, f, precision=precision, inner=inner)
    for n in (most, most + 1):
        end = sum(s * s for s in sizes[:n])
        bp = BatchPoisson(sizes[:n], precision=precision, inner=inner)
        st, psi, cyc, _ = bp.solve_host(f[:end])
        assert st == 0 and (bp.last_launches() == 1) == (n == most)
        np.testing.assert_array_equal(cyc, cyc_o[:n])
        np.testing.assert_array_equal(psi, psi_o[:end])
