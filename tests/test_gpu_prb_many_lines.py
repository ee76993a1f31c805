"""FP64 velocity solves in shared memory whose short lines put more than 512 on
a CTA (256 of a colour, one each for its threads) or just reach that: the bits
of the solve on a cluster of 8 or, where that holds as many, on global memory,
whose batches are bounded by the block."""
import numpy as np
import pytest

from test_gpu_prb_resident import ANNULUS, LAYER, TANK, _solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr,np_,variant", [(4, 512, LAYER), (4, 516, LAYER), (4, 980, LAYER), (6, 750, ANNULUS), (8, 528, LAYER),
                                            (8, 528, TANK), (4, 8256, LAYER), (6, 8256, ANNULUS)])
def test_same_bits_with_many_lines_per_cta(nr, np_, variant):
    want = _solve(nr, np_, variant, 0, 8)
    assert np.abs(want[1]).max() > 0
    for spread in (1, 0):
        for a, b in zip(want, _solve(nr, np_, variant, 0, spread)):
            np.testing.assert_array_equal(a, b)
