"""A PRB gang's solve spread changed while steps queued on the caller's stream
have not run: every step runs with the plan it was queued with, so the members'
results are those of stepping them alone."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
def test_spread_changed_under_queued_steps(gblib, precision):
    import torch
    from codesthesis_dir_gb300 import initial, lib, prb
    shapes, steps = ((16, 32), (64, 128), (32, 64)), 13
    insts, alone = [], []
    for nr, np_ in shapes:
        for store in (insts, alone):
            g = prb.PRB(nr, np_, dt=1e-5, r0=0.0, rmax=1.0, xx=2.0, Ra=1e5, Pr=1.0, tolcon=1e-8, smoother=lib.SMOOTHER_ZEBRA,
                        precision=precision)
            for name, a in initial.initial_fields(nr, np_, 0.0, 1.0, 0, 1, 3, 1e-3).items():
                g.set(name, a)
            store.append(g)
    for g in insts:
        assert gblib.gb_prb_run_begin(g._h, steps) == 0
        assert gblib.gb_prb_run_enqueue(g._h, 1, 1) == 0
    gang, n = C.c_void_p(), len(insts)
    assert gblib.gb_prb_gang_create((C.c_void_p * n)(*[g._h.value for g in insts]), (C.c_int * n)(*[steps] * n), n, C.byref(gang)) == 0
    stream = torch.cuda.Stream()
    for spread in (1, 8, 1, 8):
        assert gblib.gb_prb_gang_set_solve_spread(gang, spread) == 0
        assert gblib.gb_prb_gang_enqueue(gang, 3, stream.cuda_stream) == 0
    stream.synchronize()
    for g, a in zip(insts, alone):
        nu, sw, done = np.zeros((steps, 2)), np.zeros((steps, 2), dtype=np.int32), C.c_int()
        assert gblib.gb_prb_run_end(g._h, steps, nu.ctypes.data, sw.ctypes.data, C.byref(done)) == 0
        assert done.value == steps
        nu_a, sw_a = a.step(steps)
        np.testing.assert_array_equal(nu, nu_a)
        np.testing.assert_array_equal(sw, sw_a)
        for name in ("C", "th", "vel", "uel"):
            np.testing.assert_array_equal(g.get(name), a.get(name), err_msg=name)
    gblib.gb_prb_gang_destroy(gang)
