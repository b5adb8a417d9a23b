"""The kernel timer (tea_gb300_kernel_timer_select) sees the kernels of the
resident driver's Jacobi sweeps and of its CG iterations before the switch to
Chebyshev or PPCG, with the results of a run without it."""
import ctypes

import numpy as np
import pytest

from tealeaf_opencl_gb300 import decks, lib

pytestmark = pytest.mark.gpu


def run(deck):
    steps = lib.run_deck(deck, mode=lib.DRIVER_RESIDENT)
    return ([(s.iterations, s.inner_iterations, s.switch_iteration) for s in steps],
            lib.read_field("u"))


def launches(name):
    ms, n = ctypes.c_double(), ctypes.c_longlong()
    lib.load().tea_gb300_kernel_timer_read_name(name.encode(), ctypes.byref(ms), ctypes.byref(n))
    return n.value if ms.value > 0.0 else 0


@pytest.mark.parametrize("solver,name,count", [
    ("jacobi", "tea_leaf_jacobi_solve", lambda s: sum(i for i, _, _ in s)),
    ("chebyshev", "tea_leaf_cg_solve_calc_w", lambda s: sum(w - 1 for _, _, w in s)),
    ("ppcg", "tea_leaf_cg_solve_calc_p", lambda s: sum(w - 1 for _, _, w in s)),
])
def test_timer_sees_the_solver_kernels(solver, name, count):
    L = lib.load()
    deck = decks.five_state_deck(60, solver, "none", steps=2, eps=1e-9, max_iters=60, y_cells=45,
                                 presteps=8, inner_steps=4, extra="tl_ch_cg_epslim=1e30")
    plain = run(deck)
    L.tea_gb300_kernel_timer_select(b"*")
    try:
        timed = run(deck)
        assert launches(name) == count(timed[0]) > 0
    finally:
        L.tea_gb300_kernel_timer_select(b"")
    assert timed[0] == plain[0]
    assert np.array_equal(timed[1].view(np.int64), plain[1].view(np.int64))
