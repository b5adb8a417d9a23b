"""A change of the arithmetic form between two timesteps takes effect in the
whole next step, also in the kernels that the resident driver replays from a
graph captured before it: every field as in the per-call driver, bit for bit."""
import numpy as np
import pytest

from tealeaf_opencl_gb300 import decks, lib

pytestmark = pytest.mark.gpu


def run(deck, mode, forms):
    L = lib.load()
    L.tea_gb300_set_resident_mode(1)  # the graph of passes at any size
    drv = lib.Driver(deck, mode=mode)
    try:
        infos = []
        for form in forms:
            assert L.tea_gb300_set_arithmetic(form) == 0
            infos.append(drv.step())
        return ([(s.iterations, s.inner_iterations) for s in infos],
                [lib.read_field(f) for f in ("u", "p", "r", "energy1")])
    finally:
        drv.close()
        L.tea_gb300_set_resident_mode(0)
        L.tea_gb300_set_arithmetic(1)


@pytest.mark.parametrize("solver,prec", [("cg", "jac_diag"), ("cg", "jac_block"),
                                         ("ppcg", "none"), ("chebyshev", "jac_diag")])
@pytest.mark.parametrize("forms", [(1, 0, 2), (2, 1, 0)])
def test_arithmetic_changed_between_steps(solver, prec, forms):
    deck = decks.five_state_deck(130, solver, prec, steps=3, eps=1e-13, max_iters=400,
                                 y_cells=97, inner_steps=6, presteps=12)
    want = run(deck, lib.DRIVER_PER_CALL, forms)
    got = run(deck, lib.DRIVER_RESIDENT, forms)
    assert got[0] == want[0]
    for a, b in zip(got[1], want[1]):
        assert np.array_equal(a.view(np.int64), b.view(np.int64))
