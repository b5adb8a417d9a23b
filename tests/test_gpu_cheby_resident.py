"""Chebyshev decks in the resident driver, whose CG iterations before the
switch run in the device loop, against the oracle: iteration counts, the
iteration of the switch and the field summary of every step, at one prestep, at
a deck that converges before it switches, and in each form of the loop."""
import pytest

from oracle import oracle
from tealeaf_opencl_gb300 import decks, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("resident_mode", [0, 1, 2])
@pytest.mark.parametrize("prec,form,presteps,eps,steps", [
    ("jac_diag", "chain", 20, 1e-13, 3), ("none", "exact", 1, 1e-8, 2),
    ("jac_block", "fused", 12, 1e-12, 2), ("jac_diag", "fused", 30, 1e-2, 2)])
def test_resident_chebyshev_matches_oracle(prec, form, presteps, eps, steps, resident_mode):
    L = lib.load()
    deck = decks.five_state_deck(147, "chebyshev", prec, steps=steps, eps=eps, max_iters=3000,
                                 y_cells=118, presteps=presteps, summary_frequency=1,
                                 extra="tl_arithmetic %s" % form)
    res = oracle.run_deck(deck)
    per_call = lib.run_deck(deck)
    L.tea_gb300_set_resident_mode(resident_mode)
    try:
        got = lib.run_deck(deck, mode=lib.DRIVER_RESIDENT)
    finally:
        L.tea_gb300_set_resident_mode(0)
    n = res.n_steps
    assert [s.iterations for s in got] == list(res.iterations[:n])
    assert [s.switch_iteration for s in got] == [s.switch_iteration for s in per_call]
    assert (got[0].switch_iteration == 0) == (eps > 1e-3)
    final = res.summaries()[-1]
    last = got[-1]
    assert (last.vol, last.mass, last.ie, last.temp) == tuple(final[[1, 2, 4, 5]])
