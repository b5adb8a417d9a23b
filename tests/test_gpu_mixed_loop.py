"""The mixed solve's FP32 inner loop (one cooperative launch per correction)
against the oracle bit for bit at the edges of its tiles: columns around a quad,
a tile and a supertile, rows around a strip, more supertiles than SMs, and an
inner solve that its iteration limit ends."""
import pytest

from oracle import oracle
from tealeaf_opencl_gb300 import decks, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("x,y,max_iters", [(5, 3, 400), (31, 5, 400), (35, 4, 400),
                                           (255, 9, 400), (259, 33, 400), (200, 640, 37)])
def test_inner_loop_matches_oracle(x, y, max_iters):
    deck = decks.five_state_deck(x, solver="cg", prec="jac_diag", steps=2, eps=1e-9,
                                 max_iters=max_iters, y_cells=y,
                                 extra="tl_mixed_precision\ntl_mixed_inner_eps 1e-4\n"
                                       "tl_mixed_max_outer 6")
    steps = lib.run_deck(deck)
    res = oracle.run_deck(deck)
    n = res.n_steps
    assert [s.iterations for s in steps] == list(res.iterations[:n])
    assert [s.outer_corrections for s in steps] == list(res.outer_corrections[:n])
    assert [s.relative_residual for s in steps] == list(res.relative_residual[:n])
    final = res.summaries()[-1]
    last = steps[-1]
    assert (last.vol, last.mass, last.ie, last.temp) == tuple(final[[1, 2, 4, 5]])
