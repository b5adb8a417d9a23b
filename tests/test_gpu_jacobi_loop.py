"""The resident driver's Jacobi loop (one cooperative launch) against the
per-call entry point: iteration counts, summaries, u and un (Mi) bit for bit at
tile edges, odd and even sweep counts, reflective faces, 16-row tiles and more
sweeps than one launch makes."""
import numpy as np
import pytest

from tealeaf_opencl_gb300 import decks, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("x,y,halo,iters,eps,extra", [
    (10, 10, 1, 1000, 1e-15, ""), (1, 1, 1, 7, 1e-12, ""), (31, 5, 2, 33, 1e-30, ""),
    (33, 6, 1, 32, 1e-30, "reflective_boundary"), (257, 131, 3, 15, 1e-30,
                                                   "tl_coefficient_inverse_density"),
    (40, 37, 1, 1100, 1e-30, ""), (2049, 2434, 1, 3, 1e-30, ""),
])
def test_loop_matches_per_call(x, y, halo, iters, eps, extra):
    deck = decks.five_state_deck(x, "jacobi", steps=2, eps=eps, max_iters=iters, halo=halo,
                                 y_cells=y, extra=extra)
    got = []
    for mode in (lib.DRIVER_PER_CALL, lib.DRIVER_RESIDENT):
        steps = lib.run_deck(deck, mode=mode)
        last = steps[-1]
        got.append(([s.iterations for s in steps], [s.conduction_error for s in steps],
                    (last.vol, last.mass, last.ie, last.temp),
                    [lib.read_field(f) for f in ("u", "Mi", "energy1")]))
    a, b = got
    assert a[0] == b[0] and a[2] == b[2]
    assert np.array_equal(a[1], b[1], equal_nan=True)
    for p, q in zip(a[3], b[3]):
        assert np.array_equal(p.view(np.int64), q.view(np.int64))
