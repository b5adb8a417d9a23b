"""The exact form's two passes per CG iteration, whose products run on the
integer pipes, against the per-call kernels bit for bit: 16- and 4-row tiles,
rows cut by the top edge, reflective faces, each preconditioner."""
import numpy as np
import pytest

from tealeaf_opencl_gb300 import decks, lib

pytestmark = pytest.mark.gpu


def run(deck, mode, resident_mode=0):
    L = lib.load()
    L.tea_gb300_set_resident_mode(resident_mode)
    try:
        steps = lib.run_deck(deck, mode=mode)
    finally:
        L.tea_gb300_set_resident_mode(0)
        L.tea_gb300_set_arithmetic(1)
    return [s.iterations for s in steps], [lib.read_field(f) for f in ("u", "p", "r", "w")]


@pytest.mark.parametrize("x,y,prec,iters,extra", [
    (2049, 2434, "none", 9, ""), (2049, 2433, "jac_block", 8, "reflective_boundary"),
    (2240, 2401, "jac_diag", 7, ""), (611, 607, "none", 30, "reflective_boundary"),
    (33, 6, "jac_block", 30, ""), (4, 3, "none", 11, "")])
def test_exact_passes_match_per_call(x, y, prec, iters, extra):
    deck = decks.five_state_deck(x, "cg", prec, steps=2, eps=1e-30, max_iters=iters, y_cells=y,
                                 extra="tl_arithmetic exact\n" + extra)
    want = run(deck, lib.DRIVER_PER_CALL)
    for resident_mode in (1, 2):
        got = run(deck, lib.DRIVER_RESIDENT, resident_mode)
        assert got[0] == want[0]
        for a, b in zip(got[1], want[1]):
            assert np.array_equal(a.view(np.int64), b.view(np.int64)), resident_mode


@pytest.mark.parametrize("form", ["exact", "fused", "chain"])
@pytest.mark.parametrize("x,y", [(70, 45), (611, 607), (2049, 2434)])
def test_true_residual_exit_without_preconditioner_is_the_plain_exit(form, x, y):
    """r.z is r.r without a preconditioner, so both exits end at one iteration."""
    extra = "tl_arithmetic %s\n" % form
    deck = decks.five_state_deck(x, "cg", "none", steps=2, eps=1e-3, max_iters=60, y_cells=y,
                                 extra=extra)
    want = run(deck, lib.DRIVER_RESIDENT, 1)
    got = run(deck.replace(extra, extra + "tl_exit_true_residual\n"), lib.DRIVER_RESIDENT)
    assert got[0] == want[0] and max(want[0]) > 1
    for a, b in zip(got[1], want[1]):
        assert np.array_equal(a.view(np.int64), b.view(np.int64))
