"""The device-resident CG loop in both its forms (one cooperative launch, two
kernels per iteration from a graph) against the per-call entry points, which
are pinned to the oracle: iteration counts, summaries and every field the
loop writes, bit for bit, at the edges of its tiles (one cell, columns and
rows around 32, 256 and 4, strips cut by the top row, 16-row tiles) and past
the iterations of one launch."""
import numpy as np
import pytest

from tealeaf_opencl_gb300 import decks, lib

pytestmark = pytest.mark.gpu
FIELDS = ("u", "p", "r", "w", "energy1")


def run(deck, mode, resident_mode=0):
    L = lib.load()
    L.tea_gb300_set_resident_mode(resident_mode)
    try:
        steps = lib.run_deck(deck, mode=mode)
        prec = "z" if "preconditioner" in deck else "r"
        fields = [lib.read_field(f) for f in FIELDS + (prec,)]
    finally:
        L.tea_gb300_set_resident_mode(0)
    last = steps[-1]
    return ([s.iterations for s in steps], (last.vol, last.mass, last.ie, last.temp),
            fields)


def same_bits(a, b):
    """Equal bit patterns, any NaN equal to any NaN (a 1x1 grid divides 0 by
    0, on the host or on the GPU, which give NaNs of different signs)."""
    return np.all((a.view(np.int64) == b.view(np.int64)) | (np.isnan(a) & np.isnan(b)))


@pytest.mark.parametrize("x,y,halo,prec,form,iters,extra", [
    (1, 1, 1, "none", "fused", 40, ""),
    (31, 5, 2, "jac_diag", "chain", 60, ""),
    (33, 17, 1, "jac_block", "fused", 60, "reflective_boundary"),
    (256, 7, 3, "jac_block", "exact", 60, ""),
    (257, 130, 1, "jac_diag", "exact", 60, "tl_coefficient_inverse_density"),
    (64, 66, 1, "none", "chain", 1100, ""),
    (609, 611, 2, "jac_block", "chain", 25, "reflective_boundary"),
    (2049, 2433, 1, "jac_diag", "chain", 13, ""),
    (2049, 2434, 1, "jac_block", "fused", 12, ""),
])
def test_loop_matches_per_call(x, y, halo, prec, form, iters, extra):
    deck = decks.five_state_deck(x, "cg", prec, steps=2, eps=1e-30 if iters > 1000 else 1e-16,
                                 max_iters=iters, halo=halo, y_cells=y,
                                 extra="tl_arithmetic %s\n%s" % (form, extra))
    ref = run(deck, lib.DRIVER_PER_CALL)
    for resident_mode in (0, 1, 2):
        got = run(deck, lib.DRIVER_RESIDENT, resident_mode)
        assert got[0] == ref[0], resident_mode
        assert np.array_equal(got[1], ref[1], equal_nan=True), resident_mode
        for name, a, b in zip(FIELDS + ("z",), got[2], ref[2]):
            assert same_bits(a, b), (resident_mode, name)
