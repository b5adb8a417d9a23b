"""Which form the resident driver takes (one launch, or kernels) by the work
per SM: tiles of 16 rows count as four of 4, so grids on the far side of the
change of tile height stay with the kernels; and what a single iteration
takes."""
import pytest

from tealeaf_opencl_gb300 import decks, lib

pytestmark = pytest.mark.gpu


def launches(deck, resident_mode=0, mode=lib.DRIVER_RESIDENT, steps=1):
    """Kernel launches of the last of `steps` timesteps."""
    L = lib.load()
    L.tea_gb300_set_resident_mode(resident_mode)
    drv = lib.Driver(deck, mode=mode)
    try:
        for _ in range(steps):
            n0 = L.tea_gb300_kernel_launches()
            drv.step()
        return L.tea_gb300_kernel_launches() - n0
    finally:
        drv.close()
        L.tea_gb300_set_resident_mode(0)


def sms():
    torch = pytest.importorskip("torch")
    return torch.cuda.get_device_properties(0).multi_processor_count


# 4-row supertiles of 1501 columns: six a row of tiles
@pytest.mark.parametrize("prec,form,lo,hi", [("jac_diag", "fused", 12, 12), ("none", "chain", 14, 14),
                                             ("jac_block", "exact", 14, 14)])
def test_cg_form_follows_the_work_per_sm(prec, form, lo, hi):
    for per_sm, one_launch in ((lo, True), (hi + 0.2, False)):
        y = 4 * int(per_sm * sms() / 6)
        assert lib.load().tea_gb300_reduction_rows(1501, y) == 4
        deck = decks.five_state_deck(1501, "cg", prec, steps=1, eps=1e-30, max_iters=40, y_cells=y,
                                     extra="tl_arithmetic " + form, summary_frequency=0)
        assert launches(deck, 2) < launches(deck, 1)
        assert launches(deck) == launches(deck, 2 if one_launch else 1), (per_sm, one_launch)


@pytest.mark.parametrize("n", [2176, 2500])
def test_grids_of_16_row_tiles_take_the_kernels(n):
    assert lib.load().tea_gb300_reduction_rows(n, n) == 16
    deck = decks.five_state_deck(n, "cg", "jac_diag", steps=1, eps=1e-30, max_iters=20,
                                 summary_frequency=0)
    assert launches(deck) == launches(deck, 1) > launches(deck, 2)
    deck = decks.five_state_deck(n, "jacobi", steps=1, eps=1e-30, max_iters=20,
                                 summary_frequency=0)
    assert launches(deck) == launches(deck, mode=lib.DRIVER_PER_CALL)


def test_jacobi_form_follows_the_work_per_sm():
    for per_sm, one_launch in ((18, True), (18.2, False)):
        y = 4 * int(per_sm * sms() / 6)
        deck = decks.five_state_deck(1501, "jacobi", steps=1, eps=1e-30, max_iters=20, y_cells=y,
                                     summary_frequency=0)
        per_call = launches(deck, mode=lib.DRIVER_PER_CALL)
        assert launches(deck) == (per_call - 19 if one_launch else per_call)


@pytest.mark.parametrize("prec", ["jac_diag", "jac_block"])
def test_one_cg_iteration_is_made_per_call(prec):
    """PPCG's single CG iteration of the later timesteps takes neither form of
    the loop."""
    deck = decks.five_state_deck(100, "ppcg", prec, steps=2, eps=1e-30, max_iters=200,
                                 y_cells=70, inner_steps=4, presteps=10, summary_frequency=0,
                                 extra="tl_ch_cg_epslim=1e30")
    assert launches(deck, 1, steps=1) > launches(deck, 2, steps=1)
    assert launches(deck, 1, steps=2) == launches(deck, 2, steps=2)
