"""With no device memory left for a second buffer, the calls that would use
one take the path that needs none, with the same results: the resident CG loop
and the CG iterations before a switch (second p), Jacobi sweeps and Chebyshev
iterations with a point preconditioner (second u)."""
import numpy as np
import pytest

from tealeaf_opencl_gb300 import decks, lib

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
# a field of 2600 x 2500 cells takes 52 MiB: room for a chunk's 17, not for 18
KEEP = (17 * 52 + 30) << 20


def fill():
    held = []
    size = 16 << 30
    while size >= 2 << 20:
        if torch.cuda.mem_get_info()[0] - size < KEEP:
            size //= 2
            continue
        try:
            held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
        except torch.cuda.OutOfMemoryError:
            size //= 2
    return held


@pytest.mark.parametrize("solver,prec,mode", [
    ("cg", "jac_diag", lib.DRIVER_RESIDENT), ("jacobi", "none", lib.DRIVER_PER_CALL),
    ("jacobi", "none", lib.DRIVER_RESIDENT), ("chebyshev", "none", lib.DRIVER_PER_CALL),
    ("chebyshev", "jac_diag", lib.DRIVER_RESIDENT)])
def test_calls_without_room_for_a_second_buffer(solver, prec, mode):
    deck = decks.five_state_deck(2600, solver, prec, steps=1, eps=1e-30, max_iters=30,
                                 y_cells=2500, presteps=8, halo=2, summary_frequency=0,
                                 extra="tl_ch_cg_epslim=1e30")

    def run(tight):
        lib.load().tea_gb300_finalise()  # the chunk of the run before
        held = fill() if tight else []
        drv = lib.Driver(deck, mode=mode)
        try:
            if tight:  # the chunk has its fields and no room for one more
                assert torch.cuda.mem_get_info()[0] < 50 << 20
            info = drv.step()
            return info.iterations, [lib.read_field(f) for f in ("u", "p", "r", "w", "Mi")]
        finally:
            del held
            torch.cuda.empty_cache()
            drv.close()

    lib.run_deck(deck, mode=lib.DRIVER_PER_CALL)  # its kernels are loaded
    want, got = run(False), run(True)
    assert got[0] == want[0]
    for a, b in zip(got[1], want[1]):
        assert np.array_equal(a.view(np.int64), b.view(np.int64))
