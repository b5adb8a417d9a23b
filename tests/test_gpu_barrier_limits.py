"""tea_gb300_set_barrier_limits governs every kernel whose blocks meet at a
grid barrier: with one arrival more than the grid has and a short poll limit,
each call returns its error (a wait of a few ms, no fault), and the same call
with the normal limits then gives what it gave before."""
import ctypes

import numpy as np
import pytest

from tealeaf_opencl_gb300 import decks, lib

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def limits():
    L = lib.load()
    L.tea_gb300_set_abort_on_error(0)
    L.tea_gb300_last_error(None, 0)
    yield
    L.tea_gb300_set_barrier_limits(1 << 26, 0)
    L.tea_gb300_last_error(None, 0)


def deck_run(solver, prec, extra=""):
    deck = decks.five_state_deck(90, solver, prec, steps=1, eps=1e-9, max_iters=400, y_cells=71,
                                 presteps=10, inner_steps=5, extra=extra)

    def call():
        steps = lib.run_deck(deck, mode=lib.DRIVER_RESIDENT)
        return [s.iterations for s in steps], lib.read_field("energy1")
    return call


def batch_run():
    b = lib.Batch([(70, 33), (40, 90)])
    for i in range(2):
        x, y = b.sizes[i]
        b.set_fields(i, np.full((y, x), 2.0), 1.0 + np.arange(x * y).reshape(y, x) % 7)
    b.set_launch(1, persistent=1)

    def call():
        for i in range(2):
            x, y = b.sizes[i]
            b.set_fields(i, np.full((y, x), 2.0), 1.0 + np.arange(x * y).reshape(y, x) % 7)
        b.run(1, 0.004, 1e-10, 500)
        return [b.iterations(0), b.iterations(1)], b.read(0, "u")
    call.done = b.free
    return call


def adjoint_run():
    torch = pytest.importorskip("torch")
    adj = lib.Adjoint(65, 40)
    density = torch.full((40, 65), 3.0, dtype=torch.float64, device="cuda")
    energy = (1.0 + torch.arange(40 * 65, device="cuda", dtype=torch.float64) % 5).reshape(40, 65)
    out = torch.zeros_like(density)
    cfg = adj.config(2, 0.004, 1e-11, 500, 1)
    torch.cuda.synchronize()

    def call():
        _, st = adj.forward(density, energy, None, out, cfg)
        return [st.forward_iterations], out.cpu().numpy()
    call.done = adj.free
    return call


@pytest.mark.parametrize("make,code", [
    (lambda: deck_run("cg", "jac_block"), 25), (lambda: deck_run("jacobi", "none"), 25),
    (lambda: deck_run("chebyshev", "none"), 25),
    (lambda: deck_run("cg", "jac_diag", "tl_mixed_precision"), 25), (adjoint_run, 61),
    (batch_run, 57)], ids=["cg", "jacobi", "chebyshev", "mixed", "adjoint", "batch"])
def test_time_out_is_an_error_and_leaves_the_context_usable(make, code):
    L = lib.load()
    call = make()
    try:
        want = call()
        assert L.tea_gb300_set_barrier_limits(1 << 12, 1) == 0
        with pytest.raises(lib.TeaError) as err:
            call()
        assert "error %d" % code in str(err.value), str(err.value)
        assert L.tea_gb300_set_barrier_limits(1 << 26, 0) == 0
        L.tea_gb300_last_error(None, 0)
        got = call()
    finally:
        getattr(call, "done", lambda: None)()
    assert got[0] == want[0]
    assert np.array_equal(got[1], want[1])
