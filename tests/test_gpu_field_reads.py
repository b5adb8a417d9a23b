"""Field reads into every kind of host memory give the same bytes and write
nothing beside them: pages that nothing has touched, touched ones, a mixture,
blocks that begin inside a page, pinned memory; and a read into touched pages
costs about what one into pinned memory does."""
import ctypes
import mmap
import time

import numpy as np
import pytest

from tealeaf_opencl_gb300 import decks, lib

pytestmark = pytest.mark.gpu
N = 2000
BYTES = N * (N - 3) * 8
SLACK = 1 << 17


@pytest.fixture(scope="module")
def field():
    drv = lib.Driver(decks.five_state_deck(N, "cg", "none", steps=1, eps=1e-30, max_iters=3,
                                           y_cells=N - 3, summary_frequency=0), mode=1)
    drv.step()
    yield lib.read_field("u")
    drv.close()


def read(address):
    t = time.perf_counter()
    assert lib.load().tea_gb300_read_field(lib.FIELD["u"], ctypes.cast(address, lib.PD)) == 0
    return time.perf_counter() - t


@pytest.mark.parametrize("offset", [0, 8, 4096 + 24, 65536 - 8])
@pytest.mark.parametrize("touch", ["none", "all", "half", "last"])
def test_bytes_and_their_surroundings(field, offset, touch):
    m = mmap.mmap(-1, BYTES + 2 * SLACK)
    raw = np.frombuffer(m, dtype=np.uint8)
    lo = SLACK // 2 + offset
    if touch in ("all", "half"):
        raw[:raw.size // (1 if touch == "all" else 2)] = 7
    elif touch == "last":
        raw[-SLACK:] = 7
    before, after = raw[:lo].copy(), raw[lo + BYTES:].copy()
    read(ctypes.c_void_p(raw.ctypes.data + lo))
    got = raw[lo:lo + BYTES].view(np.float64).reshape(N - 3, N)
    assert np.array_equal(got.view(np.int64), field.view(np.int64))
    assert np.array_equal(raw[:lo], before) and np.array_equal(raw[lo + BYTES:], after)


def test_touched_pages_cost_what_pinned_memory_does(field):
    pinned = lib.load().tea_gb300_host_alloc(BYTES)
    try:
        best_pinned = min(read(ctypes.c_void_p(pinned)) for _ in range(9))
    finally:
        lib.load().tea_gb300_host_free(pinned)
    own = np.full(BYTES // 8, 1.0)
    best_own = min(read(ctypes.c_void_p(own.ctypes.data)) for _ in range(9))
    assert best_own < 2.5 * best_pinned
