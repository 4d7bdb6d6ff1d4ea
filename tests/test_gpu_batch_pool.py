"""A batch over new decks grows the device's memory pool before its workers start, in one step, and not
under them (where a growth stalls the other streams): the pool's reserved bytes are read from a second thread
while the call runs."""
import ctypes
import threading

import numpy as np
import pytest

import ferrix_b200 as fx
from ferrix_b200 import decks

pytestmark = pytest.mark.gpu


def _reserved():
    cuda = ctypes.CDLL("libcuda.so.1")
    pool, value = ctypes.c_void_p(), ctypes.c_uint64()
    assert cuda.cuDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0
    reserved_mem_current = 5  # CUmemPool_attribute
    assert cuda.cuMemPoolGetAttribute(pool, reserved_mem_current, ctypes.byref(value)) == 0
    return value.value


@pytest.mark.parametrize("npe,cells", [(4, (20, 20, 40)), (20, (10, 10, 24))])
def test_new_decks(npe, cells):
    ctx = fx.Context(0)
    projects = []
    for k in range(8):
        lengths = tuple(float(c + k) for c in cells)
        mesh = decks.tet_box(*cells, *lengths) if npe == 4 else decks.hex20_box(*cells, *lengths)
        spec = decks.DeckSpec(mesh, [(2.0e5, 0.3, None)], load_total=(1.0, 2.0, 3.0))
        p = fx.Project.from_arrays(**decks.deck_arrays(spec), ctx=ctx)
        fx.SolutionState(p.num_dofs, p.num_nodes).initialize(p)
        projects.append(p)
    seen, stop = [_reserved()], threading.Event()

    def watch():
        while not stop.is_set():
            v = _reserved()
            if v != seen[-1]:
                seen.append(v)

    t = threading.Thread(target=watch)
    t.start()
    try:
        status, _ = fx.batch_solve(ctx, projects)
    finally:
        stop.set()
        t.join()
    seen.append(_reserved())
    for p in projects:
        p.close()
    ctx.close()
    assert np.all(status == 0)
    assert len(set(seen)) <= 2, seen  # before, and after the one growth
