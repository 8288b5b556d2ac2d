"""A stage kernel of the pool whose bounded wait expires writes the pool's status word, and
the next call that waits for the device reports it.  The word is set from the host here: no
wait of a kernel is made to run out."""
import ctypes as C

import numpy as np
import pytest

from nekwave_b200 import _lib
from nekwave_b200.pool import CavityPool

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["sync", "query", "query_end", "results"])
def test_an_expired_wait_is_reported_once(gpu, call):
    word = _lib.lib().nwb_pool_status_word_
    word.restype, word.argtypes = C.POINTER(C.c_int), [C.c_void_p]
    pool = CavityPool(64 << 20, max_slots=2)
    s = pool.add_box(5, (2, 2, 2), (0, 0, 0), (1, 1, 1), 1.0, 1e-3, 4)
    pool.init_pulse(s, [(1.0, 0.4, 0.5, 0.6, 0.2)] * 6)
    pool.step(2)
    pool.sync()  # nothing expired so far

    def wait():
        if call == "query_end":
            pool.query_begin()
            pool.query_end()
        elif call == "results":
            pool.results(s)
        else:
            getattr(pool, call)()

    word(pool._h)[0] = 1
    with pytest.raises(_lib.NwbError) as e:
        wait()
    assert e.value.status == _lib.NWB_ETIMEOUT and "bounded wait" in str(e.value)
    wait()
    pool.close()


def test_results_of_several_slots_at_once(gpu):
    """Threads that each read another slot's results share the pool's pinned block, one at a
    time; ctypes calls run side by side."""
    from concurrent.futures import ThreadPoolExecutor
    n = 6
    pool = CavityPool(256 << 20, max_slots=n)
    slots = [pool.add_box(4 + i % 3, (4, 3, 2), (0, 0, 0), (1, 1, 1), 1.0, 1e-3, 4) for i in range(n)]
    for i, s in enumerate(slots):
        pool.init_pulse(s, [(1.0 + i, 0.4, 0.5, 0.6, 0.2)] * 6)
    pool.step(4)
    want = [pool.results(s) for s in slots]
    with ThreadPoolExecutor(n) as ex:
        for _ in range(50):
            for w, r in zip(want, ex.map(pool.results, slots)):
                np.testing.assert_array_equal(r["state"], w["state"])
                np.testing.assert_array_equal(r["energy"], w["energy"])
    pool.close()
