"""CPU: blocks of large result arrays come back only when the last view is gone,
from any thread, and no more than a few are kept."""
import gc
import threading

import numpy as np
import pytest

from desi_b200.api import _Results


@pytest.mark.parametrize("view", [lambda a: a.reshape(200, 200)[3:], lambda a: a[5:], lambda a: memoryview(a),
                                  lambda a: a.view(np.int64)])
def test_a_view_keeps_its_block(view):
    pool = _Results()
    a = pool.take(40000)
    at, v = a.ctypes.data, view(a)
    del a
    gc.collect()
    assert pool.take(40000).ctypes.data != at
    del v
    gc.collect()
    taken = [pool.take(40000) for _ in range(2)]
    assert at in [t.ctypes.data for t in taken]
    taken[0][:] = 1.0
    assert taken[0].sum() == 40000.0


def test_sizes_outside_the_range_are_plain_arrays():
    pool = _Results()
    for n in (1, _Results.LOW // 8 - 1, _Results.HIGH // 8 + 1):
        a = pool.take(n)
        assert a.shape == (n,) and a.flags.owndata and not a.any()
    assert not pool._spare


def test_bounded_and_returned_from_threads():
    pool = _Results()
    held = [pool.take(40000 + k % 6) for k in range(40)]
    t = threading.Thread(target=held.clear)
    t.start()
    t.join()
    gc.collect()
    assert len(pool._spare) <= 4 and sum(len(d) for d in pool._spare.values()) <= 16
