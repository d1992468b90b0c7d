"""Arrays that downloads return: ordinary ones that own their memory, large
ones starting on a huge page."""
import gc
import os
import pickle
import threading

import numpy as np
import pytest

import lbm_b200 as L

HUGE = 1 << 21


# below, at and above a huge page; an extent of one and an empty array
@pytest.mark.parametrize("shape", [(3, 5, 7), (0, 4, 4), (64, 64, 63), (64, 64, 64), (64, 65, 64), (131, 75, 90), (500000,)])
def test_download_arrays_own_their_memory(shape):
    a, b = L._host_array(shape), np.empty(shape)
    assert type(a) is np.ndarray and a.base is None
    assert (a.shape, a.dtype, a.strides) == (b.shape, b.dtype, b.strides)
    assert str(a.flags) == str(b.flags)
    if a.nbytes >= HUGE:
        assert a.ctypes.data % HUGE == 0
    a[...] = 1.5
    assert pickle.loads(pickle.dumps(a)).sum() == a.sum()
    a.resize(a.size + 300000, refcheck=False)   # in place, larger and smaller
    assert np.count_nonzero(a) == b.size and (a[:b.size] == 1.5).all()
    a.resize(5, refcheck=False)
    assert a.size == 5


def test_other_arrays_keep_their_allocator():
    from numpy._core.multiarray import get_handler_name
    a = L._host_array((64, 64, 64))
    assert get_handler_name(a) == "lbm_b200_pages"
    assert get_handler_name(np.empty((64, 64, 64))) == "default_allocator"
    names = []
    t = threading.Thread(target=lambda: names.append(get_handler_name(np.empty((64, 64, 64)))))
    t.start()
    t.join()
    assert names == ["default_allocator"]


def test_memory_is_given_back():
    def resident():
        with open("/proc/self/statm") as f:
            return int(f.read().split()[1]) * os.sysconf("SC_PAGE_SIZE")

    L._host_array((HUGE // 8,)).fill(1.0)
    gc.collect()
    before = resident()
    for _ in range(50):
        L._host_array((10 * HUGE // 8 + 1,)).fill(1.0)
    assert resident() - before < 64 << 20
