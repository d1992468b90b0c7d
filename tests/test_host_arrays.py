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
    if a.nbytes >= HUGE:   # (smaller ones start on a page)
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


def mapped_mb():
    with open("/proc/self/statm") as f:
        return int(f.read().split()[0]) * os.sysconf("SC_PAGE_SIZE") / 1e6


def test_freed_memory_is_kept_up_to_a_bound():
    """Dropped arrays are found again, and no more of them than 512 MB is held."""
    shape = (10 * HUGE // 8 - 3,)
    a = L._host_array(shape)
    at = a.ctypes.data
    a.fill(2.0)
    del a
    b = L._host_array(shape)
    assert b.ctypes.data == at          # the last one freed
    b.fill(3.0)
    del b
    gc.collect()
    before = mapped_mb()
    many = [L._host_array((HUGE // 8 * k,)) for k in range(1, 60)]   # 3.5 GB, not touched
    assert mapped_mb() - before > 3000
    del many
    gc.collect()
    assert mapped_mb() - before < 600
    # blocks of other sizes make room for those freed last
    a = L._host_array(shape)
    at = a.ctypes.data
    del a
    b = L._host_array(shape)
    assert b.ctypes.data == at
    small = [L._host_array((20000 + 100 * k,)) for k in range(400)]
    at = small[-1].ctypes.data
    while small:
        small.pop(0)
    assert L._host_array((20000 + 100 * 399,)).ctypes.data == at


def test_allocation_from_several_threads():
    def work(seed):
        rng = np.random.default_rng(seed)
        held = []
        for _ in range(60):
            n = int(rng.integers(HUGE // 8, 4 * HUGE // 8))
            a = L._host_array((n,))
            a[0] = a[-1] = a[n // 2] = seed
            held.append(a)
            if len(held) > 5:
                x = held.pop(int(rng.integers(len(held))))
                assert x[0] == x[-1] == x[len(x) // 2] == seed
        good.append(all(x[0] == x[-1] == seed for x in held))

    good = []
    threads = [threading.Thread(target=work, args=(i + 1,)) for i in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert good == [True] * 8
