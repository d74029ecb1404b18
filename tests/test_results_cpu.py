"""Memory that a model keeps for its results (dsk._Results), on a stand-in for the library's pinned memory: parts that are out at a time never overlap and all come
back, also where the cycle collector or other threads give arrays back in the middle of a call."""
import ctypes
import gc
import random
import threading

import numpy as np
import pytest

import dsk


class HostMemory:
    def __init__(self):
        self.blocks = {}

    def dsk_host_alloc(self, n):
        b = ctypes.create_string_buffer(n)
        self.blocks[ctypes.addressof(b)] = b
        return ctypes.addressof(b)

    def dsk_host_free(self, p):
        del self.blocks[p]


class Cycle:
    """An array that only the cycle collector gives back."""
    def __init__(self, a):
        self.a, self.me = a, self


def span(a):
    lo = a.__array_interface__["data"][0]
    return lo, lo + a.nbytes


def pinned(mem, a):
    return any(p <= span(a)[0] and span(a)[1] <= p + len(b) for p, b in mem.blocks.items())


def check(mem, res, held):
    """Arrays that are out lie inside of the memory or are ordinary ones, and none meets another."""
    spans = sorted(span(a) for a in held)
    assert all(x[1] <= y[0] for x, y in zip(spans, spans[1:]))
    for lo, hi in spans:
        assert all(hi <= p or lo >= p + len(b) or (lo >= p and hi <= p + len(b)) for p, b in mem.blocks.items())


@pytest.fixture
def thresholds():
    old = gc.get_threshold()
    yield gc.set_threshold
    gc.set_threshold(*old)
    gc.collect()


@pytest.mark.parametrize("seed", range(6))
def test_collected_in_the_middle_of_a_call(thresholds, seed):
    rng, mem = random.Random(seed), HostMemory()
    res = dsk._Results(mem, 2 << 20)
    whole, held = res.holes, []
    for _ in range(3000):
        thresholds(rng.randint(2, 60), 2, 2)
        a = res.rows((rng.randint(1, 40), rng.choice([5000, 16384, 20000])))
        held.append(a)
        check(mem, res, held)
        for _ in range(rng.randint(0, 2)):
            if held:
                Cycle(held.pop(rng.randrange(len(held))))
        while len(held) > 12:
            held.pop(0)
        del a
    thresholds(700, 10, 10)
    held.clear()
    gc.collect()
    assert res.live == 0 and res.holes == whole
    a = res.rows((2, 65536))
    res.close()
    assert mem.blocks and pinned(mem, a)
    Cycle(a)
    del a
    gc.collect()
    assert not mem.blocks and res.base is None


def test_threads():
    mem = HostMemory()
    res = dsk._Results(mem, 4 << 20)
    whole, wrong = res.holes, []

    def work(k):
        rng = random.Random(k)
        mine = []
        for i in range(400):
            a = res.rows((rng.randint(1, 8), 20000))
            a[:] = k
            mine.append(a)
            if len(mine) > 4:
                b = mine.pop(rng.randrange(len(mine)))
                if not np.all(b == k):
                    wrong.append(k)
    threads = [threading.Thread(target=work, args=(k,)) for k in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    gc.collect()
    assert not wrong and res.live == 0 and res.holes == whole
    res.close()
    assert not mem.blocks


def test_small_and_large_results_are_ordinary_arrays():
    mem = HostMemory()
    res = dsk._Results(mem, 1 << 20)
    assert not pinned(mem, res.rows((1, 10))) and not pinned(mem, res.rows((1, 1 << 20))) and pinned(mem, res.rows((4, 20000)))
    res.close()
    gc.collect()
    assert not mem.blocks and not pinned(mem, res.rows((4, 20000)))


def test_no_pinned_memory_to_be_had():
    class Refusing(HostMemory):
        def dsk_host_alloc(self, n):
            return None
    res = dsk._Results(Refusing(), 1 << 20)
    a = res.rows((4, 20000))
    a[:] = 1.0
    assert res.live == 0 and res.base is None
    res.close()
