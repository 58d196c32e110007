"""The memory of returned arrays (verion_gb300.backend._HostPages): reuse, its bound, views that outlive their array,
several threads, and collections that drop or ask for arrays inside its own calls."""
import gc
import threading

import numpy as np
import pytest

from verion_gb300.backend import _HostPages


class Pages(_HostPages):
    LEAST, KEEP = 1 << 12, 1 << 18  # four blocks of the least size (64 KiB)


N = 1 << 16


def idle(p):
    return sum(b for b, _ in p._idle)


def test_dropped_memory_is_used_again_up_to_the_bound():
    p = Pages()
    a = p.empty(N, np.uint8)
    at = a.ctypes.data
    view = a[10:20]
    del a
    gc.collect()
    assert idle(p) == 0  # the view still holds it
    del view
    assert idle(p) == N
    assert p.empty(N // 4, np.float32).ctypes.data == at
    many = [p.empty(N, np.uint8) for _ in range(9)]
    del many
    assert idle(p) == Pages.KEEP
    big = p.empty(2 * Pages.KEEP, np.uint8)
    del big
    assert idle(p) <= Pages.KEEP


class Hooked(list):
    """A list that runs `hook` at every look at it, as a collection at that point would."""

    def __init__(self, hook):
        super().__init__()
        self.hook, self.inside = hook, False

    def _run(self):
        if not self.inside:
            self.inside = True
            self.hook()
            self.inside = False

    def __len__(self):
        self._run()
        return super().__len__()

    def __getitem__(self, i):
        self._run()
        return super().__getitem__(i)

    def __iter__(self):
        self._run()
        return super().__iter__()


@pytest.mark.parametrize("what", ["drops", "asks"])
def test_a_collection_inside_its_calls(what):
    p = Pages()
    waiting, runs = [], [0]

    def hook():
        runs[0] += 1
        if what == "drops":
            if waiting:
                waiting.pop()
        elif runs[0] <= 100:
            assert p.empty(N, np.uint8).size == N

    p._idle = Hooked(lambda: None)
    first = [p.empty(N * (1 + k % 2), np.uint8) for k in range(4)]
    waiting.extend(p.empty(N * (1 + k % 3), np.uint8) for k in range(12))
    del first
    p._idle.hook = hook
    for k in range(12):
        a = p.empty(N * (1 + k % 2), np.uint8)
        a[:] = k
        assert a.size == N * (1 + k % 2) and (a == k).all()
        del a
    p._idle.hook = lambda: None
    assert runs[0] > 0
    waiting.clear()
    p.empty(N, np.uint8)
    assert idle(p) <= Pages.KEEP


def test_several_threads():
    p = Pages()
    bad = []

    def work(k):
        rng = np.random.default_rng(k)
        held = []
        for i in range(300):
            a = p.empty(int(rng.integers(1, 4)) * N // 4, np.uint32)
            a[:] = k << 16 | i
            held.append((a, k << 16 | i))
            if len(held) > 3:
                b, want = held.pop(int(rng.integers(4)))
                if not (b == want).all():
                    bad.append(k)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    p._settle()
    assert not bad and not p._returned and idle(p) <= Pages.KEEP
