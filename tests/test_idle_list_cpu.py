"""What threads leave behind for the next ones (idle_list.hpp), on the CPU."""
import ctypes
import os
import subprocess
import threading

import pytest

from conftest import HOSTMODEL_DIR, ROOT

SRC = os.path.join(HOSTMODEL_DIR, "idle_shim.cpp")
SO = os.path.join(HOSTMODEL_DIR, "_build", "libidle_shim.so")


@pytest.fixture(scope="module")
def L():
    hdr = os.path.join(ROOT, "bt-am_b200", "csrc", "idle_list.hpp")
    if (not os.path.exists(SO) or os.path.getmtime(SO) < max(os.path.getmtime(SRC),
                                                             os.path.getmtime(hdr))):
        os.makedirs(os.path.dirname(SO), exist_ok=True)
        subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-pthread", "-o", SO, SRC],
                       check=True)
    L = ctypes.CDLL(SO)
    L.il_create.restype = ctypes.c_void_p
    for f in (L.il_destroy, L.il_made, L.il_freed):
        f.argtypes = [ctypes.c_void_p]
    L.il_acquire.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.POINTER(ctypes.c_int),
                             ctypes.c_int]
    L.il_leave.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int]
    L.il_users.argtypes = [ctypes.c_void_p, ctypes.c_int]
    return L


class Thread:
    """One thread's view: its count of attempts and what it holds."""

    def __init__(self, L, p, dev=0):
        self.L, self.p, self.dev, self.asked, self.has = L, p, dev, ctypes.c_int(0), -1

    def ask(self, fails=0):
        if self.has < 0:
            self.has = self.L.il_acquire(self.p, self.dev, ctypes.byref(self.asked), fails)
        return self.has

    def end(self):
        if self.has >= 0:
            self.L.il_leave(self.p, self.dev, self.has)


def test_short_threads_in_turn_make_one(L):
    p = L.il_create()
    L.il_users(p, 1)
    for _ in range(100):
        t = Thread(L, p)
        assert t.ask() == 0
        t.end()
    assert (L.il_made(p), L.il_freed(p)) == (1, 0)
    L.il_users(p, -1)
    assert L.il_freed(p) == 1


def test_threads_beside_others_wait_for_theirs(L):
    p, patience = L.il_create(), L.il_patience()
    L.il_users(p, 1)
    first = Thread(L, p)
    assert first.ask() == 0
    short = [Thread(L, p) for _ in range(8)]
    for t in short:
        for _ in range(patience - 1):
            assert t.ask() == -1
    assert L.il_made(p) == 1
    assert short[0].ask() == 1  # stayed long enough
    short[0].end()
    assert short[1].ask() == 1  # left over
    first.end()
    assert short[2].ask() == 0
    assert L.il_made(p) == 2


def test_devices_bound_and_failures(L):
    p, patience = L.il_create(), L.il_patience()
    L.il_users(p, 1)
    t = Thread(L, p)
    assert t.ask(fails=1) == -1 and L.il_made(p) == 0
    assert t.ask() == 0  # a failed one does not count: still the first
    other = Thread(L, p, dev=1)
    t.end()
    assert all(other.ask() == -1 for _ in range(patience - 1))
    assert other.ask() == 1  # not the one of device 0
    more = [Thread(L, p) for _ in range(L.il_idle() + 3)]
    for m in more:
        for _ in range(patience):
            m.ask()
        assert m.has >= 0
    assert len({m.has for m in more}) == len(more)
    for m in more:
        m.end()
    other.end()
    assert L.il_freed(p) == L.il_made(p) - L.il_idle()
    L.il_users(p, -1)
    assert L.il_freed(p) == L.il_made(p)
    late = Thread(L, p)  # a thread that outlives the last user frees its own
    assert late.ask() >= 0
    late.end()
    assert L.il_freed(p) == L.il_made(p)


def test_many_threads_at_once(L):
    """No two threads hold the same one, and all of them come back."""
    p, patience = L.il_create(), L.il_patience()
    L.il_users(p, 1)
    held, lock, twice = set(), threading.Lock(), []

    def work():
        t = Thread(L, p)
        for _ in range(2 * patience):
            if t.has < 0 and t.ask() >= 0:
                with lock:
                    if t.has in held:
                        twice.append(t.has)
                    held.add(t.has)
        with lock:
            held.discard(t.has)
        t.end()

    for _ in range(20):
        ts = [threading.Thread(target=work) for _ in range(16)]
        for x in ts:
            x.start()
        for x in ts:
            x.join()
    assert not twice and not held
    assert L.il_made(p) - L.il_freed(p) <= L.il_idle()
    L.il_users(p, -1)
    assert L.il_made(p) == L.il_freed(p)
