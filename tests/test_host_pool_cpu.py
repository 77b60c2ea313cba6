"""The pool of page-locked blocks under downloads: what it keeps, what it gives back, and what it refuses."""
import ctypes
import os
import random
import subprocess
import threading

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
MB = 1 << 20


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    path = tmp_path_factory.mktemp("pool") / "libpool.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-pthread", os.path.join(HERE, "host_pool_shim.cpp"), "-o", str(path)], check=True)
    L = ctypes.CDLL(str(path))
    vp = ctypes.c_void_p
    L.pool_new.restype = L.pool_take.restype = vp
    L.pool_take.argtypes = [vp, ctypes.c_size_t]
    L.pool_give.argtypes = [vp, vp]
    for name in ("pool_delete", "pool_join", "pool_leave"):
        getattr(L, name).argtypes = [vp]
    for name in ("pool_locks", "pool_unlocks", "pool_live"):
        getattr(L, name).restype = ctypes.c_long
    return L


class Pool:
    def __init__(self, lib):
        self.lib, self.h = lib, lib.pool_new()
        self.before, self.taken = lib.pool_locks(), []
        lib.pool_join(self.h)

    def take(self, size):
        p = self.lib.pool_take(self.h, size)
        self.taken.append(p)
        return p

    def give(self, p):
        self.lib.pool_give(self.h, p)

    def locks(self):
        return self.lib.pool_locks() - self.before


@pytest.fixture
def pool(lib):
    live = lib.pool_live()
    p = Pool(lib)
    yield p
    for block in p.taken:
        p.give(block)
    lib.pool_leave(p.h)
    lib.pool_delete(p.h)
    assert lib.pool_live() == live


def test_a_released_block_serves_the_next_download(pool):
    a = pool.take(5000)
    pool.give(a)
    assert pool.take(8192) == a and pool.take(8192) != a and pool.locks() == 2


@pytest.mark.parametrize("times", [2, 3])
def test_a_block_released_twice_is_handed_out_once(pool, times):
    a = pool.take(4096)
    for _ in range(times):
        pool.give(a)
    pool.give(ctypes.addressof(ctypes.create_string_buffer(1)))            # not the pool's
    b, c = pool.take(4096), pool.take(4096)
    assert b != c


def test_blocks_stay_within_the_limit(pool):
    """256 MB in all, 64 MB in one block; a refused request leaves the kept blocks alone."""
    assert pool.take(64 * MB + 1) is None and pool.take((1 << 63) + 1) is None
    small = pool.take(4096)
    pool.give(small)
    large = [pool.take(64 * MB) for _ in range(3)]
    fourth = pool.take(64 * MB)
    assert all(large) and fourth is None
    assert pool.take(4096) == small                                          # still locked
    assert pool.take(32 * MB) and pool.take(32 * MB) is None


@pytest.mark.parametrize("sizes,together", [([64 * MB] * 5 + [4096, 1280000], True), ([200 * MB, 4096, 1280000], False)])
def test_a_loop_over_more_than_the_limit_locks_nothing_again(pool, sizes, together):
    """Fields of one round that do not fit, held together or one after the other: what fits is kept, the rest is refused."""
    rounds = []
    for _ in range(6):
        got = []
        for size in sizes:
            got.append(pool.take(size))
            if not together and got[-1]:
                pool.give(got[-1])
        rounds.append(pool.locks())
        for p in got if together else []:
            if p:
                pool.give(p)
    assert rounds[1:] == rounds[:1] * 5


def test_idle_blocks_make_room(pool):
    old = [pool.take(64 * MB) for _ in range(4)]
    for p in old:
        pool.give(p)
    assert pool.take(4096) is None                                           # just used: part of the caller's loop
    one = None
    for _ in range(300):
        one = pool.take(4096) or one
        if one:
            break
    assert one


def test_nothing_is_kept_without_a_user(lib):
    live = lib.pool_live()
    p = Pool(lib)
    a, b = p.take(4096), p.take(1 * MB)
    p.give(a)
    lib.pool_join(p.h)
    lib.pool_leave(p.h)
    assert lib.pool_live() == live + 2                                       # one user is left
    lib.pool_leave(p.h)
    assert lib.pool_live() == live + 1                                       # an array still stands on b
    p.give(b)
    assert lib.pool_live() == live
    lib.pool_delete(p.h)


def test_refused_pages_cost_no_room(pool, lib):
    lib.pool_refuse(1)
    assert [pool.take(64 * MB) for _ in range(8)] == [None] * 8
    lib.pool_refuse(0)
    got = [pool.take(64 * MB) for _ in range(4)]
    assert all(got)


def test_threads_never_share_a_block(pool):
    held, lock, errors = set(), threading.Lock(), []

    def work(seed):
        rng, mine = random.Random(seed), []
        for _ in range(400):
            if mine and rng.random() < 0.5:
                p = mine.pop(rng.randrange(len(mine)))
                with lock:
                    held.discard(p)
                pool.give(p)
            else:
                p = pool.take(rng.choice([1000, 5000, 100000, 3 * MB]))
                if p is None:
                    continue
                with lock:
                    if p in held:
                        errors.append(p)
                    held.add(p)
                mine.append(p)
        for p in mine:
            with lock:
                held.discard(p)
            pool.give(p)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
