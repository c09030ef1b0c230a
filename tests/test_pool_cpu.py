"""Bookkeeping of the device memory kept between uses, over a made-up device:
reuse, bounds, age, contexts that go away and come back, threads.  Addresses
are numbers; nothing is allocated or touched."""
import threading

import pytest

from airtoolsii_b200 import _lib

GB = 1 << 30
CTX, IDLE, PASS, GONE, ALLOC, GIVE, RELEASE, ADDR, GETS, PUTS, WRONG, TAKEN = range(12)


@pytest.fixture()
def pool():
    made = []

    def make(size=180 * GB):
        L = _lib.lib()
        h = L.airt_test_pool_new(size)
        made.append(h)
        return lambda op, arg=0: L.airt_test_pool_op(h, op, arg)
    yield make
    for h in made:
        _lib.lib().airt_test_pool_delete(h)


def test_blocks_of_about_the_size_are_reused(pool):
    p = pool()
    a = p(ALLOC, 1_000_000)
    p(GIVE, a)
    b = p(ALLOC, 990_000)
    assert p(ADDR, b) == p(ADDR, a) and p(GETS) == 1 and p(PUTS) == 0
    c = p(ALLOC, 500_000)                       # kept blocks of twice the size stay out of it
    assert p(GETS) == 2 and p(ADDR, c) != p(ADDR, b)


def test_release_gives_everything_back(pool):
    p = pool()
    held = p(ALLOC, 3 * GB)
    for n in (100, 5_000, GB):
        p(GIVE, p(ALLOC, n))
    p(RELEASE)
    assert p(TAKEN) == 3 * GB and p(WRONG) == 0
    p(GIVE, held)
    p(RELEASE)
    assert p(TAKEN) == 0 and p(PUTS) == p(GETS) and p(WRONG) == 0


def test_bounds(pool):
    p = pool()
    blocks = [p(ALLOC, GB) for _ in range(10)]
    for b in blocks:
        p(GIVE, b)
    assert p(TAKEN) == 6 * GB
    p = pool(10 * GB)                           # a small device: a quarter of what is free
    blocks = [p(ALLOC, GB) for _ in range(9)]
    for b in blocks:
        p(PASS, 2)                              # the free memory is asked for once a second
        p(GIVE, b)
    assert GB <= p(TAKEN) <= 2 * GB and p(WRONG) == 0
    assert p(ALLOC, 9 * GB) >= 0                # an allocation that does not fit empties the pool
    assert p(TAKEN) == 9 * GB


def test_the_oldest_blocks_make_room(pool):
    """A program that turns to other sizes is not left without kept blocks."""
    p = pool()
    old = [p(ALLOC, GB) for _ in range(6)]
    for b in old:
        p(PASS, 1)
        p(GIVE, b)
    for _ in range(3):                          # other sizes, a second later and within one
        a, b = p(ALLOC, GB // 2), p(ALLOC, GB // 2)
        p(GIVE, a)
        p(GIVE, b)
    assert p(GETS) == 8 and p(PUTS) == 1        # one old block went, the new ones are reused
    assert p(TAKEN) == 6 * GB
    assert p(ADDR, p(ALLOC, GB)) != p(ADDR, old[0])


def test_old_blocks_go_back(pool):
    p = pool()
    p(GIVE, p(ALLOC, GB))
    p(PASS, 20)
    p(GIVE, p(ALLOC, 4096))
    assert p(TAKEN) == GB + 4096
    p(PASS, 20)                                 # 40 s: the first one is old, the second is not
    p(ALLOC, 1 << 20)
    assert p(TAKEN) == 4096 + (1 << 20)


def test_a_block_is_not_kept_when_the_device_could_not_be_waited_for(pool):
    p = pool()
    a = p(ALLOC, GB)
    p(IDLE, 0)
    p(GIVE, a)
    assert p(TAKEN) == 0 and p(PUTS) == 1


def test_blocks_stay_in_their_context(pool):
    p = pool()
    a, b = p(ALLOC, GB), p(ALLOC, GB)
    p(GIVE, a)
    p(CTX, 2)                                   # another context of the same device
    c = p(ALLOC, GB)
    assert p(ADDR, c) not in (p(ADDR, a), p(ADDR, b)) and p(GETS) == 3
    p(GIVE, b)                                  # given up under the wrong context: freed, not kept
    assert p(PUTS) == 1 and p(WRONG) == 0
    p(RELEASE)
    assert p(PUTS) == 1                         # context 1 lives: its kept block stays
    p(CTX, 1)
    assert p(ADDR, p(ALLOC, GB)) == p(ADDR, a)


def test_nothing_of_a_context_that_is_gone_is_handed_out_or_freed(pool):
    p = pool()
    kept, held = p(ALLOC, GB), p(ALLOC, GB)
    p(GIVE, kept)
    p(GONE, 1)                                  # a reset: context 2 gets the same addresses
    p(CTX, 2)
    x, y = p(ALLOC, GB), p(ALLOC, GB)
    assert p(GETS) == 4
    assert {p(ADDR, x), p(ADDR, y)} == {p(ADDR, kept), p(ADDR, held)}
    p(GIVE, held)                               # an old handle: its address is y's by now
    assert p(PUTS) == 0 and p(TAKEN) == 2 * GB
    z = p(ALLOC, GB)
    assert p(ADDR, z) not in (p(ADDR, x), p(ADDR, y))
    p(RELEASE)
    assert p(PUTS) == 0 and p(WRONG) == 0 and p(TAKEN) == 3 * GB


def test_threads_never_share_a_block(pool):
    p = pool()
    mine, bad = {}, []
    lock = threading.Lock()

    def work(seed):
        for i in range(2000):
            b = p(ALLOC, 1000 * (1 + (seed + i) % 7))
            at = p(ADDR, b)
            with lock:
                if at in mine:
                    bad.append(at)
                mine[at] = seed
            with lock:
                del mine[at]
            p(GIVE, b)
    threads = [threading.Thread(target=work, args=(s,)) for s in range(4)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not bad and p(WRONG) == 0
    p(RELEASE)
    assert p(TAKEN) == 0
