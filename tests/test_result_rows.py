"""Result arrays in page-locked memory: blocks live as long as any view of them, are used again, bounded and given back."""
import ctypes as C
import gc
import threading

import numpy as np

from wayruntime_b200.binding import _ResultRows


class FakeLib:
    """wr_cuda_host_alloc / wr_cuda_host_release on ordinary memory."""

    def __init__(self, fail=False):
        self.live, self.made, self.fail = {}, 0, fail

    def wr_cuda_host_alloc(self, handle, size, out):
        if self.fail:
            return -5
        block = C.create_string_buffer(size)
        out._obj.value = C.addressof(block)
        self.live[out._obj.value] = block
        self.made += 1
        return 0

    def wr_cuda_host_release(self, p):
        del self.live[p]


def test_a_block_is_used_again_only_when_no_view_of_it_is_left():
    lib = FakeLib()
    rows = _ResultRows(lib, 1)
    a = rows.empty((16, 40000))
    a[:] = np.arange(16)[:, None]
    view = a[3:4]
    at = a.ctypes.data
    del a
    gc.collect()
    b = rows.empty((16, 40000))
    b[:] = -1
    assert lib.made == 2 and b.ctypes.data != at and (view == 3).all()
    del view
    c = rows.empty((14, 40000))                       # the same size class
    assert lib.made == 2 and c.ctypes.data == at and c.shape == (14, 40000) and c.dtype == np.float32


def test_small_results_and_those_beyond_the_limit_are_ordinary_arrays():
    lib = FakeLib()
    rows = _ResultRows(lib, 1)
    rows.LIMIT = 1 << 22
    assert rows.empty((1, 100)).base is None and lib.made == 0
    kept = [rows.empty((1, 1 << 18)) for _ in range(6)]
    assert lib.made == 4 and all(k.size == 1 << 18 for k in kept)
    del kept
    other = rows.empty((1, 1 << 19))                  # idle blocks of another size make room
    assert lib.made == 5 and len(lib.live) == 1 and other.nbytes == 1 << 21
    assert _ResultRows(FakeLib(fail=True), 1).empty((1, 1 << 18)).base is None


def test_what_is_held_at_close_goes_with_its_array():
    lib = FakeLib()
    rows = _ResultRows(lib, 1)
    a, b = rows.empty((1, 1 << 16)), rows.empty((1, 1 << 16))
    del b
    rows.close()
    assert len(lib.live) == 1 and rows.empty((1, 1 << 16)).base is None
    a[:] = 1
    del a
    gc.collect()
    assert not lib.live


def test_threads_take_and_give_back():
    lib = FakeLib()
    rows = _ResultRows(lib, 1)
    bad = []

    def work(i):
        for j in range(200):
            a = rows.empty((1 + j % 3, 1 << 15))
            a[:] = i
            if not (a == i).all():
                bad.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad and lib.made <= 3 * 8 * 2           # (three size classes, an old and a new array per thread)


def test_arrays_made_together_go_one_by_one():
    lib = FakeLib()
    rows = _ResultRows(lib, 1)
    some, at = rows.many(16, (1, 40000))
    assert at == [a.ctypes.data for a in some]
    for i, a in enumerate(some):
        a[:] = i
    assert lib.made == 16 and len({a.ctypes.data for a in some}) == 16
    kept = some[5]
    del some, a
    gc.collect()
    more, _ = rows.many(16, (1, 40000))                  # fifteen blocks are free again, the kept row's is not
    for a in more:
        a[:] = -1
    assert lib.made == 17 and (kept == 5).all()
    rows.LIMIT = lib.made << 18
    del more, a
    assert [a.base is None for a in rows.many(18, (1, 40000))[0]] == [False] * 16 + [True] * 2


def test_an_engine_gives_every_session_a_row_of_its_own():
    from wayruntime_b200.engine import Engine

    class Model:
        FWD_DECODE, FWD_PREFILL, ROWS_APART, vocab, max_rows = 0, 1, True, 40000, 64
        rows = _ResultRows(FakeLib(), 1)

        def kv_create(self, n):
            return None

        def forward(self, mode, kvs, positions, tokens, out_from=0, *, logits=False, argmax=False, apart=False):
            assert apart and mode == self.FWD_DECODE
            out, _ = self.rows.many(len(logits), (1, self.vocab))
            for a, i in zip(out, logits):
                a[:] = tokens[i]
            return {"logits": out}

    e = Engine(Model())
    got = e.advance([e.session(8) for _ in range(6)], [[i] for i in range(6)], [[0], [], [0], [0, 0], [0], [0]])
    for i, g in enumerate(got):
        assert g.shape == (([1, 0, 1, 2, 1, 1][i]), 40000) and (g == i).all()
    assert not any(np.shares_memory(a, b) for i, a in enumerate(got) for b in got[:i])
    assert Model.rows._bytes == 5 << 18
