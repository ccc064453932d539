"""The host side of the quantified tables (no GPU needed): columns gathered by native threads
into memory that is reused once its tables are gone."""
import gc
import threading

import numpy as np
import pytest

from alphadia_search_rs_b200 import api


def columns(rng, n_src, n_rows):
    srcs = [rng.integers(0, 255, n_src).astype(t) for t in (np.uint8, np.float32, np.uint64)]
    rows = rng.integers(0, n_src, n_rows)
    rows[:2] = 0, n_src - 1
    return [(s, r) for s in srcs for r in (rows, None)]


@pytest.mark.parametrize("n_src,n_rows", [(1, 100_000), (70_000, 65_535), (70_000, 65_536), (70_000, 65_537),
                                          (300_001, 500_000), (1000, 10)])
def test_gathered_columns(n_src, n_rows):
    """Elements of 1, 4 and 8 bytes, gathered and copied, around the 65,536 rows of a piece."""
    cols = columns(np.random.default_rng(n_src), n_src, n_rows)
    for got, (s, r) in zip(api._gather_columns(cols), cols):
        want = s.copy() if r is None else s[r]
        assert got.dtype == want.dtype and np.array_equal(got, want)
        assert got.flags.writeable and got.flags.c_contiguous


@pytest.mark.parametrize("at", [0, 65_536, 199_999])
@pytest.mark.parametrize("row", [5000, 2**40, -1])
def test_row_past_the_source(at, row):
    rows = np.zeros(200_000, np.int64)
    rows[at] = row
    with pytest.raises(ValueError):
        api._gather_columns([(np.zeros(5000, np.float32), rows)])


def test_memory_of_tables_still_held_is_not_reused():
    held = []
    for i in range(30):
        cols = columns(np.random.default_rng(i), 90_000, 120_000)
        out = api._gather_columns(cols)
        # of some tables one column, a part of one, or its bytes
        held.append((out[i % 6][i:70_000:3] if i % 2 else out[i % 6].view(np.uint8), i))
        del out
    for a, i in held:
        s, r = columns(np.random.default_rng(i), 90_000, 120_000)[i % 6]
        want = s if r is None else s[r]
        assert np.array_equal(a, want[i:70_000:3] if i % 2 else want.view(np.uint8))


def test_kept_memory_is_bounded_and_given_back():
    blocks = api._HostBlocks()
    blocks.LOCKED, blocks.KEPT = 0, 256 << 20  # ordinary memory alone
    assert blocks.empty(10, np.float32).base is None  # small ones are numpy's own
    a = blocks.empty(10**6, np.float32)
    b = blocks.empty(10**6, np.float32)
    first = a.ctypes.data
    del a
    gc.collect()
    assert 4 * 10**6 <= blocks.kept <= 4.6 * 10**6
    a = blocks.empty(10**6 - 7, np.uint32)
    assert a.ctypes.data == first and blocks.kept == 0 and len(a) == 10**6 - 7
    del a, b
    many = [blocks.empty(40_000_000 + i * 6_000_000, np.uint8) for i in range(40)]  # 6.3 GB, untouched
    del many
    gc.collect()
    assert blocks.kept <= blocks.KEPT
    big = blocks.empty(blocks.KEPT + 1, np.uint8)
    del big
    gc.collect()
    assert blocks.kept <= blocks.KEPT


def test_blocks_of_several_threads():
    blocks = api._HostBlocks()
    blocks.LOCKED = 600_000  # of both kinds
    faults = []

    def work(t):
        rng = np.random.default_rng(t)
        held = []
        for i in range(400):
            n = int(rng.integers(20_000, 60_000))
            a = blocks.empty(n, np.uint32)
            a[:] = t * 1000 + i
            held.append((a, t * 1000 + i))
            if len(held) > 5:
                x, v = held.pop(int(rng.integers(0, 6)))
                if not (x == v).all():
                    faults.append((t, i))
        if any(not (x == v).all() for x, v in held):
            faults.append(t)

    threads = [threading.Thread(target=work, args=(t,)) for t in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not faults and blocks.kept <= blocks.KEPT and blocks.locked <= blocks.LOCKED


def test_page_locked_memory_is_bounded(monkeypatch):
    """However many tables a caller holds, at most LOCKED bytes of them are page-locked
    (_host_empty, whose allocator takes powers of two and keeps them)."""
    out = {}  # address -> bytes, of the page-locked arrays that are out
    most = [0]

    class Locked(np.ndarray):
        def __del__(self):
            out.pop(self.__dict__.get("key"), None)

    def page_locked(n, dtype):
        a = np.empty(n, dtype).view(Locked)
        a.key = (a.ctypes.data, a.nbytes)
        out[a.key] = 1 << (a.nbytes - 1).bit_length()
        most[0] = max(most[0], sum(out.values()))
        return a

    monkeypatch.setattr(api, "_host_empty", page_locked)
    monkeypatch.setattr(api, "_HOST_BLOCKS", api._HostBlocks())
    limit = 16 << 20
    monkeypatch.setattr(api._HostBlocks, "LOCKED", limit)
    cols = columns(np.random.default_rng(1), 70_000, 200_000)  # 5.2 MB of tables
    held = [api._gather_columns(cols) for _ in range(8)]
    assert limit // 2 < most[0] <= limit
    for tables in held:
        for got, (s, r) in zip(tables, cols):
            assert np.array_equal(got, s if r is None else s[r])
    del held, tables, got
    gc.collect()
    most[0] = 0
    api._gather_columns(cols)
    assert 0 < most[0] <= limit  # those let go are page-locked memory's again
