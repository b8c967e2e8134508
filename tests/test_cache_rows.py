"""The block table's rows as arrays follow the tables through reservations, windows that pass pages, and steps that did not run."""

import random

import numpy as np

from ninfer_amd_mi50_b200.cache import CacheManager, OutOfPages
from ninfer_amd_mi50_b200.parts.base import CacheSpec


def test_rows_follow_the_tables():
    rng = random.Random(5)
    specs = [CacheSpec("full", num_kv_heads=1, head_dim=16), CacheSpec("window", num_kv_heads=1, head_dim=16, window=20)]
    m = CacheManager(specs, [], page_size=8, num_pages=24, max_requests=4, max_context=120, allocate=False)
    for _ in range(600):
        open_now = list(m.requests)
        if len(open_now) < 3 and rng.random() < 0.3:
            m.open(rng.randrange(10 ** 9))
        elif open_now:
            r = rng.choice(open_now)
            if rng.random() < 0.1:
                m.close(r)
                continue
            try:
                m.reserve(r, min(120, m.length(r) + rng.choice([1, 1, 1, 9, 30])))
            except OutOfPages:
                m.truncate(r)
            else:
                if rng.random() < 0.8:
                    m.commit(r, m.requests[r].reserved)
                else:
                    m.truncate(r)
        for r in m.requests:
            for g in m.groups:
                row = m.block_row(g.index, r)
                assert row.dtype == np.int32 and row.tolist() == m.block_table(g.index, r)
        m.check()


def test_rows_of_a_slot_are_kept_from_request_to_request():
    """A request's rows are its slot's, made once: nothing of the request before is left in them, and a step's rows come out
    of them as its tables say."""
    specs = [CacheSpec("full", num_kv_heads=1, head_dim=16), CacheSpec("window", num_kv_heads=1, head_dim=16, window=20)]
    m = CacheManager(specs, [], page_size=8, num_pages=64, max_requests=3, max_context=120, allocate=False)
    m.open("a")
    m.reserve("a", 100)
    m.commit("a", 100)
    kept = m.requests["a"].rows
    slot = m.slot("a")
    m.close("a")
    assert m.open("b") == slot and all(np.shares_memory(x, y) for x, y in zip(kept, m.requests["b"].rows))
    m.open("c")
    for req, n in (("b", 9), ("c", 70)):
        m.reserve(req, n)
        m.commit(req, n)
    m.reserve("b", 60)
    m.truncate("b")
    for g in m.groups:
        want = [m.block_table(g.index, r) + [-1] * (12 - len(m.block_table(g.index, r))) for r in ("c", "b")]
        assert m.block_rows(g.index, [m.slot("c"), m.slot("b")], 12).tolist() == want
        assert m.block_rows(g.index, [slot], 15).tolist() == [m.block_table(g.index, "b") + [-1] * 13]
