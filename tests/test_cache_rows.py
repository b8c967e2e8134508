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
