"""The batch's register-block items against the oracle: word counts around a
segment's and a slice's limits, row counts around a band's, generations around
both depths, with and without change tracking, and a server's requests of the
same shapes."""
import numpy as np
import pytest

import golb200
import oracle

pytestmark = pytest.mark.gpu

WORDS = (1, 2, 14, 15, 16, 29, 30, 31, 32, 59, 60, 61, 157)
ROWS = (1, 7, 8, 9, 31, 100, 257)


def work():
    out = []
    for i, w in enumerate(WORDS):
        for j, y in enumerate(ROWS):
            gens = (1, 3, 4, 7, 8, 9, 16, 33)[(i + 2 * j) % 8]
            cells = oracle.random_ones_zeros(32 * w, y, 31 * w + y)
            cells[:, 16 * w:] *= (i + j) % 2          # half of some grids dead
            out.append((cells, gens + 40 * (j % 3)))
    return out


@pytest.mark.parametrize("tracking", ["on", "off"])
def test_batch(tracking):
    jobs = work()
    with golb200.GolBatch() as b:
        ids = [b.add(c, n) for c, n in jobs]
        for gid in ids:
            b.set_tracking(gid, tracking)
        for _ in range(2):
            b.run()
            b.sync()
            for gid, (c, n) in zip(ids, jobs):
                assert np.array_equal(b.fetch(gid), oracle.life_cells(c, n)), (c.shape, n)


@pytest.mark.parametrize("k,band", [(4, 4), (4, 5), (4, 56), (3, 16), (1, 62), (2, 0)])
def test_forced_depth_and_band(k, band):
    jobs = work()[::3]
    with golb200.GolBatch() as b:
        ids = [b.add(c, n) for c, n in jobs]
        for gid in ids:
            b.set_plan(gid, 0, k, band)
        b.run()
        b.sync()
        for gid, (c, n) in zip(ids, jobs):
            assert np.array_equal(b.fetch(gid), oracle.life_cells(c, n)), (c.shape, n)


@pytest.mark.parametrize("mode", ["passes", "resident"])
def test_server(mode):
    jobs = work()[::2]
    with golb200.GolServer(arena_bytes=64 << 20, quantum=16) as s:
        s.set_mode(mode)
        ids = {s.submit(c, n): i for i, (c, n) in enumerate(jobs)}
        left = set(ids)
        while left:
            s.step()
            for rid in s.finished():
                c, n = jobs[ids[rid]]
                assert np.array_equal(s.fetch(rid), oracle.life_cells(c, n)), (c.shape, n)
                left.discard(rid)
