"""Resident runs one after another without a wait between them: the exchange
slots that one launch leaves serve the next, whatever its length, in an engine,
in a batch and in a server whose rounds hold other requests each time."""
import numpy as np
import pytest

import golb200
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("x,y", [(96, 40), (544, 700), (2048, 600), (16352, 300)])
def test_engine(x, y):
    cells = oracle.random_ones_zeros(x, y, x + y)
    lengths = (1, 7, 8, 9, 16, 17, 24, 31, 3, 64)
    with golb200.GolB200(grid_dimensions=(x, y), state_bits_count=32, algorithm="resident") as e:
        for _ in range(2):
            e.set_and_format_input_data(cells)
            e.initialize_data_structures()
            for n in lengths:
                e.run(n)
            e.finalize_data_structures()
            assert np.array_equal(e.fetch_result(), oracle.life_cells(cells, sum(lengths)))


def test_batch():
    jobs = [(oracle.random_ones_zeros(32 * w, y, w), 1 + (5 * w + y) % 40)
            for w in (2, 5, 17, 64, 130) for y in (9, 200, 1201)]
    with golb200.GolBatch() as b:
        ids = [b.add(c, n) for c, n in jobs]
        for _ in range(3):
            b.run_resident()
            b.run_resident()
            b.sync()
            for i, (c, n) in zip(ids, jobs):
                assert np.array_equal(b.fetch(i), oracle.life_cells(c, n))


def test_server():
    jobs = [(oracle.random_ones_zeros(64 * (1 + i % 9), 30 + 61 * (i % 7), i), 5 + 13 * i)
            for i in range(30)]
    with golb200.GolServer(arena_bytes=64 << 20, quantum=16) as s:
        s.set_mode("resident")
        ids, done = {}, 0
        queue = list(range(len(jobs)))
        while done < len(jobs):
            for _ in range(min(3, len(queue))):     # other requests in every round
                i = queue.pop(0)
                ids[s.submit(*jobs[i])] = i
            s.step()
            for r in s.finished():
                c, n = jobs[ids[r]]
                assert np.array_equal(s.fetch(r), oracle.life_cells(c, n)), n
                done += 1


def test_captured_and_replayed():
    torch = pytest.importorskip("torch")
    x, y, n = 1056, 400, 13
    cells = oracle.random_ones_zeros(x, y, 5)
    s = torch.cuda.Stream()
    with golb200.GolB200(grid_dimensions=(x, y), state_bits_count=32, algorithm="resident",
                         stream=s.cuda_stream) as e:
        e.set_and_format_input_data(cells)
        e.initialize_data_structures()
        e.run(40)                      # (leaves the slots with later tags than a replay's)
        e.sync()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            e.run(n)
            e.run(n)
        with torch.cuda.stream(s):
            for _ in range(3):
                graph.replay()
        e.run(n)
        e.run(4 * n)
        with torch.cuda.stream(s):
            graph.replay()
        e.run(n)
        e.run(n)
        e.finalize_data_structures()
        # the capture itself ran nothing
        assert np.array_equal(e.fetch_result(), oracle.life_cells(cells, 40 + 6 * n + 5 * n + 2 * n + 2 * n))


@pytest.mark.parametrize("replays", [0, 2])
def test_first_run_captured(replays):
    """An engine whose first run is only captured, on memory that another
    engine's slots were in."""
    torch = pytest.importorskip("torch")
    x, y = 1056, 400
    cells = oracle.random_ones_zeros(x, y, 6)
    s = torch.cuda.Stream()

    def engine():
        return golb200.GolB200(grid_dimensions=(x, y), state_bits_count=32, algorithm="resident",
                               stream=s.cuda_stream)

    with engine() as e:
        e.set_and_format_input_data(cells)
        e.initialize_data_structures()
        e.run(200)
        e.finalize_data_structures()
    with engine() as e:
        e.set_and_format_input_data(cells)
        e.initialize_data_structures()
        e.sync()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            e.run(50)
            e.run(50)
        with torch.cuda.stream(s):
            for _ in range(replays):
                graph.replay()
        e.run(9)
        e.run(70)
        e.finalize_data_structures()
        assert np.array_equal(e.fetch_result(), oracle.life_cells(cells, 100 * replays + 79))
