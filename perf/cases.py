"""The work that performance is measured on: what a user of the engine has it
do, through the public Python front end, over the ranges that are in use.

  listed()             the cases, smallest to largest of each kind
  draw(rng)            one more case of the same ranges
  prepare(case, seed)  what a user's program holds before the call
  run(state)           one pass through the public entry points
  work(case)           bytes and integer operations of one pass
  exact(case, seed)    the same result by plain torch bit operations

Sizes are those of the repository's benchmark configurations, smoke run and
tests; the ragged ones are generic. Kinds:
  contract  the Algorithm contract on host cells (set input, initialise, run,
            finalise, fetch), the instance reused round after round
  device    a grid that stays on the GPU, advanced by `gens` per call
  words     the contract on packed host words (change tracking: every pass
            starts from the same sparse input)
  pass      one stateless pass of k generations on caller-owned buffers
  batch     uneven grids in one launch, every result fetched as cells
  serve     a burst of requests through the continuous-batching server
  cells     device pack and unpack between byte cells and row words
  layout    device conversion between the rows, column and tile layouts
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "stencil-optimalizations_b200"))
import golb200  # noqa: E402

# Word operations of one generation of 64 cells, the full adder of the
# reference's 64-bit kernels.
OPS_PER_CELL = 33 / 64


def listed():
    return [
        # The smallest calls: a launch or two of work, latency counts.
        {"name": "contract 256x256", "kind": "contract", "x": 256, "y": 256, "gens": 100,
         "cells": "u8"},
        # The plain configuration: 2048 x 2048 byte cells, 128 generations.
        {"name": "contract 2048x2048", "kind": "contract", "x": 2048, "y": 2048, "gens": 128,
         "cells": "u8"},
        # The dense configuration, kept on the GPU: 16384 x 16384, 4096 generations.
        {"name": "dense 16384x16384", "kind": "device", "alg": "auto", "x": 16384, "y": 16384,
         "bits": 64, "gens": 4096, "k": 0},
        # Its 32-bit-word variant, in the shared-memory-resident mode.
        {"name": "resident 8192x8192", "kind": "device", "alg": "resident", "x": 8192, "y": 8192,
         "bits": 32, "gens": 4096, "k": 0},
        # An ordinary grid of ragged size: an odd number of words per row.
        {"name": "dense 5024x3001", "kind": "device", "alg": "auto", "x": 5024, "y": 3001,
         "bits": 32, "gens": 1000, "k": 0},
        # One generation per pass on a grid larger than L2: bound by HBM.
        {"name": "pass k=1 32768x32768", "kind": "pass", "x": 32768, "y": 32768, "k": 1},
        # One deep pass on a ragged grid.
        {"name": "pass k=8 10240x6001", "kind": "pass", "x": 10240, "y": 6001, "k": 8},
        # The sparse, settling configuration: change tracking, 20000 generations.
        {"name": "sparse 16384x16384", "kind": "words", "x": 16384, "y": 16384, "gens": 20000,
         "fraction": 0.01, "density": 0.35},
        # Uneven grids (sides 256..4096, 64..4096 generations) resident in one launch.
        {"name": "batch of 48", "kind": "batch", "mode": "resident", "grids": 48, "min_side": 256,
         "max_side": 4096, "max_gens": 4096, "draw": 42},
        # Requests (sides 128..8192, 16..8192 generations) served in the default mode.
        {"name": "serve 24 requests", "kind": "serve", "mode": "passes", "requests": 24,
         "max_side": 8192, "max_gens": 8192, "draw": 42},
        # Byte cells to words and back on the device.
        {"name": "cells 16384x16384", "kind": "cells", "x": 16384, "y": 16384},
        # A grid taken in from columns and given out as tiles.
        {"name": "layout 16384x16384", "kind": "layout", "x": 16384, "y": 16384, "bits": 64},
    ]


def _log(rng, lo, hi, multiple=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(multiple, int(round(v / multiple)) * multiple)


def draw(rng):
    kind = rng.choice(["contract", "device", "device", "device", "resident", "pass", "pass",
                       "words", "batch", "serve", "cells", "layout"])
    if kind == "contract":
        return {"kind": kind, "x": _log(rng, 128, 4096, 64), "y": _log(rng, 64, 4096),
                "gens": _log(rng, 16, 2048), "cells": rng.choice(["u8", "u8", "i32"])}
    if kind == "device":
        return {"kind": kind, "alg": "auto", "x": _log(rng, 256, 16384, 32),
                "y": _log(rng, 64, 16384), "bits": 32, "gens": _log(rng, 64, 4096),
                "k": rng.choice([0, 0, 0, 1, 2, 8])}
    if kind == "resident":
        x = _log(rng, 512, 12288, 32)
        return {"kind": "device", "alg": "resident", "x": x,
                "y": _log(rng, 256, min(8192, (1 << 26) // x)), "bits": 32,
                "gens": _log(rng, 64, 4096), "k": 0}
    if kind == "pass":
        return {"kind": kind, "x": _log(rng, 1024, 32768, 32), "y": _log(rng, 1024, 32768),
                "k": rng.choice([1, 1, 2, 4, 6, 8, 16])}
    if kind == "words":
        return {"kind": kind, "x": _log(rng, 4096, 16384, 64), "y": _log(rng, 4096, 16384, 64),
                "gens": _log(rng, 1000, 20000), "fraction": rng.choice([0.002, 0.01, 0.05]),
                "density": 0.35}
    if kind == "batch":
        return {"kind": kind, "mode": rng.choice(["resident", "passes"]),
                "grids": rng.randint(16, 64), "min_side": 256, "max_side": 4096, "max_gens": 4096,
                "draw": rng.randrange(1 << 30)}
    if kind == "serve":
        return {"kind": kind, "mode": rng.choice(["passes", "resident"]),
                "requests": rng.randint(8, 32), "max_side": 8192, "max_gens": 8192,
                "draw": rng.randrange(1 << 30)}
    if kind == "cells":
        return {"kind": kind, "x": _log(rng, 512, 16384, 32), "y": _log(rng, 512, 16384)}
    return {"kind": kind, "x": _log(rng, 512, 16384, 64), "y": _log(rng, 512, 16384, 64),
            "bits": rng.choice([16, 32, 64])}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _random_words(x, y, seed):
    """Bernoulli(0.5) cells as row words, int32 [y, x / 32] on the GPU."""
    return torch.randint(-(1 << 31), 1 << 31, (y, x // 32), dtype=torch.int32, device="cuda",
                         generator=_gen(seed))


def _random_cells(x, y, seed, density=0.5):
    """Bernoulli cells, uint8 [y, x] on the GPU."""
    return (torch.rand((y, x), device="cuda", generator=_gen(seed)) < density).to(torch.uint8)


def _pack(cells):
    y, x = cells.shape
    bit = torch.ones(32, dtype=torch.int64, device=cells.device) << torch.arange(
        32, device=cells.device)
    out = torch.empty((y, x // 32), dtype=torch.int32, device=cells.device)
    step = max(1, (1 << 26) // max(x, 1))
    for r in range(0, y, step):
        v = ((cells[r:r + step].reshape(-1, x // 32, 32) != 0).to(torch.int64) * bit).sum(-1)
        out[r:r + step] = v.to(torch.int32)
    return out


def _sparse_words(case, seed):
    """All dead but for a share of the 64 x 64 slots, filled with Bernoulli cells."""
    x, y = case["x"], case["y"]
    g = _gen(seed)
    slots = (x // 64) * (y // 64)
    n = max(1, int(slots * case["fraction"]))
    at = torch.randperm(slots, device="cuda", generator=g)[:n]
    patch = (torch.rand((n, 64, 64), device="cuda", generator=g) < case["density"]).to(torch.uint8)
    grid = torch.zeros((y // 64, x // 64, 64, 2), dtype=torch.int32, device="cuda")
    words = _pack(patch.reshape(n * 64, 64)).reshape(n, 64, 2)
    grid[at // (x // 64), at % (x // 64)] = words
    return grid.permute(0, 2, 1, 3).reshape(y, x // 32).contiguous()


def _uneven(case, n, min_side, min_gens, densities, seed):
    """Sizes and generation counts fixed by the case, densities and cells by the seed."""
    r, d, out = random.Random(case["draw"]), random.Random(seed), []
    for i in range(n):
        out.append({"x": min(case["max_side"], _log(r, min_side, case["max_side"], 64)),
                    "y": min(case["max_side"], _log(r, min_side, case["max_side"], 64)),
                    "gens": _log(r, min_gens, case["max_gens"]),
                    "density": d.uniform(*densities), "seed": d.randrange(1 << 30)})
    return out


def _grids(case, seed):
    return _uneven(case, case["grids"], case["min_side"], 64, (0.2, 0.5), seed)


def _requests(case, seed):
    return _uneven(case, case["requests"], 128, 16, (0.1, 0.5), seed)


_stream = None


def _program_stream():
    """The one stream a program that advances its grids one after another works on."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


class _View:
    """An engine's device grid as an array, kept alive by the engine."""

    def __init__(self, engine, ptr, shape):
        self.engine = engine
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<i4", "data": (ptr, False),
                                         "version": 3, "strides": None}


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "contract":
        x, y = case["x"], case["y"]
        cells = _random_cells(x, y, seed).cpu().numpy()
        s["cells"] = cells if case["cells"] == "u8" else cells.astype(np.int32)
        s["out"] = np.zeros_like(s["cells"])
        s["engine"] = golb200.GolB200(grid_dimensions=(x, y), iterations=case["gens"])
    elif kind == "device":
        x, y = case["x"], case["y"]
        e = golb200.GolB200(grid_dimensions=(x, y), state_bits_count=case["bits"],
                            algorithm=case["alg"], temporal_steps=case["k"],
                            stream=_program_stream().cuda_stream)
        e.set_input_words(_random_words(x, y, seed).cpu().numpy(), case["bits"])
        e.initialize_data_structures()
        s["engine"] = e
    elif kind == "words":
        s["words"] = _sparse_words(case, seed).cpu().numpy()
        s["engine"] = golb200.GolB200(grid_dimensions=(case["x"], case["y"]), algorithm="local",
                                      iterations=case["gens"])
    elif kind == "pass":
        s["src"] = _random_words(case["x"], case["y"], seed)
        s["dst"] = torch.empty_like(s["src"])
    elif kind == "batch":
        b = golb200.GolBatch()
        s["ids"] = [b.add(_random_cells(g["x"], g["y"], g["seed"], g["density"]).cpu().numpy(),
                          g["gens"]) for g in _grids(case, seed)]
        b.upload()
        s["batch"] = b
    elif kind == "serve":
        srv = golb200.GolServer(arena_bytes=2 << 30)
        srv.set_mode(case["mode"])
        s["server"] = srv
        s["requests"] = _requests(case, seed)
    elif kind == "cells":
        s["cells"] = _random_cells(case["x"], case["y"], seed)
        s["words"] = torch.empty((case["y"], case["x"] // 32), dtype=torch.int32, device="cuda")
        s["back"] = torch.empty_like(s["cells"])
    else:
        # column words of any value are a grid; so are rows and tiles of it
        s["columns"] = _random_words(case["x"], case["y"], seed)
        s["rows"] = torch.empty_like(s["columns"])
        s["tiles"] = torch.empty_like(s["columns"])
    return s


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "contract":
        e = s["engine"]
        e.set_and_format_input_data(s["cells"])
        e.initialize_data_structures()
        e.run(c["gens"])
        e.finalize_data_structures()
        return e.fetch_result(s["out"])
    if kind == "device":
        e = s["engine"]
        e.run(c["gens"])
        return torch.as_tensor(_View(e, e.device_grid_ptr(), (c["y"], c["x"] // 32)),
                               device="cuda")
    if kind == "words":
        e = s["engine"]
        e.set_input_words(s["words"], 32)
        e.initialize_data_structures()
        e.run(c["gens"])
        e.finalize_data_structures()
        return e.fetch_words(32).view(np.int32)
    if kind == "pass":
        golb200.rows_pass(s["src"].data_ptr(), s["dst"].data_ptr(), c["x"], c["y"], c["k"],
                          stream=torch.cuda.current_stream().cuda_stream)
        return s["dst"]
    if kind == "batch":
        b = s["batch"]
        if c["mode"] == "resident":
            b.run_resident()
        else:
            b.run()
        b.sync()
        return [b.fetch(i) for i in s["ids"]]
    if kind == "serve":
        srv = s["server"]
        ids = [srv.submit_random(r["x"], r["y"], r["gens"], r["seed"], r["density"])
               for r in s["requests"]]
        out = {}
        while len(out) < len(ids):
            srv.step()
            for i in srv.finished():
                out[i] = srv.fetch_words(i).view(np.int32)
        return [out[i] for i in ids]
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "cells":
        golb200.pack_cells_device(s["cells"].data_ptr(), s["words"].data_ptr(), c["x"], c["y"],
                                  stream)
        golb200.unpack_cells_device(s["words"].data_ptr(), s["back"].data_ptr(), c["x"], c["y"],
                                    stream)
        return {"words": s["words"], "cells": s["back"]}
    golb200.layout_to_rows_device(s["columns"].data_ptr(), s["rows"].data_ptr(), c["x"], c["y"],
                                  "columns", c["bits"], stream)
    golb200.rows_to_layout_device(s["rows"].data_ptr(), s["tiles"].data_ptr(), c["x"], c["y"],
                                  "tiles", c["bits"], stream)
    return {"rows": s["rows"], "tiles": s["tiles"]}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def work(case):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        grids = _grids(case, 0) if kind == "batch" else _requests(case, 0)
        cells = sum(g["x"] * g["y"] for g in grids)
        ops = sum(g["x"] * g["y"] * g["gens"] for g in grids) * OPS_PER_CELL
        # batch: words in, cells out; serve: made on the device, words out
        return {"bytes": cells / 8 + cells if kind == "batch" else cells / 8, "flops": ops}
    cells = case["x"] * case["y"]
    if kind == "contract":
        return {"bytes": 2 * cells * (1 if case["cells"] == "u8" else 4),
                "flops": cells * case["gens"] * OPS_PER_CELL}
    if kind == "device":
        return {"bytes": cells / 4, "flops": cells * case["gens"] * OPS_PER_CELL}
    if kind == "words":   # the filled slots alone
        return {"bytes": cells / 4,
                "flops": cells * case["fraction"] * case["gens"] * OPS_PER_CELL}
    if kind == "pass":
        return {"bytes": cells / 4, "flops": cells * case["k"] * OPS_PER_CELL}
    if kind == "cells":   # cells in, words out, words in, cells out
        return {"bytes": 2 * (cells + cells / 8), "flops": 0}
    return {"bytes": 4 * cells / 8, "flops": 0}   # two conversions, in and out


# ---------------------------------------------------------------------------
# the same by plain torch
# ---------------------------------------------------------------------------

def _life(words, gens):
    """`gens` generations of row words (int64 rows of 32 cells, values below 2^32)."""
    w = words.to(torch.int64) & 0xFFFFFFFF
    y, n = w.shape
    pad = torch.zeros((y + 2, n + 2), dtype=torch.int64, device=w.device)
    cur, nxt = pad, pad.clone()
    cur[1:-1, 1:-1] = w
    for _ in range(gens):
        c = cur[:, 1:-1]
        left = ((c << 1) & 0xFFFFFFFF) | (cur[:, :-2] >> 31)
        right = (c >> 1) | ((cur[:, 2:] & 1) << 31)
        x = left ^ right
        h0, h1 = x ^ c, (left & right) | (x & c)          # cells in three of the row
        a0, b0, p0 = h0[:-2], h0[1:-1], h0[2:]
        a1, b1, p1 = h1[:-2], h1[1:-1], h1[2:]
        t = a0 ^ b0
        t0, c0 = t ^ p0, (a0 & b0) | (t & p0)
        u = a1 ^ b1
        u0, u1 = u ^ p1, (a1 & b1) | (u & p1)
        three = t0 & (c0 ^ u0) & ~u1                      # 3 of the 3 x 3 block alive
        four = ~t0 & ((u1 & ~(c0 | u0)) | (c0 & u0 & ~u1))
        nxt[1:-1, 1:-1] = three | (four & c[1:-1])
        cur, nxt = nxt, cur
    out = cur[1:-1, 1:-1]
    return torch.where(out >= 1 << 31, out - (1 << 32), out).to(torch.int32)


def _cells(words):
    bit = torch.arange(32, device=words.device)
    y, n = words.shape
    out = torch.empty((y, n * 32), dtype=torch.uint8, device=words.device)
    step = max(1, (1 << 26) // max(n * 32, 1))
    for r in range(0, y, step):
        v = words[r:r + step].to(torch.int64)
        out[r:r + step] = ((v[:, :, None] >> bit) & 1).to(torch.uint8).reshape(-1, n * 32)
    return out


def _slow(grids):
    """Whether the torch form would take too long (about 40 operations of 8
    bytes a word a generation, at least 4 us each)."""
    return sum(g["gens"] * 40 * max(5e-6, g["x"] * g["y"] / 32 * 24 / 4e12)
               for g in grids) > 15


def _hash_words(r):
    """The cells a request of gol_serve_submit_random stands for."""
    n = r["x"] * r["y"]
    cells = np.empty(n, np.uint8)
    limit = np.uint64(int(r["density"] * 9007199254740992.0))
    for a in range(0, n, 1 << 22):
        i = np.arange(a, min(n, a + (1 << 22)), dtype=np.uint64)
        with np.errstate(over="ignore"):
            z = np.uint64(r["seed"]) + (i + np.uint64(1)) * np.uint64(0x9E3779B97F4A7C15)
            z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
            z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
            z ^= z >> np.uint64(31)
        cells[a:a + i.size] = (z >> np.uint64(11)) < limit
    return _pack(torch.from_numpy(cells.reshape(r["y"], r["x"])).cuda())


def _tiles(cells, bits):
    y, x = cells.shape
    xb, yb = golb200.layout_block("tiles", bits)
    v = cells.reshape(y // yb, yb, x // xb, xb).permute(0, 2, 1, 3).reshape(-1, bits)
    v = v.flip(1)                                         # top-left cell in the highest bit
    return _pack(v.reshape(1, -1) if bits < 32 else v).reshape(y, x // 32)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        grids = _grids(case, seed) if kind == "batch" else _requests(case, seed)
        if _slow(grids):
            return None
        if kind == "batch":
            return [_cells(_life(_pack(_random_cells(g["x"], g["y"], g["seed"], g["density"])),
                                 g["gens"])).cpu().numpy() for g in grids]
        return [_life(_hash_words(r), r["gens"]).cpu().numpy() for r in grids]
    x, y = case["x"], case["y"]
    if kind in ("contract", "device", "words") and _slow([case]):
        return None
    if kind == "contract":
        cells = _cells(_life(_pack(_random_cells(x, y, seed)), case["gens"]))
        return cells.cpu().numpy().astype(np.uint8 if case["cells"] == "u8" else np.int32)
    if kind == "device":
        return _life(_random_words(x, y, seed), case["gens"])
    if kind == "words":
        return _life(_sparse_words(case, seed), case["gens"]).cpu().numpy()
    if kind == "pass":
        return _life(_random_words(x, y, seed), case["k"])
    if kind == "cells":
        cells = _random_cells(x, y, seed)
        return {"words": _pack(cells), "cells": cells}
    bits = case["bits"]
    cols = _random_words(x, y, seed)
    # word (wy, cx) holds cells (cx, wy * bits ..), lowest bit on top
    cells = _cells(cols.reshape(1, -1)).reshape(y // bits, x, bits).permute(0, 2, 1)
    cells = cells.reshape(y, x).contiguous()
    return {"rows": _pack(cells), "tiles": _tiles(cells, bits)}
