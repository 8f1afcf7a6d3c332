"""The perft engine's work as its users have it done, one case per kind of call.

Every case goes through the package's public entry points.  Positions are
seeded random legal playouts from the initial position (pg_random_playouts),
the inputs of the repository's own workloads and tests; a case names how many
plies they run, how many positions there are and at which depths they are
counted.  Results are whole numbers, the same on every run.
"""
import math
import time

import numpy as np
import torch

import perft_gpu_gb300 as pg

MOVES = 28.0  # mean number of legal moves of a playout position, for work()

_server = []  # the serving loop is one per process, as in a serving program


def listed():
    return [
        # one shallow count, as an interactive tool or a move-generator check asks for: launches and latency
        {"name": "one_depth3", "kind": "one", "plies": 12, "min_moves": 1, "depth": 3},
        # one position at an ordinary depth
        {"name": "one_depth5", "kind": "one", "plies": 24, "min_moves": 20, "depth": 5},
        # one deep count of a middlegame position with many moves (the single-position workload)
        {"name": "one_depth7", "kind": "one", "plies": 30, "min_moves": 35, "depth": 7},
        # per-root-move counts, as an engine author compares them move by move
        {"name": "divide_depth6", "kind": "divide", "plies": 20, "min_moves": 20, "depth": 6},
        # thousands of uneven positions in one call from host arrays: the headline workload
        {"name": "batch_4096_depth3to6", "kind": "batch", "n": 4096, "plies": 60, "lo": 3, "hi": 6, "mode": "plain"},
        # an odd-sized batch already resident in device memory
        {"name": "device_777_depth2to5", "kind": "device", "n": 777, "plies": 60, "lo": 2, "hi": 5},
        # a batch as one persistent launch replayed from its graph
        {"name": "persist_257_depth3to6", "kind": "batch", "n": 257, "plies": 60, "lo": 3, "hi": 6, "mode": "persist_graph"},
        # very many shallow positions (labelling a position set)
        {"name": "shallow_100003_depth0to3", "kind": "batch", "n": 100003, "plies": 60, "lo": 0, "hi": 3, "mode": "plain"},
        # one-ply counts of a million boards
        {"name": "moves_1000003", "kind": "moves", "n": 1000003, "plies": 60},
        # the entry point for callers that cannot allocate device memory
        {"name": "noalloc_20001_depth0to3", "kind": "noalloc", "n": 20001, "plies": 60},
        # positions counted with the duplicate pass inside each level (no tables kept)
        {"name": "dedup_64_depth6", "kind": "batch", "n": 64, "plies": 60, "lo": 6, "hi": 6, "mode": "dedup"},
        # a mixed set of requests served by the continuous-batching loop
        {"name": "served_64_depth3to6", "kind": "served", "n": 64, "plies": 60, "lo": 3, "hi": 6},
    ]


def _spread(rng, lo, hi):
    """A whole number in lo..hi, even over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["one", "one", "divide", "batch", "batch", "batch", "device", "shallow", "moves", "noalloc",
                       "dedup", "served"])
    plies = rng.randint(2, 60)
    if kind in ("one", "divide"):
        return {"kind": kind, "plies": plies, "min_moves": rng.randint(1, 35),
                "depth": rng.randint(3, 7 if kind == "one" else 6)}
    if kind == "moves":
        return {"kind": kind, "n": _spread(rng, 1000, 1000003), "plies": plies}
    if kind == "noalloc":
        return {"kind": kind, "n": _spread(rng, 1000, 20001), "plies": plies}
    if kind == "shallow":
        return {"kind": "batch", "n": _spread(rng, 5000, 100003), "plies": plies, "lo": 0, "hi": rng.randint(1, 3),
                "mode": "plain"}
    hi = rng.randint(3, 6)
    lo = rng.randint(2, hi)
    if kind == "dedup":
        return {"kind": "batch", "n": _spread(rng, 4, 200), "plies": plies, "lo": lo, "hi": hi, "mode": "dedup"}
    if kind == "served":
        return {"kind": kind, "n": _spread(rng, 8, 96), "plies": plies, "lo": lo, "hi": hi}
    # a quarter of the headline's positions: all of them may be at depth 6 here
    n = _spread(rng, 3, 1000)
    if kind == "device":
        return {"kind": kind, "n": n, "plies": plies, "lo": lo, "hi": hi}
    return {"kind": "batch", "n": n, "plies": plies, "lo": lo, "hi": hi,
            "mode": rng.choice(["plain", "plain", "persist", "persist_graph"])}


def prepare(case, seed):
    pg.init()  # a no-op once the engine is up
    kind = case["kind"]
    s = {"kind": kind, "mode": case.get("mode", "plain")}
    if kind in ("one", "divide"):
        boards = pg.random_playouts(seed, 1, case["plies"], case["plies"], case["min_moves"])
        s["pos"] = pg.board_of(boards[0])
        s["depth"] = case["depth"]
        return s
    if kind == "moves":
        s["boards"] = pg.random_playouts(seed, case["n"], 0, case["plies"], 1)
        return s
    lo, hi = (0, 3) if kind == "noalloc" else (case["lo"], case["hi"])
    s["boards"], s["depths"] = pg.random_playouts(seed, case["n"], 0, case["plies"], 1, lo, hi, with_depths=True)
    if kind in ("device", "noalloc"):
        s["d_boards"] = torch.from_numpy(s["boards"].view(np.uint8).copy()).cuda()
        s["d_depths"] = torch.from_numpy(s["depths"].copy()).cuda()
        s["d_out"] = torch.zeros(case["n"], dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
    if kind == "served":
        if not _server:
            _server.append(pg.Server())
        s["requests"] = [(pg.board_of(b), int(d)) for b, d in zip(s["boards"], s["depths"])]
    return s


def run(s):
    kind = s["kind"]
    if kind == "one":
        return pg.perft(s["pos"], s["depth"])
    if kind == "divide":
        found = pg.perft_divide(s["pos"], s["depth"])
        table = np.full((256, 2), -1, dtype=np.int64)  # (move, count), one row a legal root move
        table[:len(found)] = found
        return table
    if kind == "moves":
        return pg.count_moves_batch(s["boards"]).astype(np.int64)
    if kind == "device":
        pg.perft_batch_device(s["d_boards"].data_ptr(), s["d_depths"].data_ptr(), len(s["depths"]),
                              s["d_out"].data_ptr())
        return s["d_out"]
    if kind == "noalloc":
        status = pg.load_library().pg_perft_batch_noalloc(s["d_boards"].data_ptr(), s["d_depths"].data_ptr(),
                                                          len(s["depths"]), s["d_out"].data_ptr(), None)
        if status != pg.PG_OK:
            raise pg.PerftError(status, "pg_perft_batch_noalloc")
        return s["d_out"]
    if kind == "served":
        server = _server[0]
        ids = [server.submit(b, d) for b, d in s["requests"]]
        counts = {}
        while len(counts) < len(ids):
            for rid in ids:
                if rid not in counts:
                    r, _ = server.poll(rid)
                    if r is not None:
                        counts[rid] = r
            if len(counts) < len(ids):
                time.sleep(0.0002)
        return np.array([counts[rid] for rid in ids], dtype=np.int64)
    options = {"plain": {}, "persist": {"persistent": True}, "persist_graph": {"persistent": True, "graph": True},
               "dedup": {"use_tt": "dedup"}}[s["mode"]]
    return pg.perft_batch(s["boards"], s["depths"], **options).astype(np.int64)


def work(case):
    """Bytes: each board and depth read once, each count written once.  Operations: one whole-number operation
    for each counted leaf, with MOVES legal moves a position."""
    kind = case["kind"]
    if kind in ("one", "divide"):
        return {"bytes": 48 + 8, "flops": max(MOVES, case["min_moves"]) ** case["depth"]}
    n = case["n"]
    if kind == "moves":
        return {"bytes": n * (48 + 4), "flops": n * MOVES}
    lo, hi = (0, 3) if kind == "noalloc" else (case["lo"], case["hi"])
    leaves = sum(MOVES ** d for d in range(lo, hi + 1)) / (hi - lo + 1)
    return {"bytes": n * (48 + 1 + 8), "flops": n * leaves}


def exact(case, seed):
    """No output is a floating-point number: every count is a whole number and has one right value."""
    return None
