"""The work that users of this library have it do, as measurable cases.

listed() names the fixed cases, draw(rng) gives one more of the same ranges,
prepare(case, seed) makes what a caller holds before the call (puzzle handle,
start state, buffers, engine), run(state) is one pass through the public entry
points and work(case) the bytes a pass cannot do without.

Kinds:
  solve      psb_bfs: a whole in-memory search (two-bit, three-bit, classic or
             frontier) of one puzzle from a start state, with the final bit
             arrays where the caller asks for them
  spill      psb_bfs with a spill callback: every depth's frontier as
             compressed segment streams in host memory
  expand     Puzzle.expand_device: one batch of parents, fixed slots
  encode     frontier_encode of one segment's bitmap
  decode     frontier_decode of one segment's stream
  batch      Engine: many small searches advanced together
  segmented  bfs_segmented: the out-of-core search with host-memory stores
"""
import ctypes
import math
import random

import numpy as np
import torch

import puzzlesearch_b200 as psb

MAX_DEPTHS = 512  # depths a caller makes room for (Hanoi with 17 disks has about 200)
FINAL_BYTES = 1_700_000_000  # final arrays above this stay on the GPU
BATCH_TYPES = [("sliding", 2, 3), ("sliding", 2, 4), ("sliding", 3, 3), ("sliding", 2, 5),
               ("pancake", 7, 0), ("pancake", 8, 0), ("pancake", 9, 0), ("pancake", 10, 0), ("pancake", 11, 0)]
# The last depth that a bounded search expands: the states beyond it are the
# hardest ones, which the final arrays name.
BOUND = {("sliding", 6): 18, ("sliding", 8): 30, ("sliding", 9): 28, ("sliding", 10): 48, ("sliding", 12): 48,
         ("pancake", 7): 7, ("pancake", 8): 8, ("pancake", 9): 9, ("pancake", 10): 10, ("pancake", 11): 12,
         ("pancake", 12): 13, ("pancake", 13): 14}
CLASSES = {"sliding": psb.SlidingTilePuzzleSimple, "sliding_opt": psb.SlidingTilePuzzleOptimized,
           "pancake": lambda a, b: psb.PancakeSimple(a), "pancake_opt": lambda a, b: psb.PancakeOptimized(a),
           "hanoi": lambda a, b: psb.FourPegHanoiSimple(a, bool(b)),
           "hanoi_opt": lambda a, b: psb.FourPegHanoiOptimized(a, bool(b))}


def listed():
    return [
        # A small board searched on its own: a request where latency and launches count.
        {"name": "solve_slide33", "kind": "solve", "puzzle": "sliding", "a": 3, "b": 3, "algo": "two_bit", "final": True,
         "max_depth": 28},
        # The 3x4 board, plain two-bit search over 12! indexes, all but its last few thin depths.
        {"name": "solve_slide34", "kind": "solve", "puzzle": "sliding", "a": 3, "b": 4, "algo": "two_bit", "final": True,
         "max_depth": 48},
        # Three-bit pancake search of ordinary size.
        {"name": "solve_pancake12", "kind": "solve", "puzzle": "pancake", "a": 12, "b": 0, "algo": "three_bit", "final": True,
         "max_depth": 0},
        # A large two-bit pancake search: the headline path one size down.
        {"name": "solve_pancake13", "kind": "solve", "puzzle": "pancake", "a": 13, "b": 0, "algo": "two_bit", "final": True,
         "max_depth": 14},
        # A large two-bit Hanoi search: many depths, most of them thin.
        {"name": "solve_hanoi17", "kind": "solve", "puzzle": "hanoi", "a": 17, "b": 0, "algo": "two_bit", "final": False,
         "max_depth": 0},
        # Frontier search (four operator bits per state) of the 3x4 board.
        {"name": "frontier_slide34", "kind": "solve", "puzzle": "sliding", "a": 3, "b": 4, "algo": "frontier", "final": True,
         "max_depth": 48},
        # A search whose every depth is written out as segment streams.
        {"name": "spill_hanoi13", "kind": "spill", "puzzle": "hanoi", "a": 13, "b": 0, "algo": "two_bit", "segment_bits": 0},
        # One full Expand buffer (Puzzle.MAX_INDEXES_BUFFER parents).
        {"name": "expand_pancake13", "kind": "expand", "puzzle": "pancake", "a": 13, "b": 0, "n": 2097152, "opbits": False},
        # A large segment of a thin depth: StreamVInt blocks.
        {"name": "encode_2e30", "kind": "encode", "bits": 1 << 30, "density": 0.01},
        # The way back: a stream ORed into a segment's bitmap.
        {"name": "decode_2e28", "kind": "decode", "bits": (1 << 28) - 37, "density": 0.02},
        # Many small searches at once (sliding 2x3 .. 2x5, pancake 7 .. 11).
        {"name": "batch_512", "kind": "batch", "instances": 512},
        # Out-of-core search of a small space in 16 segments.
        {"name": "segmented_hanoi10", "kind": "segmented", "puzzle": "hanoi", "a": 10, "b": 0, "segment_bits": 16,
         "max_depth": 0},
    ]


def _spread(rng, lo, hi):
    """A whole number of lo .. hi, evenly over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _bound(puzzle, a, b):
    kind = puzzle.split("_")[0]
    return BOUND.get((kind, a * b if kind == "sliding" else a), 0)


def draw(rng):
    kind = rng.choice(["solve"] * 5 + ["frontier", "spill", "expand", "expand", "encode", "decode", "batch", "segmented"])
    boards = [(2, 3), (3, 2), (2, 4), (4, 2), (3, 3), (2, 5), (5, 2), (2, 6), (3, 4), (4, 3), (6, 2)]
    if kind == "solve":
        algo = rng.choice(["two_bit", "two_bit", "three_bit", "classic"])
        puzzle = rng.choice(["sliding", "pancake", "hanoi", "pancake", "hanoi", "sliding_opt", "hanoi_opt", "pancake_opt"])
        if puzzle == "sliding":
            a, b = rng.choice(boards)
        elif puzzle == "sliding_opt":
            a, b = rng.choice([(2, 3), (2, 4), (3, 3), (2, 5), (3, 4), (4, 3)])
        elif puzzle == "pancake":
            a, b = rng.randint(7, 13 if algo == "two_bit" else 12), 0
        elif puzzle == "pancake_opt":
            a, b = rng.randint(8, 12), 0
        else:
            a, b = rng.randint(7, 17 if algo == "two_bit" else 16), rng.choice([0, 0, 1]) if algo == "two_bit" else 0
        return {"kind": "solve", "puzzle": puzzle, "a": a, "b": b, "algo": algo,
                "final": puzzle not in ("hanoi", "hanoi_opt") or a <= 14,
                "max_depth": 0 if algo == "three_bit" else _bound(puzzle, a, b),
                "direction": rng.choice(["auto", "auto", "top_down"]), "window_bits": rng.choice([0, rng.randint(12, 17)])}
    if kind == "frontier":
        if rng.random() < 0.5:
            a, b = rng.choice(boards)
            return {"kind": "solve", "puzzle": "sliding", "a": a, "b": b, "algo": "frontier", "final": True,
                    "max_depth": _bound("sliding", a, b), "window_bits": rng.choice([0, rng.randint(12, 16)])}
        return {"kind": "solve", "puzzle": "hanoi", "a": rng.randint(7, 15), "b": 0, "algo": "frontier", "final": False,
                "max_depth": 0, "window_bits": rng.choice([0, rng.randint(12, 16)])}
    if kind == "spill":
        puzzle, a, b = rng.choice([("sliding", 2, 4), ("sliding", 3, 3), ("sliding", 2, 5)]
                                  + [("pancake", n, 0) for n in (8, 9, 10, 11)]
                                  + [("hanoi", n, 0) for n in (8, 9, 10, 11, 12, 13)])
        algos = ["two_bit", "three_bit", "classic"] + ([] if puzzle == "pancake" else ["frontier"])
        return {"kind": "spill", "puzzle": puzzle, "a": a, "b": b, "algo": rng.choice(algos),
                "segment_bits": rng.choice([0, rng.randint(16, 28)])}
    if kind == "expand":
        puzzle, a, b = rng.choice([("pancake", rng.randint(7, 16), 0), ("sliding", 4, 4), ("sliding", 3, 5),
                                   ("sliding", 3, 4), ("hanoi", rng.randint(8, 31), 0), ("hanoi", rng.randint(8, 31), 1),
                                   ("pancake_opt", rng.randint(12, 16), 0), ("sliding_opt", 4, 4)])
        return {"kind": "expand", "puzzle": puzzle, "a": a, "b": b, "n": _spread(rng, 1, 2097152),
                "opbits": rng.random() < 0.5}
    if kind == "encode":
        return {"kind": "encode", "bits": _spread(rng, 1 << 12, 1 << 30), "density": 10 ** rng.uniform(-3, -0.35)}
    if kind == "decode":
        return {"kind": "decode", "bits": _spread(rng, 1 << 12, 1 << 28), "density": 10 ** rng.uniform(-3, -0.35)}
    if kind == "batch":
        return {"kind": "batch", "instances": _spread(rng, 8, 512)}
    return {"kind": "segmented", "puzzle": "hanoi", "a": rng.randint(7, 10), "b": 0, "segment_bits": rng.randint(12, 17),
            "max_depth": rng.choice([0, rng.randint(10, 40)])}


def _check(rc):
    if rc < 0:
        buf = ctypes.create_string_buffer(512)
        psb.lib().psb_last_error(buf, 512)
        raise psb.PsbError(rc, buf.value.decode(errors="replace"))


def _start(puzzle, case, rng):
    """A random start state: any permutation or peg assignment; for the packed
    boards a solvable permutation, with peg symmetry a state some moves in."""
    kind = case["puzzle"]
    if kind in ("sliding_opt", "pancake_opt"):
        n = case["a"] * case["b"] if kind == "sliding_opt" else case["a"]
        v = list(range(n))
        rng.shuffle(v)
        try:
            return puzzle.Parse(" ".join(map(str, v)))
        except psb.PsbError:  # the other parity class: swap two tiles
            i, j = [k for k in range(n) if v[k] != 0][:2]
            v[i], v[j] = v[j], v[i]
            return puzzle.Parse(" ".join(map(str, v)))
    if kind in ("hanoi", "hanoi_opt") and case["b"]:
        s = 0
        for _ in range(24 + rng.randrange(8)):
            s = rng.choice(puzzle.Expand([s])[0])
        return s
    return rng.randrange(puzzle.IndexesCount())


def _bitmap(bits, density, gen):
    """A segment's bitmap (int64 words on the GPU): states set at the density,
    in stretches of their own rates, as frontiers are."""
    words = (bits + 63) // 64
    out = torch.empty(words, dtype=torch.int64, device="cuda")
    step = 1 << 20
    shifts = (torch.arange(64, device="cuda", dtype=torch.int64))
    for w in range(0, words, step):
        n = min(step, words - w)
        rate = density * (0.5 + torch.rand((n + 1023) // 1024, device="cuda", generator=gen)).repeat_interleave(1024)[:n]
        hit = torch.rand(n, 64, device="cuda", generator=gen) < rate[:, None]
        out[w:w + n] = (hit.to(torch.int64) << shifts).sum(1)
    if bits % 64:
        out[-1] &= (1 << (bits % 64)) - 1
    return out


def prepare(case, seed):
    rng = random.Random(seed)
    kind = case["kind"]
    s = {"case": case}
    s["counts"] = (ctypes.c_uint64 * MAX_DEPTHS)()
    if kind in ("encode", "decode"):
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        s["bitmap"] = _bitmap(case["bits"], case["density"], gen)
        n = int(case["bits"] * min(1.0, 1.5 * case["density"]) * 2.5) + case["bits"] // 8 + 65536
        s["rows"] = int(case["bits"] * min(1.0, 1.5 * case["density"])) // 262144 + 2
        s["stream"] = torch.zeros(n, dtype=torch.uint8, device="cuda")
        if kind == "decode":
            torch.cuda.synchronize()
            used, s["blocks"], s["n_blocks"] = psb.frontier_encode(s["bitmap"].data_ptr(), 0, case["bits"],
                                                                   s["stream"].data_ptr(), n)
            s["stream"] = s["stream"][:used].clone()
            s["bitmap"].zero_()
        return s
    if kind == "batch":
        puzzles = {t: CLASSES[t[0]](t[1], t[2]) for t in BATCH_TYPES}
        s["items"] = []
        pool = 1 << 20
        for _ in range(case["instances"]):
            p = puzzles[BATCH_TYPES[rng.randrange(len(BATCH_TYPES))]]
            s["items"].append((p, rng.randrange(p.IndexesCount())))
            pool += psb.Engine.footprint(p)
        s["engine"] = psb.Engine(max_instances=case["instances"], max_depths=128, pool_bytes=pool)
        return s
    p = s["puzzle"] = CLASSES[case["puzzle"]](case["a"], case["b"])
    if kind == "expand":
        n, br = case["n"], p.BranchingFactor()
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        # states that name a permutation: a packed index has none at some offsets
        top = p.IndexesCount()
        s["parents"] = torch.randint(0, min(top, (1 << 63) - 1), (n,), device="cuda", generator=gen, dtype=torch.int64)
        if case["puzzle"] == "pancake_opt":
            s["parents"] = (s["parents"] >> 29 << 29) | ((s["parents"] & ((1 << 29) - 1)) % 479001600)
        s["opbits"] = (torch.randint(0, 1 << p.OperatorsCount(), (n,), device="cuda", generator=gen, dtype=torch.int32)
                       if case["opbits"] else None)
        s["children"] = torch.empty(n * br, dtype=torch.int64, device="cuda")
        s["ops"] = torch.empty(n * br, dtype=torch.int32, device="cuda")
        return s
    s["start"] = _start(p, case, rng)
    if kind == "segmented":
        return s
    o = s["opts"] = psb.BfsOpts()
    o.struct_size = ctypes.sizeof(psb.BfsOpts)
    o.device = -1
    o.max_depth = case.get("max_depth", 0)
    o.window_bits = case.get("window_bits", 0)
    o.direction = psb.DIRECTIONS[case.get("direction", "auto")]
    s["depths"] = ctypes.c_uint32()
    if kind == "spill":
        s["held"] = np.zeros(p.IndexesCount() * 5 // 2 + (4 << 20), dtype=np.uint8)
        o.segment_bits = case["segment_bits"]
    elif case["final"] and p.final_words(case["algo"]) * 8 <= FINAL_BYTES:
        s["final"] = torch.zeros(p.final_words(case["algo"]), dtype=torch.int64, pin_memory=True)
        o.final_words = ctypes.cast(s["final"].data_ptr(), psb.u64p)
        o.final_cap = s["final"].numel()
    return s


def _counts(c):
    """Per-depth counts as a caller keeps them: one row for every search."""
    out = np.zeros(MAX_DEPTHS, dtype=np.int64)
    out[:len(c)] = c
    return out


def _solve(s):
    _check(psb.lib().psb_bfs(s["puzzle"].handle, psb.ALGOS[s["case"]["algo"]], s["start"], ctypes.byref(s["opts"]),
                             s["counts"], MAX_DEPTHS, ctypes.byref(s["depths"]), None))
    return _counts(s["counts"][:s["depths"].value])


def run(state):
    s, case = state, state["case"]
    kind = case["kind"]
    if kind == "solve":
        counts = _solve(s)
        return {"counts": counts, "final": s["final"]} if "final" in s else {"counts": counts}
    if kind == "spill":
        held, table, used = s["held"], [], 0
        base = held.ctypes.data

        def spill(_user, depth, segment, data, n, states):  # the caller keeps every stream, back to back
            nonlocal used
            if used + n > held.size:
                return 1
            ctypes.memmove(base + used, data, n)
            table.append((depth, segment, used, n, states))
            used += n
            return 0

        s["opts"].spill = psb.SPILL_FN(spill)
        counts = _solve(s)
        rows = np.zeros((1 << 16, 5), dtype=np.int64)
        rows[:len(table)] = table
        return {"counts": counts, "table": rows, "streams": held}
    if kind == "expand":
        s["puzzle"].expand_device(s["parents"].data_ptr(), s["opbits"].data_ptr() if case["opbits"] else None, case["n"],
                                  s["children"].data_ptr(), s["ops"].data_ptr())
        return {"children": s["children"], "ops": s["ops"]}
    if kind == "encode":
        used, blocks, n = psb.frontier_encode(s["bitmap"].data_ptr(), 0, case["bits"], s["stream"].data_ptr(),
                                              s["stream"].numel())
        rows = np.zeros((s["rows"], 6), dtype=np.uint32)
        rows[:n] = np.frombuffer(blocks, dtype=np.uint32).reshape(-1, 6)[:n]
        return {"bytes": used, "stream": s["stream"], "blocks": rows}
    if kind == "decode":
        psb.frontier_decode(s["stream"].data_ptr(), s["blocks"], s["n_blocks"], s["bitmap"].data_ptr(), 0, case["bits"])
        return {"bitmap": s["bitmap"]}
    if kind == "batch":
        e = s["engine"]
        for i, (p, start) in enumerate(s["items"]):
            if not e.add(p, start, i):
                raise RuntimeError("the engine was made for all instances")
        done = {}
        while len(done) < len(s["items"]):
            e.step(8)
            done.update(e.poll())
        out = np.zeros((len(s["items"]), 128), dtype=np.int64)
        for i, c in done.items():
            out[i, :len(c)] = c
        return {"counts": out}
    r = psb.bfs_segmented(s["puzzle"], s["start"], segment_bits=case["segment_bits"], max_depth=case["max_depth"])
    return {"counts": _counts(r["counts"])}


def _states(name, a, b):
    """(index space, reached states, children per state) of a puzzle."""
    if name in ("sliding", "sliding_opt"):
        n = math.factorial(a * b)
        return (n if name == "sliding" else 16 * math.factorial(a * b - 1) // 2), n // 2, 3
    if name in ("pancake", "pancake_opt"):
        n = math.factorial(a)
        return (n if name == "pancake" or a < 12 else n // 479001600 << 29), n, a - 1
    return 4 ** a, 4 ** a // (6 if b else 1), 6


def work(case):
    """Bytes: every array cleared and written once, every reached state's
    children marked once per state (two bits read and written), results out.
    Operations: one per child generated."""
    kind = case["kind"]
    if kind == "encode" or kind == "decode":
        set_bits = case["bits"] * case["density"]
        out = min(set_bits * 1.3, case["bits"] / 8)  # about a byte and a quarter per state, or the bitmap
        return {"bytes": case["bits"] / 8 + out, "flops": 0}
    if kind == "expand":
        br = {"sliding": 4, "sliding_opt": 4, "hanoi": 6}.get(case["puzzle"], case["a"] - 1)
        return {"bytes": case["n"] * (8 + (4 if case["opbits"] else 0) + br * 12), "flops": case["n"] * br}
    if kind == "batch":
        every = [_states(*t) for t in BATCH_TYPES]
        mean = sum(n * 0.5 + r * 0.5 for n, r, _ in every) / len(every)
        kids = sum(r * c for _, r, c in every) / len(every)
        return {"bytes": case["instances"] * mean, "flops": case["instances"] * kids}
    n, reached, kids = _states(case["puzzle"], case["a"], case["b"])
    per = {"two_bit": 2, "three_bit": 3, "classic": 3, "frontier": 8}.get(case.get("algo"), 3)
    out = n * per / 8 if case.get("final") and n * per / 8 <= FINAL_BYTES else 0
    if kind in ("spill", "segmented"):
        out = reached * 1.25
    return {"bytes": n * per / 8 + reached * 0.5 + out, "flops": reached * kids}
