"""Performance cases of the frontier-DP engine: what a program asks of it.

Kinds of work, each through the Python binding of the C ABI:

  residues   Engine.residues: k residues of the n x n grid's path count, `lanes`
             of them per pass (lanes = 1 is the plain one-modulus form)
  multi      Engine.residues_multi: several grid sizes in one call
  serve      Engine.submit / wait: a burst of requests to a running server
  window     Engine.apply_cells: cells p_hi..p_lo of one row on the caller's state
  transfer   TransferMap.apply: one cell pair as a CSR built beforehand
  factor     FactorMap.apply: every conjugate occupancy group of one shape
  reverse2   Engine.reverse2_apply: two cells pulled at once, no CSR

Moduli are primes just below 2^32, states are uniform residues; both follow
from the seed.  Every result is an integer, so outputs compare exactly.
"""
import functools
import itertools
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oneesan-gpu_b200"))
import fdp  # noqa: E402

SERVER_BUDGET = 6 * 10**9
MAX_GROUPS = 32


def listed():
    return [
        # The published n = 9 solve with its two moduli: a first run, a smoke
        # check, the smallest requests; launches and host latency.
        {"name": "solve n9 x2", "kind": "residues", "n": 9, "k": 2, "lanes": 2},
        # A mid-size solve with four moduli, as a serving request asks it.
        {"name": "solve n16 x4", "kind": "residues", "n": 16, "k": 4, "lanes": 4},
        # The plain method: n = 18, one modulus.
        {"name": "solve n18 plain", "kind": "residues", "n": 18, "k": 1, "lanes": 1},
        # n = 20 with four moduli in one batched pass.
        {"name": "solve n20 x4", "kind": "residues", "n": 20, "k": 4, "lanes": 4},
        # An exact count's batch: 14 CRT residues in one pass (two lane spans).
        {"name": "solve n20 x14", "kind": "residues", "n": 20, "k": 14, "lanes": 14},
        # Several grid sizes in one graph, an odd lane count.
        {"name": "multi n11..17 x3", "kind": "multi", "n_lo": 11, "n_hi": 17, "k": 3},
        # A burst of the served form's smaller requests, n 12..16, k 1..8.
        {"name": "serve 16 requests", "kind": "serve", "n_lo": 12, "n_hi": 16, "requests": 16},
        # The operator window the GROUPBATCH operator test forces, 16 lanes.
        {"name": "window w14 x16", "kind": "window", "width": 14, "lanes": 16, "p_hi": 13, "p_lo": 6},
        # A whole row at n = 23, where ranks need 64 bits: the largest state.
        {"name": "row w24 x1", "kind": "window", "width": 24, "lanes": 1, "p_hi": 23, "p_lo": 1},
        # Operator variants: the paired transfer map, the factorized map over
        # all conjugate groups of one shape, the two-cell pull.
        {"name": "transfer w16 x4", "kind": "transfer", "width": 16, "p": 8, "lanes": 4},
        {"name": "factor w17 8:4", "kind": "factor", "width": 17, "p": 10, "fixed": 8, "occupied": 4},
        {"name": "reverse2 w15 x8", "kind": "reverse2", "width": 15, "p": 8, "lanes": 8},
    ]


def draw(rng):
    kind = rng.choice(["residues"] * 5 + ["multi", "serve", "window", "window", "transfer", "factor", "reverse2"])
    if kind == "residues":
        n = rng.randint(8, 20)  # the state count grows about 2.8 x per n
        k = rng.randint(1, 4 if n == 20 else 8 if n == 19 else 16)
        return {"kind": kind, "n": n, "k": k, "lanes": rng.choice([1, k, rng.randint(1, k)])}
    if kind == "multi":
        lo = rng.randint(8, 14)
        return {"kind": kind, "n_lo": lo, "n_hi": lo + rng.randint(1, 5), "k": rng.randint(1, 9)}
    if kind == "serve":
        lo = rng.randint(9, 13)
        return {"kind": kind, "n_lo": lo, "n_hi": lo + rng.randint(1, 4), "requests": rng.randint(4, 32)}
    if kind == "window":
        width = rng.choice([24] + list(range(9, 22)) * 2)
        lanes = 1 if width == 24 else rng.randint(1, 16 if width < 20 else 5)
        lo, hi = sorted(rng.sample(range(1, width), 2))
        return {"kind": kind, "width": width, "lanes": lanes, "p_hi": hi, "p_lo": lo}
    if kind == "factor":
        width = rng.randint(11, 18)
        p = rng.randint(5, width - 1)
        fixed = rng.randint(2, p - 2)
        return {"kind": kind, "width": width, "p": p, "fixed": fixed, "occupied": rng.randint(0, fixed)}
    width = rng.randint(9, 16)
    return {"kind": kind, "width": width, "p": rng.randint(2, width - 1), "lanes": rng.randint(1, 8)}


# ---- inputs ---------------------------------------------------------------------


@functools.cache
def primes_below_2_32(count):
    small = [q for q in range(3, 1 << 16, 2) if all(q % d for d in range(3, math.isqrt(q) + 1, 2))]
    out, x = [], (1 << 32) - 1
    while len(out) < count:
        if all(x % q for q in small):
            out.append(x)
        x -= 2
    return tuple(out)


def moduli_of(rng, k):
    return rng.sample(primes_below_2_32(48), k)


@functools.cache
def engine():
    """The engine a program creates once and keeps."""
    return fdp.Engine(0)


@functools.cache
def server():
    """An engine whose server runs as long as the program."""
    eng = fdp.Engine(0)
    eng.server_start(hbm_budget_bytes=SERVER_BUDGET, max_active=8, max_lanes=16)
    return eng


@functools.cache
def stream():
    return torch.cuda.Stream()


def uniform(count, below, gen):
    """`count` uniform words in [0, below), as the uint32 bits of an int32 tensor on the GPU."""
    out = torch.empty(count, dtype=torch.int32, device="cuda")
    for part in out.split(1 << 27):
        part.copy_(torch.randint(below, part.shape, dtype=torch.int64, device="cuda", generator=gen))
    return out


def state(width, moduli, seed):
    """Main and blocked vectors of len(moduli) lanes with uniform residues."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    low = min(moduli)
    return (uniform(motzkin(width) * len(moduli), low, gen), uniform(motzkin(width - 1) * len(moduli), low, gen))


def masks_of(case):
    return [sum(1 << q for q in c) for c in itertools.combinations(range(case["fixed"]), case["occupied"])]


def requests_of(case):
    """(n, k) of the requests of a burst: n over its range, k over 1..8; the seed decides their order."""
    return [(case["n_lo"] + i % (case["n_hi"] - case["n_lo"] + 1), 1 + 3 * i % 8) for i in range(case["requests"])]


def prepare(case, seed):
    rng = random.Random(seed)
    kind = case["kind"]
    s = {"case": case}
    if kind == "residues":
        s["eng"] = engine()
        s["moduli"] = moduli_of(rng, case["k"])
    elif kind == "multi":
        s["eng"] = engine()
        s["problems"] = [(n, moduli_of(rng, case["k"])) for n in range(case["n_lo"], case["n_hi"] + 1)]
    elif kind == "serve":
        s["eng"] = server()
        s["problems"] = [(n, moduli_of(rng, k)) for n, k in requests_of(case)]
        rng.shuffle(s["problems"])
    else:
        s["eng"] = engine()
        s["moduli"] = moduli_of(rng, case.get("lanes", 1))
        with torch.cuda.stream(stream()):
            s["main"], s["block"] = state(case["width"], s["moduli"], seed)
            if kind != "window":
                s["out_main"], s["out_block"] = torch.zeros_like(s["main"]), torch.zeros_like(s["block"])
        if kind == "transfer":
            s["map"] = s["eng"].transfer_map(case["width"], case["p"], paired=True)
        elif kind == "factor":
            s["map"] = s["eng"].factor_map(case["width"], case["p"], case["fixed"], case["occupied"], paired=True,
                                           max_groups=MAX_GROUPS)
            masks = masks_of(case)
            s["masks"] = [masks[i:i + MAX_GROUPS] for i in range(0, len(masks), MAX_GROUPS)]
    return s


# ---- one pass -------------------------------------------------------------------


def run(s):
    case, eng = s["case"], s["eng"]
    kind = case["kind"]
    if kind == "residues":
        return np.array(eng.residues(case["n"], s["moduli"], case["lanes"]).residues, dtype=np.int64)
    if kind == "multi":
        return np.array(eng.residues_multi(s["problems"])[0], dtype=np.int64)
    if kind == "serve":
        ids = [eng.submit(n, moduli) for n, moduli in s["problems"]]
        return np.array([r for i in ids for r in eng.wait(i)["residues"]], dtype=np.int64)
    main, block, on = s["main"], s["block"], stream().cuda_stream
    if kind == "window":
        eng.apply_cells(case["width"], case["p_hi"], case["p_lo"], s["moduli"], main.data_ptr(), block.data_ptr(), on)
        return main, block
    args = (main.data_ptr(), block.data_ptr(), s["out_main"].data_ptr(), s["out_block"].data_ptr(), on)
    if kind == "transfer":
        s["map"].apply(s["moduli"], *args)
    elif kind == "factor":
        for masks in s["masks"]:
            s["map"].apply(s["moduli"][0], masks, *args)
    else:
        eng.reverse2_apply(case["width"], case["p"], s["moduli"], *args)
    return s["out_main"], s["out_block"]


# ---- what a pass cannot do without ------------------------------------------------


@functools.cache
def completions(length, height):
    """Words of N, R, L that lead from `height` to 0 without going below it."""
    if height < 0 or height > length:
        return 0
    return 1 if length == 0 else sum(completions(length - 1, height + d) for d in (0, -1, 1))


def motzkin(width):
    """Main states of a frontier of `width` positions (start height 1); blocked ones are those of width - 1."""
    return completions(width, 1)


@functools.cache
def group_states(width, fixed, occupied):
    """Words of `width` symbols whose bottom `fixed` positions hold R or L at `occupied` given places, N elsewhere."""
    ways = {1: 1}
    for length in range(width, 0, -1):
        free, taken = length > fixed, length <= occupied
        nxt = {}
        for h, w in ways.items():
            for d, ok in ((0, free or not taken), (-1, free or taken), (1, free or taken)):
                if ok and 0 <= h + d:
                    nxt[h + d] = nxt.get(h + d, 0) + w
        ways = nxt
    return ways.get(0, 0)


def solve_work(n, k):
    """One read and one write of the state, and one addition a state and cell, for each row of vertices."""
    m = motzkin(n + 1)
    return {"bytes": 8 * m * max(1, n - 1) * k, "flops": m * n * max(1, n - 1) * k}


def work(case):
    kind = case["kind"]
    if kind == "residues":
        return solve_work(case["n"], case["k"])
    if kind in ("multi", "serve"):
        asked = [(n, case["k"]) for n in range(case["n_lo"], case["n_hi"] + 1)] if kind == "multi" else requests_of(case)
        parts = [solve_work(n, k) for n, k in asked]
        return {m: sum(p[m] for p in parts) for m in ("bytes", "flops")}
    states = motzkin(case["width"]) + motzkin(case["width"] - 1)
    if kind == "window":
        return {"bytes": 8 * states * case["lanes"], "flops": states * case["lanes"] * (case["p_hi"] - case["p_lo"] + 1)}
    if kind == "factor":
        count = math.comb(case["fixed"], case["occupied"])
        states = count * (group_states(case["width"], case["fixed"], case["occupied"]) +
                          group_states(case["width"] - 1, case["fixed"], case["occupied"]))
    return {"bytes": 8 * states * case.get("lanes", 1), "flops": 4 * states * case.get("lanes", 1)}


def tolerance(case):
    return "exact"


# ---- the same results in plain numpy ----------------------------------------------
# A word is an integer with two bits a position (N = 0, R = 1, L = 2), so the
# canonical order (N < R < L from the top) is numeric order and a rank is a
# place in the sorted array of all legal words.


@functools.cache
def words(width):
    w, h = np.zeros(1, np.int64), np.ones(1, np.int64)
    for left in range(width - 1, -1, -1):
        w, h = np.concatenate([4 * w + c for c in (0, 1, 2)]), np.concatenate([h, h - 1, h + 1])
        ok = (h >= 0) & (h <= left)
        w, h = w[ok], h[ok]
    return np.sort(w)


def symbol(w, q):
    return (w >> (2 * q)) & 3


def with_pair(w, p, a, b):
    return (w & ~(np.int64(15) << (2 * p - 2))) | np.int64((a << 2 | b) << (2 * p - 2))


def closures(u, width, p, downwards):
    """(places in u, sources): each closure predecessor of the words u, whose pair at (p, p - 1) is NN.  Downwards: the
    depth-1 L's of the low part, as R under a pair LL; upwards: the depth-1 R's of the high part, as L under RR."""
    opening, closing = (2, 1) if downwards else (1, 2)
    depth = np.ones(len(u), np.int64)
    for q in range(p - 2, -1, -1) if downwards else range(p + 1, width):
        s = symbol(u, q)
        hit = np.flatnonzero((s == opening) & (depth == 1))
        yield hit, with_pair(u[hit] ^ (np.int64(3) << (2 * q)), p, opening, opening)
        depth = np.where(depth > 0, depth + (s == opening) - (s == closing), 0)


@functools.cache
def cell_sources(width, p):
    """Pairs (targets, sources) of one cell over the main vector followed by the blocked one, beside main' += main."""
    t, b = words(width), words(width - 1)
    got = []

    def add(to, w, blocked=False):
        got.append((to, np.searchsorted(b, w) + len(t) if blocked else np.searchsorted(t, w)))

    pair = (t >> (2 * p - 2)) & 15
    moves = {(2, 1): (0, 0), (0, 1): (1, 0), (0, 2): (2, 0)}  # target pair: source pair
    if p == 1:
        moves |= {(1, 0): (0, 1), (2, 0): (0, 2)}
        nn = np.flatnonzero(pair == 0)
        for hit, w in closures(t[nn], width, p, False):
            add(nn[hit], w)
    for (a, c), source in moves.items():
        to = np.flatnonzero(pair == (a << 2 | c))
        add(to, with_pair(t[to], p, *source))
    to = np.flatnonzero(symbol(t, p) == 0)  # the blocked word with position p taken out
    low = (np.int64(1) << (2 * p)) - 1
    add(to, (t[to] & low) | ((t[to] & ~low) >> 2), blocked=True)
    if p >= 2:
        u = (b & low) | ((b & ~low) << 2)
        turn = symbol(u, p - 1) != 0
        add(len(t) + np.flatnonzero(turn), u[turn])
        n = np.flatnonzero(~turn)
        high = np.ones(len(n), np.int64)  # height above position p
        for q in range(p + 1, width):
            s = symbol(u[n], q)
            high += (s == 2).astype(np.int64) - (s == 1)
        add(len(t) + n[high > 0], with_pair(u[n[high > 0]], p, 1, 2))
        for downwards in (True, False):
            for hit, w in closures(u[n], width, p, downwards):
                add(len(t) + n[hit], w)
    return got


def cell(width, p, main, block, modulus):
    both = np.concatenate([main, block])
    out = np.concatenate([main, np.zeros_like(block)])
    for to, source in cell_sources(width, p):
        out[to] += both[source]  # a target appears once in each pair of arrays
    out %= modulus
    return out[:len(main)], out[len(main):]


def residue(n, modulus):
    """Rows 1..n-1 of the sweep between the states of the first row and the same states' sum."""
    width = n + 1
    edges = np.arange(1 << n, dtype=np.int64)
    first = np.full(1 << n, np.int64(1) << (2 * n))
    for p in range(n, 0, -1):
        pair = (first >> (2 * p - 2)) & 15
        turned = np.where(pair == 0, 9, np.where(pair == 4, 1, 2))  # NN -> LR, RN -> NR, LN -> NL
        first = np.where((edges >> (p - 1)) & 1, first ^ ((pair ^ turned) << (2 * p - 2)), first)
    first = np.searchsorted(words(width), first)
    main, block = np.zeros(len(words(width)), np.int64), np.zeros(len(words(width - 1)), np.int64)
    main[first] = 1
    for _ in range(1, n):
        block[:] = 0
        for p in range(n, 0, -1):
            main, block = cell(width, p, main, block, modulus)
    return int(main[first].sum() % modulus)


def unpacked(flat, lanes):
    """[lane][state] int64 of a panel-layout tensor."""
    flat = flat.cpu().numpy().view(np.uint32)
    return fdp.unpack_lanes(flat, len(flat) // lanes, lanes).T.astype(np.int64)


def packed(rows):
    return np.ascontiguousarray(fdp.pack_lanes(np.stack(rows, 1).astype(np.uint32)).view(np.int32))


def exact(case, seed):
    kind = case["kind"]
    if kind == "serve" or (kind == "multi" and case["n_hi"] > 11) or (kind == "residues" and case["n"] > 11):
        return None
    if kind in ("residues", "multi"):
        rng = random.Random(seed)
        sizes = [case["n"]] if kind == "residues" else range(case["n_lo"], case["n_hi"] + 1)
        got = [[residue(n, m) for m in moduli_of(rng, case["k"])] for n in sizes]
        return np.array(got[0] if kind == "residues" else got, dtype=np.int64)
    if case["width"] > 15 or kind == "factor":  # a factor map writes its groups' rows alone
        return None
    moduli = moduli_of(random.Random(seed), case["lanes"])
    main, block = (unpacked(x, case["lanes"]) for x in state(case["width"], moduli, seed))
    cells = range(case["p_hi"], case["p_lo"] - 1, -1) if kind == "window" else (case["p"], case["p"] - 1)
    out_main, out_block = [], []
    for m, a, b in zip(moduli, main, block):
        for p in cells:
            a, b = cell(case["width"], p, a, b, m)
        out_main.append(a)
        out_block.append(b)
    return packed(out_main), packed(out_block)
