"""The work that users of the blocking engine have it do, as cases to be timed.

A case names an entry point, a table shape and its sizes:

* ``session``: both tables resident on the GPU (:class:`Session`), one batched
  run into the caller's device buffers, then the candidate set in row order
  (what a matcher downstream reads);
* ``blocker``: the reference's class shape (:class:`HyperBlocker`) over two CSV
  files read at construction: ``Run()``, host tables to sorted host pairs;
* ``block`` / ``streamed``: the one-shot calls from host tables to host pairs,
  whole or in partition windows under a device-memory bound;
* ``cli``: ``run_hyperblocker_exec`` from two CSV files to the pair file;
* ``serve``: requests of left records against a resident right table, all
  submitted, then all polled.

Table shapes (the package's synthetic generators):

* ``dblp``: titles, authors, 5 venues, years 1994-2003; one rule (same year,
  titles and authors alike) -- the DBLP-ACM shape;
* ``scholar``: 500 skewed venues, years 1980-2005; two rules -- the
  DBLP-Scholar shape;
* ``rules8``: the same columns and a skewed key, 8 rules of 1-2 equalities and
  1-3 similarities, 64 uneven partitions;
* ``long``: titles and authors of 64-256 characters, a skewed key of 2^20
  values, 3 rules, 64 partitions.

Outputs are row numbers, counts and bytes, all whole: there is nothing to hold
against 64-bit arithmetic, so the file has no ``exact``.  They come in buffers
sized from the tables, as a program that keeps its buffers between calls has
them: the pairs in row order first, then padding.
"""
from __future__ import annotations

import math
import os
import tempfile

import numpy as np
import torch

import hyperblocker_gb300 as hb
from hyperblocker_gb300 import synth, synth_big

VENUES5 = synth_big.VENUES[:5]
YEARS10 = [str(y).encode() for y in range(1994, 2004)]
DBLP_RULES = [synth.rule_yaml([4], [(1, 0.89), (2, 0.85)])]
SCHOLAR_RULES = [synth.rule_yaml([4], [(1, 0.89), (2, 0.85)]), synth.rule_yaml([3], [(1, 0.95)])]


def listed():
    return [
        # the reference's own example size, tables kept on the GPU: the
        # smallest run, where launches and latency count
        {"name": "dblp_session", "call": "session", "shape": "dblp", "left": 2616, "right": 2294,
         "partitions": 1},
        # the same through the reference's class shape, encoding included
        {"name": "dblp_blocker", "call": "blocker", "shape": "dblp", "left": 2616, "right": 2294,
         "partitions": 1},
        # a small table against a large one, resident and one-shot
        {"name": "scholar_session", "call": "session", "shape": "scholar", "left": 2600,
         "right": 64263, "partitions": 8},
        {"name": "scholar_block", "call": "block", "shape": "scholar", "left": 2600,
         "right": 64263, "partitions": 8},
        # many rules over uneven partitions: medium and large
        {"name": "rules8_session_30k", "call": "session", "shape": "rules8", "left": 30011,
         "right": 29989, "partitions": 64},
        {"name": "rules8_session_150k", "call": "session", "shape": "rules8", "left": 150_000,
         "right": 150_000, "partitions": 64},
        # long strings and a large key domain: resident, and streamed in
        # windows as for tables that do not fit
        {"name": "long_session", "call": "session", "shape": "long", "left": 40_013,
         "right": 59_999, "partitions": 64},
        {"name": "long_streamed", "call": "streamed", "shape": "long", "left": 40_000,
         "right": 60_000, "partitions": 64, "window_mb": 64},
        # the whole program, CSV files to pair file
        {"name": "cli_files", "call": "cli", "shape": "rules8", "left": 25_000, "right": 40_000,
         "partitions": 64},
        # serving: one small request (latency), and a burst of mixed sizes
        {"name": "serve_single", "call": "serve", "resident": 1_000_000, "requests": 1,
         "min_rows": 16, "max_rows": 16},
        {"name": "serve_burst", "call": "serve", "resident": 1_000_000, "requests": 24,
         "min_rows": 1, "max_rows": 5000},
    ]


def _log(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["session dblp", "session scholar", "session rules8", "session rules8",
                       "session long", "blocker dblp", "block scholar", "streamed long",
                       "cli rules8", "serve", "serve"])
    if kind == "serve":
        lo = _log(rng, 1, 64)
        return {"call": "serve", "resident": _log(rng, 200_000, 1_000_000),
                "requests": _log(rng, 1, 24), "min_rows": lo, "max_rows": _log(rng, lo, 5000)}
    call, shape = kind.split()
    left, right = {"dblp": ((300, 6000), (300, 6000)), "scholar": ((500, 6000), (5000, 80_000)),
                   "rules8": ((4000, 140_000), (4000, 140_000)),
                   "long": ((4000, 45_000), (4000, 60_000))}[shape]
    if call == "cli":
        left, right = (4000, 30_000), (4000, 40_000)
    case = {"call": call, "shape": shape, "left": _log(rng, *left), "right": _log(rng, *right),
            "partitions": {"dblp": rng.choice([1, 2, 3]), "scholar": rng.choice([1, 5, 8, 16])}.get(
                shape, rng.choice([16, 64, 100]))}
    if call == "streamed":
        case["window_mb"] = rng.choice([32, 64, 96])
    return case


# ------------------------------------------------------------------ inputs
_kept = {}


def _gen(seed):
    """The generators over one vocabulary, drawing from the seed."""
    if "gen" not in _kept:
        _kept["gen"] = synth_big.Gen(0)
    g = _kept["gen"]
    g.rng = np.random.Generator(np.random.PCG64(int(seed)))
    return g


def _dblp_rows(g, n, base):
    return [synth_big._ids(base, n), g.titles(n), g.authors(n),
            synth_big._categorical(VENUES5, g.rng.integers(0, 5, size=n)),
            synth_big._categorical(YEARS10, g.rng.integers(0, 10, size=n))]


def _tables(case, seed):
    """(left BlobTable, right BlobTable, rule documents) of a case's shape and
    sizes; a share of the right rows are perturbed copies of left rows."""
    g = _gen(seed)
    n_l, n_r = case["left"], case["right"]
    shape = case["shape"]
    if shape == "dblp":
        names, rules = synth_big.NAMES5, DBLP_RULES
        rows = lambda n, base: _dblp_rows(g, n, base)  # noqa: E731
        n_true = min(n_l, n_r) * 9 // 10
    elif shape == "scholar":
        names, rules = synth_big.NAMES5, SCHOLAR_RULES
        rows = lambda n, base: synth_big.make_rows(g, n, base, False)  # noqa: E731
        n_true = min(n_l, n_r // 12)
    elif shape == "rules8":
        if "rules8" not in _kept:  # the rule set does not depend on the rows
            _kept["rules8"] = synth_big.c3(64, 64, 1).rules
        names, rules = synth_big.NAMES6, _kept["rules8"]
        rows = lambda n, base: synth_big.make_rows(g, n, base, True)  # noqa: E731
        n_true = min(n_l, n_r) // 50
    else:
        if "long" not in _kept:
            _kept["long"] = synth_big.c5(64, 64, 1).rules
        names, rules = synth_big.NAMES_C5, _kept["long"]
        keys = g.rng.integers(0, 1 << 32, size=1 << 20, dtype=np.uint64)
        rows = lambda n, base: synth_big._c5_rows(g, n, base, keys)  # noqa: E731
        n_true = min(n_l, n_r) // 50
    left = synth_big._with_header(names, rows(n_l, 10_000_000))
    right = rows(n_r - n_true, 50_000_000)
    src = np.sort(g.rng.integers(0, n_l, size=n_true))
    right = synth_big._append(right, synth_big.perturbed_copies(
        g, left, src, 50_000_000 + n_r - n_true))
    return left, synth_big._with_header(names, right), rules


def _write_csv(path, table):
    """Every text cell quoted, the header line first, as DBLP-ACM's files are."""
    cols = []
    for blob, off in table.cols:
        raw, o = blob.tobytes(), off.tolist()
        cols.append([raw[o[i]:o[i + 1]] for i in range(len(o) - 1)])
    with open(path, "wb") as f:
        f.write(b"".join(b'"' + b'","'.join(row) + b'"\r\n' for row in zip(*cols)))


def _files(case, seed):
    """The tables as CSV files and the rules as a directory, in a folder that
    goes when the state does."""
    left, right, rules = _tables(case, seed)
    folder = tempfile.TemporaryDirectory(prefix="hbx_cases_")
    paths = {"left": os.path.join(folder.name, "l.csv"), "right": os.path.join(folder.name, "r.csv"),
             "rules": os.path.join(folder.name, "rules"), "out": os.path.join(folder.name, "pairs.csv")}
    _write_csv(paths["left"], left)
    _write_csv(paths["right"], right)
    os.mkdir(paths["rules"])
    for k, doc in enumerate(rules):
        with open(os.path.join(paths["rules"], "%d.yaml" % k), "w") as f:
            f.write(doc)
    return folder, paths


def _context():
    """One context for the process, as a program that blocks more than one
    pair of tables keeps it."""
    if "ctx" not in _kept:
        _kept["ctx"] = hb.Context(0)
    return _kept["ctx"]


def _server(resident):
    """The server over the resident table: what stays open between requests.
    The last one opened is kept for the next state of the same size."""
    if _kept.get("server", (0, None))[0] != resident:
        _kept.pop("server", None)
        ctx = hb.Context(0)
        plans = [hb.Plan.from_yaml([doc], ctx) for doc in synth_big.SERVE_RULES]
        g = _gen(4)
        table = synth_big._with_header(
            synth_big.NAMES5, synth_big.make_rows(g, resident, 100_000_000, False))
        _kept["server"] = (resident, hb.Server(ctx, plans, hb.Table.from_columns(table.cols, ctx)),
                           table)
    return _kept["server"]


def _request_rows(case):
    lo, hi, k = case["min_rows"], case["max_rows"], case["requests"]
    rows = [int(round(lo * (hi / lo) ** ((i + 0.5) / k))) for i in range(k)]
    return [rows[i * 7 % k] for i in range(k)] if k % 7 else rows


def _requests(case, seed, resident_table):
    """(plan, columns) per request: numbers of fresh records evenly spread over
    the logarithm of the case's range, small and large ones mixed, one in fifty
    a perturbed copy of a resident row."""
    g = _gen(seed)
    out = []
    for i, n in enumerate(_request_rows(case)):
        k = max(1, n // 50)
        cols = synth_big.make_rows(g, n - k, 900_000_000, False) if n > k else None
        src = g.rng.integers(0, resident_table.n_rows - 1, size=k)
        copies = synth_big.perturbed_copies(g, resident_table, src, 900_000_000 + n - k)
        out.append(((i + 1) % len(synth_big.SERVE_RULES),
                    synth_big._append(cols, copies) if cols else copies))
    return out


def _room(case):
    """Pairs that a program sizes its buffers for: about one and a half times
    what such tables match (the text's distribution settles it)."""
    n_l, n_r = case["left"], case["right"]
    return {"dblp": min(n_l, n_r) + 64,
            "scholar": int(3e-3 / min(8, case["partitions"]) * n_l * n_r) + n_r // 6,
            "rules8": int(4.5e-4 * n_l * n_r) + 20_000,
            "long": int(3e-4 * n_l * n_r) + 8192}[case["shape"]]


def prepare(case, seed):
    call = case["call"]
    if call == "serve":
        _, server, table = _server(case["resident"])
        return {"call": call, "server": server, "requests": _requests(case, seed, table),
                "room": [60 * n + 8000 for n in _request_rows(case)]}
    if call in ("blocker", "cli"):
        folder, paths = _files(case, seed)
        state = {"call": call, "folder": folder, "out": paths["out"], "room": _room(case)}
        if call == "blocker":
            state["blocker"] = hb.HyperBlocker(paths["rules"], paths["left"], paths["right"], "",
                                               case["partitions"])
        else:
            state["argv"] = ["run_hyperblocker_exec", "-data_l", paths["left"], "-data_r",
                             paths["right"], "-rule_dir", paths["rules"], "-n_partitions",
                             str(case["partitions"]), "-o", paths["out"]]
        return state
    left, right, rules = _tables(case, seed)
    ctx = _context()
    state = {"call": call, "ctx": ctx, "partitions": case["partitions"], "room": _room(case),
             "plan": hb.Plan.from_yaml(rules, ctx), "left": hb.Table.from_columns(left.cols, ctx),
             "right": hb.Table.from_columns(right.cols, ctx)}
    if call == "streamed":
        state["window"] = case["window_mb"] << 20
    if call == "session":
        if "stream" not in _kept:
            _kept["stream"] = torch.cuda.Stream()
        state["stream"] = _kept["stream"]
        state["session"] = hb.Session(ctx, state["plan"], state["left"], state["right"],
                                      case["partitions"])
        n = state["session"].count("batched", state["stream"].cuda_stream)
        state["rows"] = torch.empty((2, max(state["room"], n)), dtype=torch.int32, device="cuda")
    return state


# ------------------------------------------------------------------ one pass
def _padded(pairs, room):
    out = np.full((max(room, len(pairs)), 2), 0xffffffff, dtype=np.uint32)
    out[:len(pairs)] = pairs
    return out


def _in_order(rows, room):
    """Left and right rows as one sorted array of left << 32 | right."""
    out = np.full(max(room, len(rows[0])), -1, dtype=np.int64)
    keys = out[:len(rows[0])]
    np.left_shift(rows[0], 32, out=keys, dtype=np.int64, casting="unsafe")
    keys |= rows[1]
    keys.sort()
    return out


def run(state):
    call = state["call"]
    if call == "session":
        stream, rows = state["stream"], state["rows"]
        with torch.cuda.stream(stream):
            rows.fill_(0x7fffffff)
            n = state["session"].run_device("batched", rows[0].data_ptr(), rows[1].data_ptr(),
                                            rows.shape[1], stream.cuda_stream)
            # left row in the high half, right row in the low half
            keys = torch.stack((rows[1], rows[0]), 1).view(torch.int64).view(-1)
            return {"n": n, "pairs": torch.sort(keys).values}
    if call == "serve":
        server, requests, room = state["server"], state["requests"], state["room"]
        for k, (plan, cols) in enumerate(requests):
            server.submit(k, plan, cols)
        done = {}
        while len(done) < len(requests):
            res = server.poll(-1)
            if res["status"] != hb.OK:
                raise RuntimeError("request %d: status %d" % (res["id"], res["status"]))
            done["request %02d" % res["id"]] = _padded(res["pairs"], room[res["id"]])
        return done
    if call == "blocker":
        return _padded(state["blocker"].Run(), state["room"])
    if call == "cli":
        if os.path.exists(state["out"]):  # the program appends
            os.remove(state["out"])
        if hb.run_cli(state["argv"]) != 0:
            raise RuntimeError("run_hyperblocker_exec failed")
        size = os.path.getsize(state["out"])
        text = np.zeros(max(20 * state["room"], size), dtype=np.uint8)
        with open(state["out"], "rb") as f:
            f.readinto(text[:size])
        return text
    if call == "block":
        rows, _ = hb.block(state["ctx"], state["plan"], state["left"], state["right"],
                           state["partitions"], stack=False)
    else:
        rows, _ = hb.block_streamed(state["ctx"], state["plan"], state["left"], state["right"],
                                    state["partitions"], state["window"])
        rows = rows[:, 0], rows[:, 1]
    return _in_order(rows, state["room"])


# ------------------------------------------------------------------ its work
def _zipf_equal(n, s):
    """Probability that two draws of a Zipf(s) over n values agree."""
    w = 1.0 / np.arange(1, n + 1, dtype=np.float64) ** s
    return float(np.sum((w / w.sum()) ** 2))


def work(case):
    """Bytes: the text and codes that the path reads once (of a resident
    table: the records of the candidates) and the pairs (8 bytes each) it
    writes once.  Operations: for each candidate pair -- same
    partition, a rule's equalities hold -- one upper bound of its symbol
    matches, packed four to a word (8 minima and 8 sums over 32 symbol
    counts), without which no pair can be ruled out."""
    if case["call"] == "serve":
        lo, hi = case["min_rows"], case["max_rows"]
        mean = (hi - lo) / math.log(hi / lo) if hi > lo else lo
        rows = case["requests"] * mean
        pairs = rows * case["resident"] * _zipf_equal(500, 1.0) / 26
        return {"bytes": 160.0 * rows + 64.0 * min(pairs, case["resident"]), "flops": 16.0 * pairs}
    n_l, n_r, shape = case["left"], case["right"], case["shape"]
    if shape == "dblp":
        row, pairs, out = 140, n_l * n_r / 10, min(n_l, n_r)
    elif shape == "scholar":
        row, out = 140, n_r // 12
        pairs = n_l * n_r * (1 / 26 + _zipf_equal(500, 1.0) / min(26, case["partitions"]))
    elif shape == "rules8":
        same = _zipf_equal(256, 1.3)
        same += (1 - same) / case["partitions"]  # other keys of the same partition
        row, out = 150, 5.2e-4 * n_l * n_r
        pairs = n_l * n_r * same * (1 / 26 + _zipf_equal(500, 1.0))
    else:
        row, pairs, out = 330, n_l * n_r * _zipf_equal(1 << 20, 1.0), min(n_l, n_r) // 50
    return {"bytes": row * (n_l + n_r) + 8.0 * out, "flops": 16.0 * pairs}
