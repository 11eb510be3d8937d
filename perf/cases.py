"""Workloads that stand for what the reducer is used for, through its public API.

A case is one kind of call a program makes: normalising one net (boot, normal,
readback), many nets in one batch, a burst of requests to a server, the
no-allocation call, and pre-reducing a Book.  Programs come from
`workloads.py` and from the reference's own example programs; every size is a
depth (2^depth leaves or keys), a loop count or a number of nets.

    listed()            the named cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) the Book and the handle a program keeps
    run(state)          one pass: the normal forms' texts and the Rewrites
    work(case)          bytes and operations of one pass
    exact(case, seed)   the results that plain Python can give
"""
import math
import os
import random
import sys
import time

import numpy as np

ROOT = os.getcwd()
PKG = os.path.join(ROOT, "hvm-64_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import hvm64  # noqa: E402
import workloads as W  # noqa: E402

TIMEOUT_MS = 60000
RADIX = "examples::sort::radix::radix_sort_ctr"
TAIL = "tests::programs::stress_tests::sum_tail"

# Forced Church towers by their numerals, and their interactions (the oracle's
# counts): exponents above these take minutes on one CPU thread.
TOWERS = {"222": 169, "223": 701, "232": 4169, "323": 52588}


def listed():
    return [
        # the smallest call: a command-line run of a small program, all latency
        {"name": "net_sum_6", "kind": "net", "program": "sum", "depth": 6, "heap_mb": 512},
        # the plain configuration: one parallel tree sum of 2^18 leaves
        {"name": "net_sum_18", "kind": "net", "program": "sum", "depth": 18, "heap_mb": 2048},
        # an ordinary single net: a sort of 2^9 keys, its sorted tree read back
        {"name": "net_sort_9", "kind": "net", "program": "sort", "depth": 9, "heap_mb": 2048},
        # a large single net: REF expansion dominates, 2^15 keys read back
        {"name": "net_sort_15", "kind": "net", "program": "sort", "depth": 15, "heap_mb": 4096},
        # Defs of about 60 redexes each, commutation and numeric operators
        {"name": "net_radix_11", "kind": "net", "program": "radix", "depth": 11, "heap_mb": 2048},
        # label-heavy lambda calculus: DUP labels, a frontier of a few redexes
        {"name": "net_church_323", "kind": "net", "program": "church", "tower": "323", "heap_mb": 1024},
        # a sequential loop (a tail-recursive program): one redex at a time
        {"name": "net_tail_1500", "kind": "net", "program": "tail", "count": 1500, "heap_mb": 1024},
        # the flagship: an uneven batch, one persistent launch replayed as a graph
        {"name": "batch_graph_451", "kind": "batch", "nets": 451, "dmin": 8, "dmax": 13, "graph": True,
         "plain": False, "create": False},
        # end to end: a batch of small nets created, reduced and read back each time
        {"name": "batch_new_97", "kind": "batch", "nets": 97, "dmin": 4, "dmax": 9, "graph": False, "plain": False,
         "create": True},
        # serving: a burst of requests to a server started for it
        {"name": "serve_24", "kind": "serve", "requests": 24, "top": 1000000},
        # a caller that must not allocate device memory
        {"name": "noalloc_sort_5", "kind": "noalloc", "program": "sort", "depth": 5, "blocks": 4},
        # ahead-of-time reduction of a Book, Def by Def
        {"name": "pre_reduce_sort_4", "kind": "pre_reduce", "program": "sort", "depth": 4, "heap_mb": 256},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["net", "net", "net", "net", "batch", "batch", "serve", "noalloc", "pre_reduce"])
    if kind == "net":
        case = {"kind": kind, "program": rng.choice(["sum", "sort", "radix", "church", "tail"]),
                "heap_mb": _log_int(rng, 512, 4096)}
        if case["program"] == "church":
            case["tower"] = rng.choice(sorted(TOWERS))
        elif case["program"] == "tail":
            case["count"] = _log_int(rng, 15, 1500)
        else:  # (the depth is the logarithm of the size)
            case["depth"] = rng.randint(2, {"sum": 18, "sort": 14, "radix": 12}[case["program"]])
        return case
    if kind == "batch":
        # (plain: one net per launch; its heap keeps every earlier net's nodes)
        plain, dmin = rng.random() < 0.2, rng.randint(3, 8)
        return {"kind": kind, "nets": _log_int(rng, 2, 40 if plain else 350), "dmin": dmin,
                "dmax": rng.randint(dmin, 11), "graph": rng.random() < 0.5, "plain": plain,
                "create": rng.random() < 0.5}
    if kind == "serve":
        return {"kind": kind, "requests": _log_int(rng, 4, 48), "top": _log_int(rng, 2000, 1000000)}
    if kind == "noalloc":
        program = rng.choice(["sum", "sort"])
        return {"kind": kind, "program": program, "depth": rng.randint(2, 11 if program == "sum" else 7),
                "blocks": rng.randint(1, 4)}
    return {"kind": kind, "program": rng.choice(["sum", "sort"]), "depth": rng.randint(2, 6),
            "heap_mb": _log_int(rng, 128, 1024)}


def _program(case, seed):
    """The case's Book text; the seed picks keys, labels or start values."""
    if case["program"] == "sum":
        return W.tree_sum(case["depth"], seed)
    if case["program"] == "sort":
        return W.bitonic(case["depth"], seed)
    if case["program"] == "radix":
        src, old = W._template(RADIX), "@gen ~ (20 (0 d))"
        new = f"@gen ~ ({case['depth']} ({seed % 4096} d))"
    elif case["program"] == "tail":
        src, old = W._template(TAIL), "@sum ~ (10000000 (0 a))"
        new = f"@sum ~ ({case['count']} ({W.seed24(seed)} a))"
    else:
        # the tower's boolean selects one of two numbers
        src = W.church_big(tuple(int(n) for n in case["tower"]))
        src = src.replace("(@N (@T R))", f"(@N (@T ({W.seed24(seed)} ({W.seed24(seed + 1)} R))))")
        labels = random.Random(seed).sample(range(1, 1 << 10), len(case["tower"]))
        for i in range(len(labels)):
            src = src.replace(f"#{i + 1}{{", f"#<{i}>{{")
        for i, lab in enumerate(labels):
            src = src.replace(f"#<{i}>{{", f"#{lab}{{")
        return src
    if old not in src:
        raise ValueError("the example program changed")
    return src.replace(old, new)


def _entries(case, seed):
    """A batch's nets: the kinds and depths are the case's, the keys the seed's."""
    return [(kind, d, j + (seed % 100000) * case["nets"])
            for kind, d, j in W.batch_entries(case["nets"], case["dmin"], case["dmax"])]


def _requests(case, seed):
    """A server's requests: tree sums, sorts and a few Church nets, sizes
    log-uniform between 10^3 interactions and the case's `top`."""
    rng = random.Random(case["requests"] * 1000003 + case["top"])
    out = []
    for i in range(case["requests"]):
        size = math.exp(rng.uniform(math.log(1e3), math.log(case["top"])))
        j = i + (seed % 100000) * case["requests"]
        r = rng.random()
        if r < 0.47:
            out.append(("sum", max(3, int(round(math.log2(size / 54)))), j))
        elif r < 0.94:
            d = 2
            while W.est_interactions("sort", d + 1) <= size:
                d += 1
            out.append(("sort", d, j))
        else:
            out.append(("church", (4, 2 + i % 4), j))
    return out


def prepare(case, seed):
    state = {"case": case, "cap": _text_cap(case), "tuning": hvm64.Tuning(timeout_ms=TIMEOUT_MS)}
    kind = case["kind"]
    if kind == "pre_reduce":
        state["text"] = _program(case, seed)
    elif kind == "net":
        state["book"] = hvm64.Book.from_str(_program(case, seed))
        state["net"] = hvm64.Net(state["book"], case["heap_mb"] << 20)
    elif kind == "noalloc":
        state["book"] = hvm64.Book.from_str(_program(case, seed))
        state["tuning"].blocks_per_sm = case["blocks"]
    elif kind == "serve":
        reqs = _requests(case, seed)
        state["book"] = hvm64.Book.from_str(W.serving_book(reqs))
        state["requests"] = [(f"main_{j}", W.est_request_nodes(k, p)) for k, p, j in reqs]
    else:
        entries = _entries(case, seed)
        state["book"] = hvm64.Book.from_str(W.batch_book(entries))
        state["names"] = [f"main_{j}" for _, _, j in entries]
        state["mode"] = hvm64.PLAIN if case["plain"] else hvm64.PERSISTENT
        if case["graph"]:
            state["tuning"].flags |= hvm64.TUNE_GRAPH
        if not case["create"]:
            state["batch"] = hvm64.Batch(state["book"], state["names"], 4 << 30)
    return state


def _net_cap(program, depth):
    """Room for one net's normal form: a sorted tree prints at most 48 bytes a leaf."""
    return 16 + (48 << depth if program == "sort" else 16)


def _text_cap(case):
    kind = case["kind"]
    if kind == "batch":
        return sum(_net_cap(k, d) for k, d, _ in _entries(case, 0))
    if kind == "serve":
        return sum(_net_cap(k, p if k != "church" else 0) for k, p, _ in _requests(case, 0))
    if kind == "pre_reduce":
        return 1 << 16
    return _net_cap(case["program"], case.get("depth", 0))


def _bytes(text, cap):
    """The text's bytes in an array whose size depends on the case alone."""
    data = text.encode()
    if len(data) > cap:
        raise ValueError(f"{len(data)} bytes of text, room for {cap}")
    out = np.zeros(cap, dtype=np.uint8)
    out[:len(data)] = np.frombuffer(data, dtype=np.uint8)
    return out


def _counts(rwts):
    return np.array([[r.anni, r.comm, r.eras, r.dref, r.oper] for r in rwts], dtype=np.int64)


def _answers(state, texts, rwts):
    return {"text": _bytes("\n".join(texts), state["cap"]), "rewrites": _counts(rwts)}


def _run_serve(state):
    reqs = state["requests"]
    server = hvm64.Server(state["book"], slots=16, out_pairs=1 << 16, heap_bytes=2 << 30, tuning=state["tuning"])
    try:
        texts, rwts, owner, i = [None] * len(reqs), [None] * len(reqs), {}, 0
        left = len(reqs)
        while left:
            busy = False
            while i < len(reqs) and len(owner) < server.slots:
                name, nodes = reqs[i]
                owner[server.submit(name, nodes=nodes)] = i
                i += 1
                busy = True
            for ticket in server.poll():
                k = owner.pop(ticket)
                texts[k], rwts[k], _ = server.result(ticket)
                left -= 1
                busy = True
            if not busy:
                time.sleep(0.0002)
    finally:
        server.close()
    return _answers(state, texts, rwts)


def run(state):
    kind = state["case"]["kind"]
    if kind == "net":
        net = state["net"]
        net.boot("main")
        rwts = net.normal(state["tuning"])
        return _answers(state, [net.readback()], [rwts])
    if kind == "noalloc":
        text, rwts = hvm64.normal_noalloc(state["book"], "main", state["tuning"])
        return _answers(state, [text], [rwts])
    if kind == "pre_reduce":
        text, rwts, late = hvm64.pre_reduce(state["text"], heap_bytes=state["case"]["heap_mb"] << 20, tuning=state["tuning"])
        return {"not_normal": len(late), **_answers(state, [text], [rwts])}
    if kind == "serve":
        return _run_serve(state)
    batch = state.get("batch") or hvm64.Batch(state["book"], state["names"], 4 << 30)
    batch.normal(state["mode"], state["tuning"])
    return _answers(state, [batch.readback(i) for i in range(batch.n)], batch.rwts)


def _interactions(case):
    """Interactions of one pass (exact for sums, loops and towers; the sorts'
    are fitted on the oracle's counts)."""
    kind = case["kind"]
    if kind == "batch":
        return sum(W.est_interactions(k, d) for k, d, _ in _entries(case, 0))
    if kind == "serve":
        return sum(600 if k == "church" else W.est_interactions(k, p) for k, p, _ in _requests(case, 0))
    if case["program"] in ("sum", "sort"):
        # (pre-reduce also visits about 40 Defs of a few interactions each)
        return W.est_interactions(case["program"], case["depth"]) + (200 if kind == "pre_reduce" else 0)
    if case["program"] == "radix":
        return 1260 * (1 << case["depth"])
    if case["program"] == "tail":
        return 12 * case["count"] + 9
    return TOWERS[case["tower"]]


def work(case):
    """An interaction reads the two 16-byte nodes of its redex and writes at
    least the two wires it joins (8 bytes each); one operation each."""
    n = _interactions(case)
    return {"bytes": 48.0 * n, "flops": float(n)}


def exact(case, seed):
    """The normal form where it is a number that plain Python can give; the
    other outputs are texts and counts, which stay equal."""
    if case["kind"] in ("net", "noalloc") and case["program"] in ("sum", "tail"):
        if case["program"] == "sum":
            keys = np.arange(1 << case["depth"], dtype=np.int64) ^ W.seed24(seed)
            t = (keys * W.K1) & W.M24
            u = ((t ^ (t >> 12)) * W.K2) & W.M24
            value = int((u ^ (u >> 11)).sum()) & W.M24
        else:
            n = case["count"]
            value = (W.seed24(seed) + n * (n - 1) // 2) & W.M24
        return {"text": _bytes(str(value), _text_cap(case)), "rewrites": None}
    return None
