"""The measured work of this framework, through its public Python binding.

What a user does with it is: generate a graph, hand it on as an edge list or as
a CSR, look at its degrees, generate many graphs at once, write one out.  Every
case is one such call.  A graph is a pure function of its parameters, so the
inputs of a generation are the parameters and a graph seed drawn from the
case's seed; the later passes (CSR, degrees, text) take a graph that has been
generated before.

listed() holds the cases measured by name, draw() further ones of the same
ranges, prepare() makes a case's state, run() is one pass.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "cuppa-public_b200"))

import cuppa_b200 as cb  # noqa: E402

CLIQUE, STAR = cb.PA_SEED_CLIQUE, cb.PA_SEED_STAR_REF


def _graph(name, op, n, d, p, bits=32, star=False, slots=False, ba=False):
    case = {"name": name} if name else {}
    return {**case, "op": op, "n": n, "d": d, "p": p, "bits": bits, "star": star,
            "slots": slots, "ba": ba}


def listed():
    return [
        # the 10^5-node graph of the smallest benchmark configuration: a call
        # whose launches and dependency chains are all its time
        _graph("gen_small", "gen", 100_000, 4, 0.5),
        # an ordinary mid-sized graph, neither n nor d round, most slots copies,
        # the reference's star seed
        _graph("gen_mid", "gen", 1_234_567, 7, 0.3, star=True),
        # the headline configuration's d, p and id width at the largest size of
        # which three states fit the card
        _graph("gen_large", "gen", 1 << 28, 4, 0.5, bits=64),
        # pure copying (p = 0), the model's other extreme, targets only
        _graph("gen_copy", "gen", 1 << 24, 4, 0.0, slots=True),
        # the Barabasi-Albert model of -A sba
        _graph("gen_ba", "gen", 20_000_003, 5, 0.0, bits=64, star=True, ba=True),
        # more edges per node than a warp has lanes
        _graph("gen_wide", "gen", 200_000, 100, 0.4),
        # 64 graphs of the many-instances mix (n = round(10^U(3,7))) in one call
        {"name": "batch_mix", "op": "batch", "count": 64, "n_lo": 1e3, "n_hi": 1e7,
         "mix": 0},
        # adjacency of a small graph, as a request server's express lane builds it
        _graph("csr_small", "csr", 20_000, 6, 0.5),
        # adjacency with hubs and 32-bit ids, a mid size
        _graph("csr_mid", "csr", 3_000_017, 9, 0.2),
        # d, p and id width of the adjacency benchmark configuration, at a quarter of its nodes
        _graph("csr_large", "csr", 25_000_000, 16, 0.5, bits=64),
        # the degree pass behind the degree distribution
        _graph("degrees", "degrees", 1 << 24, 8, 0.3),
        # the edge list as text, taken over by the host chunk by chunk
        _graph("text", "text", 1_000_000, 4, 0.5),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["gen", "gen", "gen", "gen", "wide", "batch", "csr", "csr", "degrees", "text"])
    if op == "batch":
        return {"op": "batch", "count": rng.randint(8, 64), "n_lo": 1e3,
                "n_hi": float(_logint(rng, 1e4, 5e6)), "mix": rng.randint(1, 10 ** 6)}
    p = round(rng.uniform(0.1, 0.9), 6)
    bits = rng.choice([32, 64])
    star = rng.random() < 0.3
    if op == "wide":
        d = rng.randint(33, 160)
        return _graph("", "gen", _logint(rng, 5e3, 2e7 / d), d, p, bits, star)
    d = rng.randint(1, 32)
    edges = {"gen": 2.0 ** 28, "csr": 2.0 ** 28, "degrees": 2.0 ** 27, "text": 4e6}[op]
    n = max(d + 2, _logint(rng, 1e4, edges / d))
    if op != "gen":
        return _graph("", op, n, d, p, bits, star)
    kind = rng.choice(["pairs", "pairs", "slots", "copy", "ba"])
    if kind == "copy":
        n, p = max(d + 2, n // 8), 0.0
    return _graph("", "gen", n, d, 0.0 if kind == "ba" else p, bits, star or kind == "ba",
                  kind == "slots", kind == "ba")


def _params(case, seed):
    return cb.make_params(case["n"], case["d"], case["p"], seed=1000 + seed, id_bits=case["bits"],
                          seed_mode=STAR if case["star"] else CLIQUE,
                          layout=cb.PA_LAYOUT_SLOTS if case["slots"] else cb.PA_LAYOUT_PAIRS,
                          model=cb.PA_MODEL_BA if case["ba"] else cb.PA_MODEL_COPY)


def _mix(case, seed):
    """The many-instances mix: n = round(10^U), d = U{1..32}, p = U(0.1, 0.9);
    the sizes are the case's, the graph seeds come from the seed."""
    rng = random.Random(case["mix"])
    out = []
    for i in range(case["count"]):
        d = rng.randint(1, 32)
        n = max(_logint(rng, case["n_lo"], case["n_hi"]), d + 1)
        out.append((n, d, round(rng.uniform(0.1, 0.9), 6), 1000 + 4096 * seed + i))
    return out


def prepare(case, seed):
    if case["op"] == "batch":
        return {"op": "batch",
                "batch": cb.Batch([cb.make_params(n, d, p, seed=s) for n, d, p, s in _mix(case, seed)])}
    prm = _params(case, seed)
    st = {"op": case["op"], "prm": prm}
    if case["op"] == "gen":
        # buffers kept by the caller, as in a loop over graph seeds
        st["edges"], st["scratch"] = cb.alloc_buffers(prm)
    else:
        st["edges"], _ = cb.generate(prm)
    if case["op"] == "text":
        width = len(str(case["n"] - 1))
        st["text"] = np.zeros(cb.edge_count(prm) * (2 * width + 2), dtype=np.uint8)
    return st


def run(st):
    op = st["op"]
    if op == "gen":
        cb.generate_into(st["prm"], st["edges"], st["scratch"])
        return st["edges"]
    if op == "batch":
        st["batch"].generate()
        return st["batch"].edges
    if op == "csr":
        return cb.build_csr(st["prm"], st["edges"])
    if op == "degrees":
        return cb.degrees(st["prm"], st["edges"])
    buf, at = st["text"], 0

    def sink(chunk):
        nonlocal at
        buf[at:at + len(chunk)] = np.frombuffer(chunk, dtype=np.uint8)
        at += len(chunk)

    cb.stream_edges(st["prm"], st["edges"], sink)
    return buf, at


def _edge_count(n, d, star):
    return (d if star else d * (d + 1) // 2) + (n - d - 1) * d


def work(case):
    """Each input read once and each output written once; no arithmetic is counted."""
    if case["op"] == "batch":
        # the mix's mean edge count (log-uniform n, mean d 16.5), 8 bytes per pair
        lo, hi = case["n_lo"], case["n_hi"]
        mean_n = (hi - lo) / math.log(hi / lo)
        return {"bytes": 8.0 * 16.5 * mean_n * case["count"], "flops": 0}
    n, d, idb = case["n"], case["d"], case["bits"] // 8
    E = _edge_count(n, d, case["star"])
    if case["op"] == "gen":
        return {"bytes": (n - d - 1) * d * idb if case["slots"] else 2 * E * idb, "flops": 0}
    if case["op"] == "csr":        # pairs in; both directions' ids and the row starts out
        return {"bytes": 2 * E * idb + 2 * E * idb + 8 * (n + 1), "flops": 0}
    if case["op"] == "degrees":    # pairs in, one 64-bit count per node out
        return {"bytes": 2 * E * idb + 8 * n, "flops": 0}
    return {"bytes": 2 * E * idb + E * (2 * math.log10(n) + 2), "flops": 0}


# ---------------------------------------------------------------------------
# The definition, in plain Python integers (the smaller cases only)
# ---------------------------------------------------------------------------
def _philox(c0, c2, c3, key):
    """Word quadruple of Philox4x32-10 at counter (c0, 0, c2, c3)."""
    m32 = 0xFFFFFFFF
    c1, k0, k1 = 0, key & m32, key >> 32
    for _ in range(10):
        a, b = 0xD2511F53 * c0, 0xCD9E8D57 * c2
        c0, c1, c2, c3 = (b >> 32) ^ c1 ^ k0, b & m32, (a >> 32) ^ c3 ^ k1, a & m32
        k0, k1 = (k0 + 0x9E3779B9) & m32, (k1 + 0xBB67AE85) & m32
    return c0, c1, c2, c3


def _sequential(n, d, p, key, star, ba):
    """Target rows of nodes 0..n-1, generated one node after the other."""
    if star:
        rows = [[v] * d for v in range(d)] + [list(range(d))]
    else:
        rows = [[j for j in range(d + 1) if j != v] for v in range(d + 1)]
    pth = min(int(p * 4294967296.0), 1 << 32)
    for u in range(d + 1, n):
        row = []
        for i in range(d):
            r = 0
            while True:
                w0, w1, w2, w3 = _philox(u, i, r, key)
                x = (w1 << 32 | w0) * u
                v = x >> 64
                if ba:
                    q = (x & ((1 << 64) - 1)) * 2 * d >> 64
                    direct, k = q & 1, q >> 1
                else:
                    direct, k = w2 < pth, w3 * d >> 32
                t = v if direct else rows[v][k]
                if t not in row:
                    break
                r += 1
            row.append(t)
        rows.append(row)
    return rows


def exact(case, seed):
    if case["op"] not in ("gen", "csr", "degrees"):
        return None
    n, d, bits = case["n"], case["d"], case["bits"]
    if n * d > 500_000:
        return None
    rows = _sequential(n, d, case["p"], 1000 + seed, case["star"], case["ba"])
    dt = torch.int64 if bits == 64 else torch.int32
    targets = torch.tensor(rows[d + 1:], dtype=torch.int64)
    if case["op"] == "gen" and case["slots"]:
        return targets.to(dt)
    head = [(d, j) for j in range(d)] if case["star"] else \
        [(v, j) for v in range(1, d + 1) for j in range(v)]
    src = torch.arange(d + 1, n, dtype=torch.int64).repeat_interleave(d)
    pairs = torch.cat([torch.tensor(head, dtype=torch.int64).reshape(-1, 2),
                       torch.stack([src, targets.reshape(-1)], dim=1)])
    if case["op"] == "gen":
        return pairs.to(dt)
    both = torch.cat([pairs, pairs.flip(1)])
    deg = torch.bincount(both[:, 0], minlength=n)
    if case["op"] == "degrees":
        return deg
    rowptr = torch.cat([torch.zeros(1, dtype=torch.int64), torch.cumsum(deg, 0)])
    order = torch.sort(both[:, 0] * n + both[:, 1]).indices
    return rowptr, both[order, 1].to(dt)
