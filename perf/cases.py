"""What the engine's users run, as cases to be timed and compared.

Two kinds of work.  "koszul" cases are the synthetic Koszul operators
(KoszulEngine, KoszulBatch): single applications of d, d^T and S on device
buffers, sequence sessions, and whole sequences through host buffers, in both
arithmetic forms.  "cyclic" cases are the eliminated cyclic operator of one
sector (CyclicEngine), on instances made here with the shape of the published
ones (genus g, order g / 2, character blocks of at most two rows).

Sizes are those of bench.py's workloads (r = 10, 19 and 23; the batched
sectors' r = 19-21, k = 8-10, dims 12-40), of the tests' ragged shapes, and of
the published genera from 12 up.
"""
import json
import math
import os
import tempfile
from itertools import combinations

import numpy as np
import torch

from prym_green_ancillary_b200 import CyclicEngine, KoszulBatch, KoszulEngine

PRIME = 32003          # the synthetic workloads' prime; 32749 is the largest below 2^15
PRIMES = (32003, 32003, 32749, 10007)


def _koszul(name, call, form, r, k, ci, co, n, steps=0, p=PRIME):
    return {"name": name, "kind": "koszul", "call": call, "form": form, "r": r, "k": k, "ci": ci, "co": co,
            "n": n, "p": p, "steps": steps}


def listed():
    return [
        # One application on the smallest workload: launch latency and the call itself.
        _koszul("apply_small_int8", "apply", "int8", 10, 4, 16, 24, 8),
        # The smallest workload's whole sequence (2 N / n + 16 moments): thousands of short kernels.
        _koszul("sequence_small_int8", "sequence", "int8", 10, 4, 16, 24, 8, 855),
        # Single d and d^T on device buffers, as a caller that owns the iteration uses them: the genus-20-like
        # operator, and a ragged sector of the batched range (odd dimension, 32-wide block).
        _koszul("forward_genus20_int8", "forward", "int8", 19, 9, 20, 28, 16),
        _koszul("transpose_ragged_int8", "transpose", "int8", 20, 8, 21, 29, 32),
        # One application in the plain form on odd dimensions and another prime.
        _koszul("apply_ragged_plain", "apply", "plain", 17, 7, 17, 25, 32, p=32749),
        # The sequence session that the framework is for: the genus-20-like workload in both forms (the plain
        # form's as a check run, shorter), and the genus-24-like one, the largest that the benchmark has.
        _koszul("sequence_genus20_int8", "sequence", "int8", 19, 9, 20, 28, 16, 64),
        _koszul("sequence_genus20_plain", "sequence", "plain", 19, 9, 20, 28, 16, 16),
        _koszul("sequence_genus24_int8", "sequence", "int8", 23, 11, 32, 40, 32, 8),
        # The same call on host buffers: copies in and out included.
        _koszul("sequence_host_genus20_int8", "host", "int8", 19, 9, 20, 28, 16, 100),
        # Uneven sectors advanced together (the batched workload's ranges, four of its sectors' sizes).
        {"name": "batch_sectors_int8", "kind": "batch", "sectors": "19,8,14,22,8;19,9,24,32,16;20,8,18,26,32;19,8,33,41,16",
         "p": PRIME, "steps": 16},
        # The paper operator: the smallest published genus, where launches count, and one whose tables exceed
        # the L2.  Rounds of four moments (two applications each) and the download of the sequence.
        {"name": "cyclic_genus20", "kind": "cyclic", "genus": 20, "sector": 0, "rounds": 1000},
        {"name": "cyclic_genus26", "kind": "cyclic", "genus": 26, "sector": 3, "rounds": 100},
    ]


def draw(rng):
    kind = rng.choice(["koszul"] * 5 + ["batch"] + ["cyclic"] * 2)
    if kind == "cyclic":
        genus = rng.choice([12, 14, 16, 18, 20, 22, 24])
        return {"kind": kind, "genus": genus, "sector": rng.randrange(genus // 2),
                "rounds": round(math.exp(rng.uniform(math.log(20), math.log(400))))}
    if kind == "batch":
        sectors = []
        for _ in range(rng.randint(2, 5)):
            r, ci = rng.randint(9, 18), rng.randint(12, 32)
            sectors.append((r, max(2, r // 2 - rng.randint(0, 2)), ci, ci + 8, rng.choice([8, 16, 32])))
        return {"kind": kind, "sectors": ";".join(",".join(map(str, s)) for s in sectors), "p": PRIME,
                "steps": rng.randint(8, 40)}
    call = rng.choice(["forward", "transpose", "apply", "sequence", "sequence", "host"])
    form = rng.choice(["int8", "int8", "plain"])
    r = rng.randint(8, 20 if form == "int8" else 17)
    k = max(2, min(r - 1, r // 2 + rng.randint(-2, 1)))
    ci = rng.randint(8, 36)
    steps = round(math.exp(rng.uniform(math.log(4), math.log(120)))) if call in ("sequence", "host") else 0
    case = _koszul("", call, form, r, k, ci, ci + rng.randint(1, 10), rng.choice([4, 8, 16, 32]), steps,
                   rng.choice(PRIMES))
    del case["name"]
    # no longer than the listed sequences (the plain form runs at a tenth of the other's rate)
    while case["steps"] > 4 and _work_koszul(case)["flops"] > (5e12 if form == "int8" else 5e11):
        case["steps"] -= case["steps"] // 4
    return case


# ------------------------------------------------------------------ koszul


def _sizes(c):
    return math.comb(c["r"], c["k"]) * c["ci"], math.comb(c["r"], c["k"] - 1) * c["co"]


def _residues(shape, p, gen, low=0):
    return torch.randint(low, p, shape, dtype=torch.int32, device="cuda", generator=gen)


def _maps(c, seed):
    return np.random.default_rng(seed).integers(0, c["p"], (c["r"], c["co"], c["ci"]), dtype=np.uint32)


def _inputs(c, seed):
    """maps, diag, X, Y, Z of a koszul case: canonical residues, the same whatever the call."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n_src, n_tgt = _sizes(c)
    diag = _residues((n_src,), c["p"], gen, 1)
    y = _residues((n_src, c["n"]), c["p"], gen)
    x = _residues((n_src, c["n"]), c["p"], gen) if c["steps"] else None
    z = _residues((n_tgt, c["n"]), c["p"], gen) if c["call"] == "transpose" else None
    return _maps(c, seed), diag, x, y, z


def _engine_args(c, maps, diag):
    return dict(r=c["r"], k=c["k"], dim_in=c["ci"], dim_out=c["co"], prime=c["p"], block_width=c["n"],
                maps=maps, diag=diag, form=c["form"])


def _prepare_koszul(c, seed):
    maps, diag, x, y, z = _inputs(c, seed)
    engine = KoszulEngine(**_engine_args(c, maps, diag))
    st = {"engine": engine, "call": c["call"], "steps": c["steps"], "keep": diag}
    if c["call"] == "host":     # pinned host buffers, as a pipeline that streams sectors keeps them
        st["x"], st["y"] = ((t.cpu().pin_memory()).numpy().view(np.uint32) for t in (x, y))
        seq = torch.empty((c["steps"] + 1, c["n"], c["n"]), dtype=torch.int32).pin_memory()
        last = torch.empty((engine.n_src, c["n"]), dtype=torch.int32).pin_memory()
        st["out"] = (seq.numpy().view(np.uint32), last.numpy().view(np.uint32))
        return st
    st["x"], st["y"], st["z"] = x, y, z
    rows = engine.n_tgt if c["call"] == "forward" else engine.n_src
    st["out"] = torch.empty((rows, c["n"]), dtype=torch.int32, device="cuda")
    if c["call"] == "sequence":
        st["seq"] = torch.empty((c["steps"] + 1, c["n"], c["n"]), dtype=torch.int32, device="cuda")
    return st


def _run_koszul(st):
    engine, call = st["engine"], st["call"]
    if call == "forward":
        engine.forward(st["y"], st["out"])
    elif call == "transpose":
        engine.transpose(st["z"], st["out"])
    elif call == "apply":
        engine.apply(st["y"], st["out"])
    elif call == "host":
        return engine.sequence_host(st["x"], st["y"], st["steps"] + 1, out=st["out"])
    else:
        engine.seq_start(st["x"], st["y"], st["seq"])
        engine.seq_step(st["steps"])
        engine.seq_finish(st["out"])
        return st["seq"], st["out"]
    return st["out"]


def _work_koszul(c):
    """Blocks as 32-bit residues: an application reads Y and writes Z, reads Z and writes S Y; a step's projection
    reads X too.  Two operations a multiply-add."""
    n_src, n_tgt = _sizes(c)
    block = 4 * c["n"]
    pairs = math.comb(c["r"], c["k"] - 1) * (c["r"] - c["k"] + 1)
    half = 2 * pairs * c["ci"] * c["co"] * c["n"]
    once = (n_src + n_tgt) * block
    if c["call"] in ("forward", "transpose"):
        return {"bytes": once, "flops": half}
    if c["call"] == "apply":
        return {"bytes": 2 * once, "flops": 2 * half}
    proj = 2 * n_src * c["n"] * c["n"]
    return {"bytes": c["steps"] * (2 * once + n_src * block), "flops": c["steps"] * (2 * half + proj)}


# ------------------------------------------------------------------- batch


def _batch_cases(c):
    out = []
    for s in c["sectors"].split(";"):
        r, k, ci, co, n = map(int, s.split(","))
        out.append({"call": "sequence", "form": "int8", "r": r, "k": k, "ci": ci, "co": co, "n": n, "p": c["p"],
                    "steps": c["steps"]})
    return out


def _prepare_batch(c, seed):
    specs, xs, ys, seqs, outs = [], [], [], [], []
    for i, s in enumerate(_batch_cases(c)):
        maps, diag, x, y, _ = _inputs(s, seed * 64 + i)
        specs.append(_engine_args(s, maps, diag))
        xs.append(x)
        ys.append(y)
        seqs.append(torch.empty((s["steps"] + 1, s["n"], s["n"]), dtype=torch.int32, device="cuda"))
        outs.append(torch.empty_like(y))
    return {"batch": KoszulBatch(specs), "x": xs, "y": ys, "seq": seqs, "out": outs, "steps": c["steps"]}


def _run_batch(st):
    st["batch"].seq_start(st["x"], st["y"], st["seq"])
    st["batch"].seq_step(st["steps"])
    st["batch"].seq_finish(st["out"])
    return st["seq"], st["out"]


# ------------------------------------------------------------------ cyclic


def _instance_prime(order):
    p = 501
    while p % order != 1 or any(p % f == 0 for f in range(2, int(p ** 0.5) + 1)):
        p += 1
    return p


def _cyclic_weights(genus):
    """Weights with the published instances' blocks: A0 two rows a character; V and A1 two, but one for three of
    them (the characters of mu_w's kernel, shifted by w's weight)."""
    order, n = genus // 2, genus - 3
    a1 = [(2 + j) % order for j in range(n)]
    return order, n, [2] + sorted(a1[1:]), [j // 2 for j in range(genus)], a1


def _cyclic_instance(genus, seed):
    """An instance file's content: random mu with the character grading, a right inverse and a kernel basis of
    mu_w."""
    rng = np.random.default_rng(seed)
    order, n, wv, wa0, wa1 = _cyclic_weights(genus)
    p = _instance_prime(order)
    mu = rng.integers(1, p, (n, n, genus))
    v, a1, a0 = np.array(wv), np.array(wa1), np.array(wa0)
    mu[(v[:, None, None] + a0[None, None, :] - a1[None, :, None]) % order != 0] = 0
    right = np.zeros((genus, n), dtype=np.int64)
    kernel, kernel_weights = [], []
    for q in range(order):
        rows, cols = np.flatnonzero(a1 == (q + wv[0]) % order), np.flatnonzero(a0 == q)
        m = mu[0][np.ix_(rows, cols)]
        if len(rows) == 2:
            while (m[0, 0] * m[1, 1] - m[0, 1] * m[1, 0]) % p == 0:
                m[0, 0] = m[0, 0] % (p - 1) + 1
            mu[0][np.ix_(rows, cols)] = m
            det = pow(int(m[0, 0] * m[1, 1] - m[0, 1] * m[1, 0]) % p, -1, p)
            right[np.ix_(cols, rows)] = np.array([[m[1, 1], -m[0, 1]], [-m[1, 0], m[0, 0]]]) * det % p
        else:
            right[cols[0], rows[0]] = pow(int(m[0, 0]), -1, p)
            column = np.zeros(genus, dtype=np.int64)
            column[cols] = [-m[0, 1] % p, m[0, 0]]
            kernel.append(column)
            kernel_weights.append(q)
    columns, rows_of = _cyclic_sizes(genus)
    return {"genus": genus, "modulus": p, "cyclic": {"order": order},
            "weights": {"V": wv, "A0": wa0, "A1": wa1},
            "artinian": {"mu": {"n": n, "g": genus, "values": mu.reshape(-1).tolist()}},
            "third_section_elimination": {
                "w_V_index": 0, "w_weight": wv[0], "right_inverse_A0_by_A1": right.tolist(),
                "kernel_basis_A0_by_3": np.stack(kernel, axis=1).tolist(), "kernel_weights": kernel_weights,
                "sector_columns": columns, "sector_rows": rows_of}}


def _cyclic_sizes(genus):
    """Columns and rows of the eliminated operator of every sector."""
    order, n, wv, wa0, wa1 = _cyclic_weights(genus)
    m = genus // 2
    subsets = np.zeros((m + 1, order), dtype=np.int64)   # [degree][weight]: subsets of V without w
    subsets[0, 0] = 1
    for w in wv[1:]:
        for d in range(m, 0, -1):
            subsets[d] += np.roll(subsets[d - 1], w)
    kernel = [(c - wv[0]) % order for c in range(order) if wa1.count(c) == 1]

    def pairs(degree, weights, sector):
        return int(sum(subsets[degree][(sector - w) % order] for w in weights))

    columns = [pairs(m, wa0, s) + pairs(m - 1, kernel, (s - wv[0]) % order) for s in range(order)]
    return columns, [pairs(m - 2, wa1, (s - wv[0]) % order) for s in range(order)]


def _prepare_cyclic(c, seed):
    fd, path = tempfile.mkstemp(suffix=".json")
    try:
        with os.fdopen(fd, "w") as f:
            json.dump(_cyclic_instance(c["genus"], seed), f)
        return {"engine": CyclicEngine(path, c["sector"], seed=seed + 1), "moments": 1 + 4 * c["rounds"]}
    finally:
        os.unlink(path)


def _run_cyclic(st):
    st["engine"].generate(st["moments"])
    return st["engine"].download()


def _work_cyclic(c):
    """An application reads and writes the 4-wide 32-bit blocks of the operator's two sides; two operations a
    multiply-add of the two Koszul differentials (blocks of at most two by two) and their transposes."""
    columns, rows = (s[c["sector"]] for s in _cyclic_sizes(c["genus"]))
    n, m = c["genus"] - 4, c["genus"] // 2
    incidences = math.comb(n, m) * m + math.comb(n, m - 1) * (m - 1)
    return {"bytes": 2 * c["rounds"] * 2 * (rows + columns) * 16, "flops": 2 * c["rounds"] * 2 * incidences * 2 * 16}


# ------------------------------------------------------------------- exact


def _neighbours(r, k):
    """For every generator i: ranks of the (k-1)-subsets T without i, of T u {i}, and the sign of i's position."""
    binom = np.array([[math.comb(a, b) for b in range(k + 2)] for a in range(r + 1)], dtype=np.int64)
    subsets = np.array(list(combinations(range(r), k - 1)), dtype=np.int64).reshape(-1, k - 1)
    out = []
    for i in range(r):
        t = np.flatnonzero((subsets != i).all(axis=1))
        s = np.sort(np.concatenate([subsets[t], np.full((len(t), 1), i)], axis=1), axis=1)
        rank = binom[r, k] - 1 - sum(binom[r - 1 - s[:, q], k - q] for q in range(k))
        sign = 1 - 2 * ((subsets[t] < i).sum(axis=1) % 2)
        out.append(tuple(torch.from_numpy(v).cuda() for v in (t, rank, sign)))
    return out


def exact(case, seed):
    """The koszul cases in 64-bit floating point (every sum is below 2^53, so it is exact).  None for the rest:
    their outputs are whole numbers of whole runs (thousands of applications)."""
    c = dict(case)
    if c["kind"] != "koszul" or math.comb(c["r"], c["k"]) > 200_000 or c["steps"] > 200:
        return None
    maps, diag, x, y, z = _inputs(c, seed)
    p, n, r = c["p"], c["n"], c["r"]
    n_src, n_tgt = _sizes(c)
    near = _neighbours(r, c["k"])
    m = torch.from_numpy(maps.astype(np.float64)).cuda()

    def d(v):
        v = v.view(-1, c["ci"], n)
        out = torch.zeros((n_tgt // c["co"], c["co"], n), dtype=torch.float64, device="cuda")
        for i, (t, s, sign) in enumerate(near):
            out[t] += sign[:, None, None] * (m[i] @ v[s])
        return torch.remainder(out, p).view(n_tgt, n)

    def dt(v, scale=True):
        v = v.view(-1, c["co"], n)
        out = torch.zeros((n_src // c["ci"], c["ci"], n), dtype=torch.float64, device="cuda")
        for i, (t, s, sign) in enumerate(near):
            out[s] += sign[:, None, None] * (m[i].T @ v[t])
        return torch.remainder(torch.remainder(out, p).view(n_src, n) * diag[:, None].double(), p)

    whole = lambda v: v.to(torch.int32)  # noqa: E731
    if c["call"] == "forward":
        return whole(d(y.double()))
    if c["call"] == "transpose":
        return whole(dt(z.double()))
    if c["call"] == "apply":
        return whole(dt(d(y.double())))
    cur, xt = y.double(), x.double().T.contiguous()
    moments = []
    for i in range(c["steps"] + 1):
        if i:
            cur = dt(d(cur))
        # at most 2^20 rows a product: partial sums stay below 2^53
        moments.append(torch.remainder(sum(torch.remainder(a @ b, p) for a, b in
                                           zip(xt.split(1 << 20, dim=1), cur.split(1 << 20))), p))
    seq = whole(torch.stack(moments))
    if c["call"] == "host":
        return seq.cpu().numpy().view(np.uint32), whole(cur).cpu().numpy().view(np.uint32)
    return seq, whole(cur)


# ---------------------------------------------------------------- interface


def prepare(case, seed):
    return {"koszul": _prepare_koszul, "batch": _prepare_batch, "cyclic": _prepare_cyclic}[case["kind"]](case, seed)


def run(state):
    if "batch" in state:
        return _run_batch(state)
    return _run_cyclic(state) if "moments" in state else _run_koszul(state)


def work(case):
    if case["kind"] == "koszul":
        return _work_koszul(case)
    if case["kind"] == "cyclic":
        return _work_cyclic(case)
    parts = [_work_koszul(s) for s in _batch_cases(case)]
    return {key: sum(w[key] for w in parts) for key in ("bytes", "flops")}
