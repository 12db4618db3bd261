"""Workloads of the alignment engine for timing and for comparing two builds of it.

A case is a dict of plain values:

* kind "pairs": one batch of query/target pairs through one extension engine, resident in
  HBM (`phr_extend_batch_device`, where a caller keeps its sequences on the device) or
  from host buffers (`Engine.extend_packed`, the shape of the reference's own calls).
* kind "reads": `align_read` for a batch of reads against a target index, host buffers in
  and out (`Engine.align_packed`, with variant observations `Engine.align_packed_variants`).

Sequences follow the repository's own workloads (phraya_b200.datagen / casegen): i.i.d.
ACGT with substitutions and short indels, protein over the 20 residues with substitutions.
One `Engine` serves every case of the process, as a program keeps one context.
"""
import ctypes as C
import math

import numpy as np
import torch

from phraya_b200 import _abi as A
from phraya_b200 import api as P
from phraya_b200 import casegen as G
from phraya_b200 import datagen as D
from phraya_b200.batch import PackedReads

ENGINES = {"linear": A.ENGINE_WFA_LINEAR, "affine": A.ENGINE_WFA_AFFINE, "myers": A.ENGINE_MYERS_GLOBAL,
           "myers_fit": A.ENGINE_MYERS_FIT}
STRATEGIES = {"fast": A.FAST, "balanced": A.BALANCED, "sensitive": A.SENSITIVE}
AMINO = torch.tensor(list(G.AMINO_ACIDS.encode()), dtype=torch.uint8)


def _pairs(name, engine, n, lo, hi, div, where="device", alphabet="dna", log=False, tail=0.0, costs=(2, 4, 1)):
    return {"name": name, "kind": "pairs", "engine": engine, "n": n, "lo": lo, "hi": hi, "div": div, "where": where,
            "alphabet": alphabet, "log": log, "tail": tail, "mismatch": costs[0], "gap_open": costs[1],
            "gap_extend": costs[2]}


def _reads(name, n, genome, strategy, length=150, error=0.0105, variants=False):
    """length 150..500: reads of that length; 0: long reads, lognormal around 8 kb."""
    return {"name": name, "kind": "reads", "n": n, "genome": genome, "strategy": strategy, "length": length,
            "error": error, "variants": variants}


def listed():
    return [
        # one call per pair, as the reference's wfa_extend_affine is called: latency and launches
        _pairs("one_pair", "affine", 1, 150, 150, 0.02, where="host"),
        # the batched extension microbench: 100-300 bp at 0-5 % divergence, affine costs 4/6/2 ...
        _pairs("pairs_affine", "affine", 1_000_000, 100, 300, 0.05, costs=(4, 6, 2)),
        # ... and linear
        _pairs("pairs_linear", "linear", 1_000_000, 100, 300, 0.05),
        # edit distance + CIGAR of pairs from 64 bp to 2 kb, the microbench's Myers set
        _pairs("pairs_myers", "myers", 1_000_000, 64, 2048, 0.05, log=True),
        # short-read windows under the fitting mode: the target runs on past the alignment's end
        _pairs("windows_myers_fit", "myers_fit", 200_000, 100, 300, 0.05, tail=0.5),
        # 5,000 protein pairs of 200-800 residues at 30 % substitutions (byte comparisons)
        _pairs("protein_linear", "linear", 5_000, 200, 800, 0.30, alphabet="protein"),
        # long reads against their windows, linear gaps (what balanced align_read extends)
        _pairs("long_linear", "linear", 500, 4_000, 16_000, 0.10),
        # the same under affine gaps (what sensitive align_read extends)
        _pairs("long_affine", "affine", 200, 4_000, 16_000, 0.10),
        # one read per call, the shape of the reference's align_read: latency and launches
        _reads("one_read", 1, 1_000_000, "balanced"),
        # 20,000 reads of 150 bp on a 1 Mbp genome in one call
        _reads("reads_balanced", 20_000, 1_000_000, "balanced"),
        # the same reads under the sensitive strategy (affine gaps, up to 50 chains)
        _reads("reads_sensitive", 20_000, 1_000_000, "sensitive"),
        # long noisy reads on a 5 Mbp genome with repeats: long chains, long extensions
        _reads("reads_long", 1_000, 5_000_000, "balanced", length=0, error=0.05),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: any of the listed kinds at another size, divergence or option."""
    kind = rng.choice(["short", "short", "myers", "fit", "protein", "long", "host", "reads", "reads", "long_reads"])
    engine = rng.choice(["linear", "affine"])
    costs = rng.choice([(2, 4, 1), (4, 6, 2)])
    div = round(rng.uniform(0.005, 0.05), 4)
    if kind == "short":
        c = _pairs("", engine, _log_int(rng, 300, 900_000), rng.randint(60, 120), rng.randint(150, 420), div,
                   costs=costs)
    elif kind == "myers":
        c = _pairs("", "myers", _log_int(rng, 300, 900_000), rng.randint(33, 128), rng.randint(200, 2047), div,
                   log=True)
    elif kind == "fit":
        c = _pairs("", "myers_fit", _log_int(rng, 100, 200_000), rng.randint(60, 140), rng.randint(150, 500), div,
                   tail=round(rng.uniform(0.05, 0.9), 2))
    elif kind == "protein":
        c = _pairs("", rng.choice(["linear", "affine", "myers"]), _log_int(rng, 50, 5_000), rng.randint(100, 250),
                   rng.randint(300, 800), round(rng.uniform(0.1, 0.3), 3), alphabet="protein")
    elif kind == "long":
        c = _pairs("", engine, _log_int(rng, 5, 180), rng.randint(2_500, 5_000), rng.randint(6_000, 16_000),
                   round(rng.uniform(0.02, 0.10), 3), costs=costs)
    elif kind == "host":
        c = _pairs("", rng.choice(["linear", "affine", "myers", "myers_fit"]), _log_int(rng, 2, 60_000),
                   rng.randint(60, 120), rng.randint(150, 420), div, where="host")
    elif kind == "reads":
        c = _reads("", _log_int(rng, 2, 19_000), rng.choice([300_007, 1_000_000, 2_000_003]),
                   rng.choice(["fast", "balanced", "sensitive"]), length=rng.randint(75, 301),
                   error=round(rng.uniform(0.002, 0.02), 4), variants=rng.random() < 0.4)
    else:
        c = _reads("", _log_int(rng, 3, 900), 5_000_000, "balanced", length=0, error=round(rng.uniform(0.02, 0.06), 3))
    del c["name"]
    return c


_shared = {}


def _engine():
    """The process's one device context."""
    if "engine" not in _shared:
        _shared["engine"] = P.Engine(torch.cuda.current_device())
    return _shared["engine"]


def _protein_device(n, lo, hi, div, seed):
    """Pairs over the 20 residues: each target its query with substitutions at `div`."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    ln = torch.randint(lo, hi + 1, (n,), generator=g, device="cuda")
    total = int(ln.sum().item())
    res = torch.randint(0, 20, (total,), generator=g, device="cuda")
    sub = torch.rand(total, generator=g, device="cuda") < div
    alt = (res + torch.randint(1, 20, (total,), generator=g, device="cuda")) % 20
    table = AMINO.cuda()
    seq = torch.cat([table[res], table[torch.where(sub, alt, res)], torch.zeros(64, dtype=torch.uint8, device="cuda")])
    off = torch.zeros(n, dtype=torch.long, device="cuda")
    off[1:] = torch.cumsum(ln, 0)[:-1]
    return {"seq": seq, "q_off": off.to(torch.uint64), "q_len": ln.to(torch.uint32),
            "t_off": (off + total).to(torch.uint64), "t_len": ln.to(torch.uint32), "n": n, "seq_bytes": 2 * total}


def _pair_inputs(c, seed):
    if c["alphabet"] == "protein":
        return _protein_device(c["n"], c["lo"], c["hi"], c["div"], seed)
    d = D.extension_pairs_device(c["n"], c["lo"], c["hi"], c["div"], seed=seed, log_uniform=c["log"])
    if c["tail"]:
        # a window that runs on past the alignment's end: the next pair's query bytes follow
        t = d["t_len"].to(torch.int64)
        q = d["q_len"].to(torch.int64)
        more = torch.zeros_like(t)
        more[:-1] = torch.minimum((q[:-1] * c["tail"]).long(), q[1:])
        d["t_len"] = (t + more).to(torch.uint32)
    return d


def prepare(case, seed):
    c = dict(case)
    eng = _engine()
    if c["kind"] == "reads":
        if c["length"]:
            genome = D.random_reference(c["genome"], seed=seed)
            rng = np.random.default_rng([seed, 1])
            packed, _, _ = G.reads_from_genome(genome, np.full(c["n"], c["length"]), rng, c["error"], 0.95, 3)
        else:
            genome = G.repeat_reference(c["genome"], 20, seed=seed)
            packed, _, _ = G.long_reads(genome, c["n"], seed=seed + 1, error=c["error"])
        return {"c": c, "eng": eng, "index": eng.index(genome), "reads": packed}
    d = _pair_inputs(c, seed)
    if c["where"] == "host":
        packed = D.to_packed(d)
        return {"c": c, "eng": eng, "pairs": packed}
    b = A.PairBatch()
    b.n_pairs = d["n"]
    b.seq, b.seq_bytes = d["seq"].data_ptr(), d["seq_bytes"]
    b.q_off, b.q_len = d["q_off"].data_ptr(), d["q_len"].data_ptr()
    b.t_off, b.t_len = d["t_off"].data_ptr(), d["t_len"].data_ptr()
    b.q_seed = b.t_seed = None
    cap = _cigar_room(c)
    aln = torch.zeros((d["n"], 10), dtype=torch.int32, device="cuda")  # phr_alignment: ten 32-bit words
    cigar = torch.zeros(cap, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()  # the engine launches on its own stream
    return {"c": c, "eng": eng, "inputs": d, "batch": b, "aln": aln, "cigar": cigar, "cap": cap}


def _cigar_room(c):
    """CIGAR bytes to hold a case's results, whatever the seed: about 6 characters an edit
    and one edit per `div` / 2 bases (protein: per `div`), with room to spare."""
    if c["kind"] == "reads":
        longest = c["length"] or 50_000
        mean = c["length"] or 8000 * math.exp(0.125)
        return int(c["n"] * (128 + 16 * c["error"] * mean)) + 12 * longest
    return int(c["n"] * (128 + 8 * c["div"] * _mean_len(c))) + 12 * c["hi"]


def _room(values, rows):
    """`values` at the front of an array of `rows` rows (how many there are depends on the seed)."""
    if len(values) > rows:
        raise RuntimeError("%d rows of results, room for %d" % (len(values), rows))
    out = np.zeros((rows,) + values.shape[1:], dtype=values.dtype)
    out[:len(values)] = values
    return out


def _costs(c):
    return c["mismatch"], c["gap_open"], c["gap_extend"]


def _alignments(aln):
    """phr_alignment records as an array of their 32-bit words."""
    return np.ascontiguousarray(aln).view(np.uint32).reshape(len(aln), 10)


def run(state):
    c, eng = state["c"], state["eng"]
    if c["kind"] == "reads":
        args = (state["index"], state["reads"], STRATEGIES[c["strategy"]], A.GAP_AFFINE)
        if c["variants"]:
            rr, aln, cig, stats, off, var, cov, al = eng.align_packed_variants(*args)
        else:
            rr, aln, cig, stats = eng.align_packed(*args)
        n = c["n"]
        out = {"outcome": rr["outcome"], "has_result": rr["has_result"], "reverse": rr["reverse"],
               "n_aln": rr["n_aln"], "aln_off": rr["aln_off"].astype(np.int64),
               "alignments": _room(_alignments(aln), 4 * n + 64), "cigar": _room(cig, _cigar_room(c)),
               "stats": np.array(stats)}
        if c["variants"]:
            rows = int(n * (16 + 4 * c["error"] * c["length"])) + 64
            whole = np.ascontiguousarray(var).view(np.uint32).reshape(len(var), 16)
            out.update(variant_off=off.astype(np.int64),
                       variants=_room(whole[:, [0, 1, 2, 3, 8, 9, 10, 11, 12, 13, 14]], rows),
                       confidence=_room(var["confidence"], rows), uniqueness=_room(var["kmer_uniqueness"], rows),
                       coverage=_room(cov, 301 * rows), allele_base=_room(al["base"], 2 * rows),
                       allele_count=_room(al["count"], 2 * rows))
        return out
    if c["where"] == "host":
        aln, cig = eng.extend_packed(ENGINES[c["engine"]], state["pairs"], P.AffineCosts(*_costs(c)))
        return {"alignments": _alignments(aln), "cigar": _room(cig, _cigar_room(c))}
    arena = A.ResultArena(state["aln"].data_ptr(), state["cigar"].data_ptr(), state["cap"], 0)
    eng.check(eng._lib.phr_extend_batch_device(eng.handle, ENGINES[c["engine"]], C.byref(state["batch"]),
                                               A.AffineCosts(*_costs(c)), C.byref(arena)))
    return {"alignments": state["aln"], "cigar": state["cigar"]}


def exact(case, seed):
    """Results are whole numbers and text; a variant's two real numbers follow from its
    alignment, which plain arithmetic over the inputs does not give."""
    return None


def _mean_len(c):
    lo, hi = c["lo"], c["hi"]
    return (hi - lo) / math.log(hi / lo) if c["log"] and hi > lo else (lo + hi) / 2.0


def work(case):
    """Bytes: the sequences and offsets in, the records and CIGAR text out. "flops" counts
    integer operations: a wavefront diagonal of a linear / affine score step is 10 / 30
    operations and a 16-base compare 4; a 32-row word of a Myers column is 22, over a band
    as wide as the distance."""
    c = case
    if c["kind"] == "reads":
        mean = c["length"] or 8000 * math.exp(0.125)
        dist = c["error"] * mean * (1.0 if c["length"] else 1.6)
        per_in, per_out = mean + 12, 24 + 40 + 4 * dist
        step = 30.0 if c["strategy"] == "sensitive" else 10.0
        # both strands sketched (about 20 operations a base), one placement extended
        ops = 40 * mean + (step * dist * dist + 4 * mean / 16 if not c["length"] or step == 30.0
                           else 22.0 * mean * max(1.0, mean / 32.0))
        return {"bytes": c["n"] * (per_in + per_out), "flops": c["n"] * ops}
    mean = _mean_len(c)
    protein = c["alphabet"] == "protein"
    dist = mean * (c["div"] if protein else c["div"] / 2 * 1.6)
    per_in = 2 * mean + c["tail"] * mean + 24
    per_out = 40 + min(4 * dist + 4, 2 * mean)
    if c["engine"] in ("myers", "myers_fit"):
        rows = mean if c["engine"] == "myers_fit" else min(mean, 2 * dist + 32)
        ops = 22.0 * mean * (1 + c["tail"]) * rows / 32.0
    elif c["engine"] == "affine":
        # the score of an edit is its mismatch or gap cost; reachable scores step by their common divisor
        score = dist * c["mismatch"] / (math.gcd(c["mismatch"], math.gcd(c["gap_open"] + c["gap_extend"],
                                                                         c["gap_extend"])))
        ops = 30.0 * score * max(1.0, score / 2) + 4 * mean / 16
    else:
        ops = 10.0 * dist * dist + 4 * mean / 16
    return {"bytes": c["n"] * (per_in + per_out), "flops": c["n"] * ops}
