"""Performance cases of the overlap hot path, through the public entry points.

A case is one call (or one request mix) as Flye's worker threads, its
read-to-graph stage or a serving loop make it: host arrays of reads in, host
arrays of records out, against an index that stays resident in a context.  The
inputs are seeded synthetic reads of the shapes that ``cuflye_gb300.synth``
names: uniform genomes, HiFi-like reads over a repeat-bearing genome, ONT-like
reads over interspersed repeats, an assembly graph of log-uniform edges, and
a mix of serving requests.  Only their sizes vary from case to case.

Every context runs under a memory budget, as the seam's
``--cuda-memory-budget-bytes`` gives it.
"""

from __future__ import annotations

import ctypes
import math
import random

import numpy as np
import torch

from cuflye_gb300 import abi, synth
from cuflye_gb300.backend import (CuflyeError, OverlapParams, R2GParams, Sequences,
                                  load_library)

BUDGET = 64 << 30

# Read profiles: length distribution (lognormal mean, sd, least, most), error
# rates (substitution, insertion, deletion) and k.
PROFILES = {
    "plain": dict(lengths=(10_000, 5_000, 1_000, 50_000), errors=(0.01, 0.005, 0.005), k=15),
    "hifi": dict(lengths=(15_000, 3_000, 1_000, 100_000), errors=(0.001, 0.0005, 0.0005), k=17),
    "ont": dict(lengths=(25_000, 15_000, 1_000, 150_000), errors=(0.02, 0.02, 0.02), k=17),
    "graph": dict(lengths=(20_000, 12_000, 1_000, 150_000), errors=(0.03, 0.025, 0.025), k=15),
}


def listed() -> list[dict]:
    return [
        # One read a call: Flye's worker threads without batching, where
        # latency and launches count.
        dict(name="overlap_one_read", kind="overlap", profile="plain", genome=1_000_000,
             coverage=20.0, queries=1),
        # A worker's small batch on HiFi reads with repeats, ragged lengths.
        dict(name="overlap_hifi_33", kind="overlap", profile="hifi", genome=2_000_000,
             coverage=40.0, queries=33),
        # The plain overlap stage of a 1 Mb genome, all reads in one call.
        dict(name="overlap_plain_all", kind="overlap", profile="plain", genome=1_000_000,
             coverage=20.0, queries=0),
        # The batched overlap stage of a repeat-bearing 5 Mb genome at 40x.
        dict(name="overlap_hifi_all", kind="overlap", profile="hifi", genome=5_000_000,
             coverage=40.0, queries=0),
        # Noisy long reads over interspersed repeats at 30x, all reads.
        dict(name="overlap_ont_all", kind="overlap", profile="ont", genome=3_000_000,
             coverage=30.0, queries=0),
        # Candidate records of a few reads, as Flye's candidate seam collects
        # them.
        dict(name="candidates_17", kind="candidates", profile="plain", genome=1_000_000,
             coverage=20.0, queries=17),
        # One read of the read-to-graph stage.
        dict(name="graph_one_read", kind="graph", genome=20_000_000, edges=400, queries=1),
        # Read-to-graph alignment of a batch against the full edge set.
        dict(name="graph_3000", kind="graph", genome=20_000_000, edges=400, queries=3000),
        # Candidate chains before the divergence filter, for a replay payload.
        dict(name="graph_chains_250", kind="chains", genome=5_000_000, edges=101, queries=250),
        # Building the resident index of a read set, and the first batch on it.
        dict(name="index_plain", kind="index", profile="plain", genome=2_000_000, coverage=20.0,
             queries=64),
        # A burst of single-read serving requests, 1-100 kb, two workers.
        dict(name="serving_burst_200", kind="serving", genome=16_000_000, queries=200),
        # The segmented sort on its own: ragged segments with equal keys.
        dict(name="sort_segments", kind="sort", elements=2_000_003, segments=611, distinct=0.7),
    ]


def _log_uniform(rng: random.Random, lo: float, hi: float) -> float:
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["overlap"] * 6 + ["candidates", "graph", "graph", "chains", "index",
                                         "serving", "sort"])
    if kind in ("overlap", "candidates", "index"):
        profile = rng.choice(["plain", "hifi", "ont"])
        if kind == "candidates":
            profile = rng.choice(["plain", "ont"])
        most = {"plain": 4e6, "hifi": 5e6, "ont": 3e6}[profile]
        genome = int(_log_uniform(rng, 2e5, 2e6 if kind == "index" else most))
        coverage = round(rng.uniform(10.0, 30.0 if profile == "ont" else 40.0), 1)
        reads = genome * coverage / PROFILES[profile]["lengths"][0]
        if kind == "overlap":
            # from one read to all of them
            queries = int(_log_uniform(rng, 1, 1.3 * reads))
            queries = 0 if queries > 0.8 * reads else queries
        else:
            queries = int(_log_uniform(rng, 1, min(reads, 17 if kind == "candidates" else 64)))
        return dict(kind=kind, profile=profile, genome=genome, coverage=coverage, queries=queries)
    if kind in ("graph", "chains"):
        genome = int(_log_uniform(rng, 5e5, 2e7))
        return dict(kind=kind, genome=genome, edges=max(5, int(genome / rng.uniform(3e4, 8e4))),
                    queries=int(_log_uniform(rng, 1, 3000)))
    if kind == "serving":
        return dict(kind=kind, genome=int(rng.uniform(4e6, 16e6)),
                    queries=int(_log_uniform(rng, 8, 200)))
    return dict(kind="sort", elements=int(_log_uniform(rng, 1e3, 2e6)),
                segments=int(_log_uniform(rng, 1, 600)), distinct=round(rng.uniform(0.3, 2.0), 2))


# ---------------------------------------------------------------- inputs


def _sample_reads(rng: np.random.Generator, genome: np.ndarray, lengths: np.ndarray,
                  errors) -> Sequences:
    """Reads of the given lengths from uniform positions and strands, with
    uniform substitutions, insertions and deletions; ids 1..n."""
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(rng.integers(0, 2**62)))
    n = len(lengths)
    start = torch.from_numpy(rng.integers(0, len(genome) - lengths + 1)).to(dev)
    rev = torch.from_numpy(rng.random(n) < 0.5).to(dev)
    ln = torch.from_numpy(lengths).to(dev)
    offs = torch.zeros(n + 1, dtype=torch.int64, device=dev)
    offs[1:] = torch.cumsum(ln, 0)
    total = int(offs[-1])
    code = np.zeros(256, dtype=np.uint8)
    code[synth.BASES] = np.arange(4, dtype=np.uint8)
    g = torch.from_numpy(code[genome]).to(dev)
    read = torch.repeat_interleave(torch.arange(n, device=dev), ln, output_size=total)
    at = torch.arange(total, device=dev) - offs[read]
    r = rev[read]
    b = g[start[read] + torch.where(r, ln[read] - 1 - at, at)]
    b = torch.where(r, 3 - b, b)
    del read, at, r
    sub, ins, dele = errors
    u = torch.rand(total, device=dev, generator=gen)
    shift = torch.randint(1, 4, (total,), device=dev, generator=gen, dtype=torch.uint8)
    b = torch.where(u < sub, (b + shift) & 3, b)
    u = torch.rand(total, device=dev, generator=gen)
    insert = (u >= dele) & (u < dele + ins)
    reps = (u >= dele).to(torch.int64) + insert.to(torch.int64)
    ends = torch.cumsum(reps, 0)
    out = torch.repeat_interleave(b, reps)
    where = ends[insert] - 1  # an inserted base follows its anchor
    out[where] = torch.randint(0, 4, (len(where),), device=dev, generator=gen, dtype=torch.uint8)
    noffs = torch.zeros(n + 1, dtype=torch.int64, device=dev)
    noffs[1:] = ends[offs[1:] - 1]
    bases = torch.from_numpy(synth.BASES.copy()).to(dev)[out.to(torch.int64)].cpu().numpy()
    noffs = noffs.cpu().numpy()
    del u, shift, insert, reps, ends, out, where, b, g
    torch.cuda.empty_cache()
    return Sequences(np.arange(1, n + 1, dtype=np.int64), noffs, bases)


def _lengths_for(rng, total: float, profile: dict, longest: int) -> np.ndarray:
    mean, sd, lo, hi = profile["lengths"]
    v = synth.lognormal_lengths(rng, int(1.2 * total / mean) + 64, mean, sd, lo, hi)
    v = np.minimum(v, longest)
    return v[np.cumsum(v) <= total + v[0]]


def _pick(reads: Sequences, queries: int) -> Sequences:
    """`queries` reads spread evenly over the set (0: all of them)."""
    if queries <= 0 or queries >= reads.n:
        return reads
    idx = (np.arange(queries) * reads.n) // queries + reads.n // (2 * queries)
    parts = [reads.bases[reads.offsets[i]:reads.offsets[i + 1]] for i in idx]
    offs = np.zeros(queries + 1, dtype=np.int64)
    offs[1:] = np.cumsum([len(p) for p in parts])
    return Sequences(reads.ids[idx].copy(), offs, np.concatenate(parts))


def _ont_genome(rng: np.random.Generator, length: int) -> np.ndarray:
    """Uniform bases with 10 % interspersed repeats: families of 1-20 kb,
    copies at 0.5-5 % divergence."""
    genome = synth.random_genome(rng, length)
    placed = 0
    while placed < 0.10 * length:
        family = synth.random_genome(rng, int(rng.integers(1_000, 20_001)))
        for _ in range(int(rng.integers(2, 10))):
            at = int(rng.integers(0, length - len(family)))
            copy = synth.mutate(rng, family, float(rng.uniform(0.005, 0.05)))
            genome[at:at + len(copy)] = copy
            placed += len(copy)
    return genome


def _read_set(case: dict, rng: np.random.Generator) -> Sequences:
    prof = PROFILES[case["profile"]]
    n = case["genome"]
    if case["profile"] == "hifi":
        genome = synth.repeat_genome(rng, n, 5_000, max(2, n // 166_667), 0.01, 0.02)
    elif case["profile"] == "ont":
        genome = _ont_genome(rng, n)
    else:
        genome = synth.random_genome(rng, n)
    lengths = _lengths_for(rng, case["coverage"] * n, prof, n)
    return _sample_reads(rng, genome, lengths, prof["errors"])


def _frequencies(case: dict) -> tuple[int, int]:
    c = case["coverage"]
    least = max(2, int(round(c / 10))) if case["profile"] == "ont" else 2
    return least, int(5 * c)


def _graph_inputs(case: dict, rng: np.random.Generator):
    """A genome cut into edges of log-uniform lengths, a tenth of them
    duplicated at 0.5 % divergence, and ONT-like reads over it."""
    n, ne = case["genome"], case["edges"]
    genome = synth.random_genome(rng, n)
    raw = np.exp(rng.uniform(np.log(5_000), np.log(500_000), size=ne))
    cuts = np.concatenate([[0], np.cumsum(raw / raw.sum() * n).astype(np.int64)])
    cuts[-1] = n
    seqs = [genome[cuts[i]:cuts[i + 1]] for i in range(ne)]
    left, right = list(range(0, 2 * ne, 2)), list(range(2, 2 * ne + 2, 2))
    for d in sorted(rng.choice(ne, size=max(1, ne // 10), replace=False)):
        seqs.append(synth.mutate(rng, seqs[d], 0.005))
        left.append(left[d])
        right.append(right[d])
    ids = np.arange(1, len(seqs) + 1, dtype=np.int64)
    offs = np.zeros(len(seqs) + 1, dtype=np.int64)
    offs[1:] = np.cumsum([len(s) for s in seqs])
    prof = PROFILES["graph"]
    mean, sd, lo, hi = prof["lengths"]
    lengths = np.minimum(synth.lognormal_lengths(rng, case["queries"], mean, sd, lo, hi), n)
    reads = _sample_reads(rng, genome, lengths, prof["errors"])
    return Sequences(ids, offs, np.concatenate(seqs)), left, right, reads


class Context:
    """A context of the C ABI; closed with the state that holds it."""

    def __init__(self):
        self.lib = load_library()
        self.handle = ctypes.c_void_p()
        status = self.lib.cuflye_open(0, BUDGET, ctypes.byref(self.handle))
        if status:
            raise CuflyeError(status, self.lib.cuflye_last_error(None).decode())

    def call(self, name: str, *args) -> None:
        status = getattr(self.lib, name)(self.handle, *args)
        if status:
            raise CuflyeError(status, self.lib.cuflye_last_error(self.handle).decode())

    def build_index(self, targets: Sequences, k: int, min_freq: int, max_freq: int) -> dict:
        self.call("cuflye_index_build", k, *_sequences(targets), min_freq, max_freq)
        counts = [ctypes.c_uint64() for _ in range(3)]
        self.call("cuflye_index_stats", *map(ctypes.byref, counts))
        return {n: c.value for n, c in zip(("keys", "positions", "repetitive"), counts)}

    def __del__(self):
        if self.handle:
            self.lib.cuflye_close(self.handle)


class Server:
    """A serving loop over a context's index (the context stays open)."""

    def __init__(self, owner: Context, params: OverlapParams, workers: int, batch_bases: int):
        self.owner, self.params = owner, params
        self.handle = ctypes.c_void_p()
        owner.call("cuflye_server_open", workers, ctypes.byref(params), batch_bases,
                   ctypes.byref(self.handle))

    def check(self, status: int) -> None:
        if status:
            message = self.owner.lib.cuflye_server_last_error(self.handle)
            raise CuflyeError(status, message.decode())

    def submit(self, request: Sequences) -> int:
        ticket = ctypes.c_uint64()
        self.check(self.owner.lib.cuflye_submit(self.handle, *_sequences(request),
                                                ctypes.byref(ticket)))
        return ticket.value

    def wait(self, ticket: int, rows: np.ndarray) -> int:
        n = ctypes.c_size_t()
        self.check(self.owner.lib.cuflye_poll(self.handle, ticket, -1, rows.ctypes.data,
                                              len(rows), ctypes.byref(n)))
        return n.value

    def __del__(self):
        if self.handle:
            self.owner.lib.cuflye_server_close(self.handle)


def _pointer(a: np.ndarray, kind):
    return a.ctypes.data_as(ctypes.POINTER(kind))


def _sequences(s: Sequences) -> tuple:
    """The leading arguments of a call on reads."""
    return (s.n, _pointer(s.ids, ctypes.c_int64), _pointer(s.offsets, ctypes.c_int64),
            s.bases.ctypes.data_as(ctypes.c_char_p))


def _buffer(n: int, dtype, pinned: bool = False) -> np.ndarray:
    """A caller-owned output buffer, zeroed (page-locked on request)."""
    t = torch.zeros(max(n, 1) * dtype.itemsize, dtype=torch.uint8, pin_memory=pinned)
    return t.numpy().view(dtype)


def _row_capacity(case: dict) -> int:
    """Room for 256 overlap rows a read, as the binding's default."""
    reads = case["queries"]
    if not reads:
        mean = PROFILES[case["profile"]]["lengths"][0]
        reads = int(1.2 * case["genome"] * case["coverage"] / mean) + 64
    return 256 * max(reads, 4)


def prepare(case: dict, seed: int) -> dict:
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    state = {"kind": kind}
    ctx = state["context"] = Context()
    if kind == "sort":
        n, ns = case["elements"], case["segments"]
        cuts = np.sort(rng.integers(0, n + 1, size=ns - 1))
        state["offsets"] = np.concatenate([[0], cuts, [n]]).astype(np.uint64)
        # keys as the path's: a target id above a position, drawn from about
        # `distinct` values per element of an average segment
        most = max(1, int(case["distinct"] * n / ns / 64))
        state["keys"] = ((rng.integers(0, 64, size=n).astype(np.uint64) << np.uint64(32)) |
                         rng.integers(0, most, size=n).astype(np.uint64))
        state["values"] = rng.integers(0, 2**31, size=n).astype(np.uint32)
        state["out"] = (np.empty_like(state["keys"]), np.empty_like(state["values"]))
        return state
    if kind == "serving":
        sw = synth.serving_workload(seed=seed, genome_len=case["genome"],
                                    n_queries=case["queries"])
        q = sw.queries
        state["requests"] = [
            Sequences(q.ids[i:i + 1].copy(),
                      np.array([0, q.offsets[i + 1] - q.offsets[i]], dtype=np.int64),
                      q.bases[q.offsets[i]:q.offsets[i + 1]].copy()) for i in range(q.n)]
        ctx.build_index(Sequences.of(sw.targets), sw.k, sw.min_freq, sw.max_freq)
        state["server"] = Server(ctx, OverlapParams.make(**sw.params), 2, 32_000_000)
        state["rows"] = _buffer(1024 * q.n + 8192, abi.OVERLAP_DTYPE)
        return state
    if kind in ("graph", "chains"):
        edges, left, right, reads = _graph_inputs(case, rng)
        ctx.build_index(edges, 15, 1, 64)
        lft, rgt = np.array(left, dtype=np.int32), np.array(right, dtype=np.int32)
        ctx.call("cuflye_graph_set", edges.n, _pointer(edges.ids, ctypes.c_int64),
                 _pointer(edges.ids, ctypes.c_int64), _pointer(lft, ctypes.c_int32),
                 _pointer(rgt, ctypes.c_int32))
        state["reads"] = reads
        state["params"] = OverlapParams.make(**dict(synth.OVERLAP_PARAMS, kmer_size=15,
                                                    min_overlap=100, check_overhang=0,
                                                    max_overhang=0, only_max_ext=0))
        state["r2g"] = R2GParams.make(**synth.R2G_PARAMS)
        dtype = abi.READ_ALIGNMENT_DTYPE if kind == "graph" else abi.CHAIN_RECORD_DTYPE
        state["rows"] = _buffer(max(1024, 64 * case["queries"]), dtype)
        state["inputs"] = np.zeros(case["queries"], dtype=np.uint64)
        return state
    reads = _read_set(case, rng)
    prof = PROFILES[case["profile"]]
    least, most = _frequencies(case)
    state["queries"] = _pick(reads, case["queries"])
    state["params"] = OverlapParams.make(**dict(synth.OVERLAP_PARAMS, kmer_size=prof["k"]))
    if kind == "index":
        state["build"] = (reads, prof["k"], least, most)
    else:
        ctx.build_index(reads, prof["k"], least, most)
    if kind == "candidates":
        # room for the expected records of one call and half as many again
        survive = (1 - sum(prof["errors"])) ** prof["k"]
        bases = (case["queries"] + 6) * prof["lengths"][0]
        n = int(bases * (1.6 * case["coverage"] * survive**2 + 2))
        state["rows"] = _buffer(n, abi.CANDIDATE_DTYPE)
        state["filtered"] = _buffer(bases, abi.FILTERED_DTYPE)
        return state
    # the whole read set streams through page-locked buffers
    whole = not case["queries"]
    state["rows"] = _buffer(_row_capacity(case), abi.OVERLAP_DTYPE, pinned=whole)
    if whole:
        q = state["queries"]
        bases = _buffer(len(q.bases), np.dtype(np.uint8), pinned=True)
        bases[:] = q.bases
        state["queries"] = Sequences(q.ids, q.offsets, bases)
    return state


# ------------------------------------------------------------------ run


def _columns(rows: np.ndarray) -> dict:
    """A record array's columns."""
    return {f: rows[f].view(np.int64) if rows.dtype[f] == np.uint64 else rows[f]
            for f in rows.dtype.names if f != "reserved"}


def run(state: dict):
    """One call; the program's own output buffers come back whole, with the
    number of records in them."""
    kind, ctx = state["kind"], state["context"]
    n = ctypes.c_size_t()
    if kind == "sort":
        keys, values = state["out"]
        np.copyto(keys, state["keys"])
        np.copyto(values, state["values"])
        ctx.call("cuflye_std_sort_segments", _pointer(keys, ctypes.c_uint64),
                 _pointer(values, ctypes.c_uint32), _pointer(state["offsets"], ctypes.c_uint64),
                 len(state["offsets"]) - 1)
        return {"keys": keys.view(np.int64), "values": values.view(np.int32)}
    rows = state["rows"]
    if kind == "serving":
        server = state["server"]
        tickets = [server.submit(r) for r in state["requests"]]
        counts, at = [], 0
        for t in tickets:
            counts.append(server.wait(t, rows[at:]))
            at += counts[-1]
        return {"counts": np.array(counts), "rows": _columns(rows)}
    if kind == "candidates":
        nf = ctypes.c_size_t()
        filtered = state["filtered"]
        ctx.call("cuflye_candidates", *_sequences(state["queries"]), rows.ctypes.data, len(rows),
                 ctypes.byref(n), filtered.ctypes.data, len(filtered), ctypes.byref(nf))
        return {"n": n.value, "n_filtered": nf.value, "rows": _columns(rows),
                "filtered": _columns(filtered)}
    if kind == "graph":
        ctx.call("cuflye_read_to_graph", *_sequences(state["reads"]),
                 ctypes.byref(state["params"]), ctypes.byref(state["r2g"]), rows.ctypes.data,
                 len(rows), ctypes.byref(n))
        return {"n": n.value, "rows": _columns(rows)}
    if kind == "chains":
        ctx.call("cuflye_read_to_graph_chains", *_sequences(state["reads"]),
                 ctypes.byref(state["params"]), ctypes.byref(state["r2g"]), rows.ctypes.data,
                 len(rows), ctypes.byref(n), _pointer(state["inputs"], ctypes.c_uint64))
        return {"n": n.value, "inputs": state["inputs"].view(np.int64), "rows": _columns(rows)}
    stats = ctx.build_index(*state["build"]) if kind == "index" else {}
    ctx.call("cuflye_overlaps", *_sequences(state["queries"]), ctypes.byref(state["params"]),
             rows.ctypes.data, len(rows), ctypes.byref(n))
    return {**stats, "n": n.value, "rows": _columns(rows)}


def work(case: dict) -> dict:
    """Compulsory bytes: the ASCII bases in, a 16-byte table entry per k-mer
    window, 8 bytes per bucket entry hit (the expected number: coverage times
    the chance that both copies of a k-mer are free of errors) and the
    records out.  Index builds: the bases in, the positions and table out.
    Integer work only, so no floating-point operations are counted."""
    kind = case["kind"]
    if kind == "sort":
        return {"bytes": 24.0 * case["elements"], "flops": 0.0}
    if kind == "serving":
        bases = case["queries"] * 99_000 / math.log(100)
        survive = 0.5 * 0.99**15 + 0.5 * 0.92**15
        return {"bytes": bases * (1 + 16 + 8 * survive) + 64.0 * case["queries"], "flops": 0.0}
    if kind in ("graph", "chains"):
        bases = 20_000.0 * case["queries"]
        return {"bytes": bases * (1 + 16 + 8 * 1.1 * 0.92**15) + 128.0 * case["queries"],
                "flops": 0.0}
    prof = PROFILES[case["profile"]]
    mean, rate, k = prof["lengths"][0], sum(prof["errors"]), prof["k"]
    all_bases = case["genome"] * case["coverage"]
    bases = mean * case["queries"] if case["queries"] else all_bases
    bases = min(bases, all_bases)
    survive = (1 - rate) ** k
    hits = bases * survive * case["coverage"] * survive
    rows = 2.0 * case["coverage"] * bases / mean
    if kind == "candidates":
        return {"bytes": bases * 17 + 40.0 * hits, "flops": 0.0}
    total = bases * 17 + 8.0 * hits + 56.0 * rows
    if kind == "index":
        keys = case["genome"] + all_bases * (1 - survive)
        total += all_bases + 8.0 * all_bases * survive + 16.0 * keys
    return {"bytes": total, "flops": 0.0}


def exact(case: dict, seed: int):
    """Records are integers throughout; their one float column, the k-mer
    divergence, follows from each chain's match count, which takes the whole
    chaining to recompute: far over the time given on the host."""
    return None
