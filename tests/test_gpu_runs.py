"""GPU: the run path (hits found, sorted and chained as runs, the default on a
built index of an odd k) against the hit path and the oracle, row for row,
divergence bits included.  The cases put run and tile edges everywhere: reads
of every length around the 32-window tiles, reads that end at a target's ends,
tandem arrays (equal positions at every sort point, split runs, groups and
queries left to the hit path), long targets out of ext order and noisy reads."""

import numpy as np
import pytest

from test_gpu_parity import oracle_index, overlap_tuples_gpu, overlap_tuples_oracle

pytestmark = pytest.mark.gpu

VARIANTS = ({}, {"only_max_ext": 0}, {"only_max_ext": 0, "check_overhang": 0, "min_overlap": 100},
            {"max_overlaps": 3}, {"max_jump": 40, "max_gap": 10})


def _check(gpu, oracle_mod, targets, queries, k, min_freq, max_freq, params, variants=VARIANTS):
    from cuflye_gb300.backend import OverlapParams
    oracle_mod.set_stable(False)
    idx, _ = oracle_index(oracle_mod, targets, k, min_freq, max_freq)
    gpu.build_index(targets, k, min_freq, max_freq)
    b = oracle_mod.SeqBatch(queries.ids, queries.offsets, queries.bases.tobytes())
    rows = 0
    for variant in variants:
        pv = dict(params, kmer_size=k, **variant)
        runs = gpu.overlaps(queries, OverlapParams.make(**pv))
        gpu.set_sorted_emission(0)
        try:
            hits = gpu.overlaps(queries, OverlapParams.make(**pv))
        finally:
            gpu.set_sorted_emission(1)
        exp = oracle_mod.overlaps(idx, b, oracle_mod.default_params(**pv))
        assert runs.tobytes() == hits.tobytes(), variant
        assert overlap_tuples_gpu(runs) == overlap_tuples_oracle(exp), variant
        rows += len(runs)
    return rows


@pytest.mark.parametrize("k", [11, 15, 16, 17, 31])
def test_read_lengths_around_tiles(gpu, oracle_mod, k):
    """Reads whose windows end just before, at and after a 32-window tile,
    some of them a target's very ends, both strands, one base apart."""
    from cuflye_gb300 import synth
    rng = np.random.default_rng(k)
    genome = synth.random_genome(rng, 3000)
    lengths = [k - 1, k, k + 1, k + 30, k + 31, k + 32, k + 62, k + 63, k + 64, k + 65, 400, 900]
    seqs = []
    for n in lengths:
        for s in (0, 1, 31, 32, 33, 500, len(genome) - n):
            seqs.append(genome[s:s + n])
    seqs += [genome[:1500], genome[1400:], synth.revcomp(genome[700:2200])]
    for i in range(0, len(seqs), 3):
        seqs[i] = synth.revcomp(seqs[i])
    for i in range(0, len(seqs), 4):
        seqs[i] = synth.mutate(rng, seqs[i], 0.01, 0.003, 0.003)
    reads = synth.ReadSet.from_strings(np.arange(1, len(seqs) + 1), [x.tobytes() for x in seqs])
    params = dict(synth.OVERLAP_PARAMS, min_overlap=40)
    assert _check(gpu, oracle_mod, reads, reads, k, 1, 1000, params) > 0


@pytest.mark.parametrize("seed", [1, 2, 3, 4, 5, 6])
def test_tandem_arrays(gpu, oracle_mod, seed):
    from cuflye_gb300 import synth
    wl = synth.tandem_case(20 + seed, genome_len=10_000, coverage=4.0, arrays=1,
                           copy_div=(0.0, 0.01, 0.04, 0.1, 0.2, 0.02)[seed - 1])
    assert _check(gpu, oracle_mod, wl.reads, wl.reads, wl.k, wl.min_freq, 1000, wl.params) > 0


@pytest.mark.parametrize("sub,indel", [(0.0, 0.0), (0.002, 0.001), (0.02, 0.02), (0.05, 0.03)])
def test_error_rates(gpu, oracle_mod, sub, indel):
    from cuflye_gb300 import synth
    wl = synth.small_overlap_case(31, genome_len=50_000, coverage=8.0, sub=sub, ins=indel,
                                  dele=indel, repeat=True)
    _check(gpu, oracle_mod, wl.reads, wl.reads, wl.k, 1, wl.max_freq, wl.params)


def test_long_targets_and_strands(gpu, oracle_mod):
    """Groups sorted by ext pos, queries under positive, negative and unknown
    ids, and an indexed id whose sequence differs from the indexed one."""
    from cuflye_gb300 import synth
    rng = np.random.default_rng(77)
    sw = synth.serving_workload(seed=9, genome_len=1_500_000, n_queries=40, piece=400_000)
    q = sw.queries
    seqs = [np.frombuffer(q.seq(i), dtype=np.uint8) for i in range(q.n)]
    t0 = np.frombuffer(sw.targets.seq(0), dtype=np.uint8)[1000:31_000]
    seqs += [t0, synth.revcomp(t0), synth.mutate(rng, t0, 0.02, 0.01, 0.01)]
    ids = list(q.ids) + [1, -1, 2]
    qs = synth.ReadSet.from_strings(np.array(ids, dtype=np.int64), [x.tobytes() for x in seqs])
    assert _check(gpu, oracle_mod, sw.targets, qs, sw.k, 1, 32, sw.params, VARIANTS[:3]) > 0


def test_run_path_is_taken(gpu):
    """The default takes runs (its algorithmic sort bytes count runs, far fewer
    than hits); an even k has no run tables."""
    from cuflye_gb300 import synth
    from cuflye_gb300.backend import OverlapParams
    wl = synth.small_overlap_case(5, genome_len=60_000, sub=0.001, ins=0.0, dele=0.0)
    for k, fewer in ((15, True), (16, False)):
        gpu.build_index(wl.reads, k, 2, 40)
        p = OverlapParams.make(**dict(wl.params, kmer_size=k))
        gpu.overlaps(wl.reads, p)
        runs = gpu.last_timing()[1][1]
        gpu.set_sorted_emission(0)
        try:
            gpu.overlaps(wl.reads, p)
        finally:
            gpu.set_sorted_emission(1)
        hits = gpu.last_timing()[1][1]
        assert (runs * 4 < hits) == fewer


def test_queries_around_the_sort_capacity(gpu, oracle_mod):
    """Queries of a few runs up to more than a block sorts on chip (4096)."""
    from cuflye_gb300 import synth
    from cuflye_gb300.backend import OverlapParams
    rng = np.random.default_rng(4096)
    genome = synth.random_genome(rng, 4000)
    seqs = [synth.mutate(rng, genome[:n], 0.04, 0.01, 0.01)
            for n in np.linspace(60, 4000, 160).astype(int)]
    reads = synth.ReadSet.from_strings(np.arange(1, len(seqs) + 1), [x.tobytes() for x in seqs])
    params = dict(synth.OVERLAP_PARAMS, min_overlap=200)
    assert _check(gpu, oracle_mod, reads, reads, 11, 1, 1000, params, VARIANTS[:2]) > 0
    runs = []
    for i in (0, reads.n - 1):
        one = synth.ReadSet.from_strings(np.array([i + 1]), [reads.seq(i)])
        gpu.overlaps(one, OverlapParams.make(**dict(params, kmer_size=11)))
        runs.append(gpu.last_timing()[1][1] // 24)
    assert runs[0] < 4096 < runs[1]


@pytest.mark.parametrize("nq", [1, 8191, 8193, 32767, 32768, 32769])
def test_query_counts_around_the_scans(gpu, oracle_mod, nq):
    """Scans of one block (up to 32768 entries) and of three kernels."""
    from cuflye_gb300 import synth
    rng = np.random.default_rng(nq)
    genome = synth.random_genome(rng, 30_000)
    at = rng.integers(0, len(genome) - 60, size=nq)
    reads = synth.ReadSet.from_strings(
        np.arange(100, 100 + nq), [genome[s:s + 60].tobytes() for s in at])
    targets = synth.ReadSet.from_strings(
        np.arange(1, 31), [genome[i:i + 1000].tobytes() for i in range(0, 30_000, 1000)])
    params = dict(synth.OVERLAP_PARAMS, min_overlap=40)
    assert _check(gpu, oracle_mod, targets, reads, 15, 1, 100, params, VARIANTS[1:2]) > 0


@pytest.mark.parametrize("k,kind", [(15, "sub"), (15, "ins"), (15, "del"), (31, "sub"), (17, "hole")])
def test_run_ends_around_the_expected_place(gpu, oracle_mod, k, kind):
    """Long runs that end at every distance from the group's next run: a second
    error (or a stretch of repetitive k-mers) at each offset from the first."""
    from cuflye_gb300 import synth
    rng = np.random.default_rng(k)
    target = synth.random_genome(rng, 700)
    unit = synth.random_genome(rng, 25)
    filler = [np.concatenate([synth.random_genome(rng, 30), unit] * 8)] if kind == "hole" else []
    queries = []
    for d in range(0, 90):
        s = target.copy()
        s[250] = ord("ACGT"["TGCA".index(chr(s[250]))])
        if kind == "sub" and d:
            s[250 + d] = ord("ACGT"["TGCA".index(chr(s[250 + d]))])
        elif kind == "ins":
            s = np.insert(s, 250 - d, s[250 - d])
        elif kind == "del":
            s = np.delete(s, 250 + d)
        elif kind == "hole":
            s[200 - d:225 - d] = unit
        queries.append(s if d % 2 else synth.revcomp(s))
    targets = [target] + filler
    if kind == "hole":
        targets.append(queries[7])  # shares the stretch, at one place
    t = synth.ReadSet.from_strings(np.arange(1, len(targets) + 1), [x.tobytes() for x in targets])
    q = synth.ReadSet.from_strings(np.arange(50, 50 + len(queries)), [x.tobytes() for x in queries])
    params = dict(synth.OVERLAP_PARAMS, min_overlap=100)
    assert _check(gpu, oracle_mod, t, q, k, 1, 6, params, VARIANTS[:2]) >= len(queries)


@pytest.mark.parametrize("passes", [0, 7])
def test_queries_around_the_large_sort(gpu, oracle_mod, passes):
    """Queries of up to more runs than the large sort takes on chip (16384), in
    one pass and in passes."""
    from cuflye_gb300 import synth
    from cuflye_gb300.backend import OverlapParams
    rng = np.random.default_rng(16384)
    genome = synth.random_genome(rng, 12_000)
    seqs = [synth.mutate(rng, genome[:n], 0.05, 0.01, 0.01)
            for n in rng.permutation(np.linspace(60, 12_000, 160).astype(int))]
    reads = synth.ReadSet.from_strings(np.arange(1, len(seqs) + 1), [x.tobytes() for x in seqs])
    params = dict(synth.OVERLAP_PARAMS, min_overlap=200)
    gpu.set_batch_queries(passes)
    try:
        assert _check(gpu, oracle_mod, reads, reads, 11, 1, 1000, params, VARIANTS[:1]) > 0
    finally:
        gpu.set_batch_queries(0)
    runs = []
    for n in (200, 2500, 12_000):
        i = int(np.argmin([abs(len(x) - n) for x in seqs]))
        one = synth.ReadSet.from_strings(np.array([i + 1]), [reads.seq(i)])
        gpu.overlaps(one, OverlapParams.make(**dict(params, kmer_size=11)))
        runs.append(gpu.last_timing()[1][1] // 24)
    assert runs[0] < 4096 < runs[1] < 16384 < runs[2], runs


@pytest.mark.parametrize("copies", [2, 3, 6])
@pytest.mark.parametrize("longer_query", [False, True])
def test_ties_at_the_first_position(gpu, oracle_mod, copies, longer_query):
    """Several hits at a group's first position, one of them the chain's start:
    which of them is element 0 decides the chain's score."""
    from cuflye_gb300 import synth
    rng = np.random.default_rng(10 * copies + longer_query)
    targets, queries = [], []
    for i in range(24):
        base = synth.random_genome(rng, 900)
        parts = [base]
        for c in range(copies - 1):  # copies of its start, before or after it
            copy = base[:int(rng.integers(20, 120))]
            gap = synth.random_genome(rng, int(rng.integers(10, 200)))
            parts = [copy, gap] + parts if rng.random() < 0.5 else parts + [gap, copy]
        t = np.concatenate(parts)
        q = synth.mutate(rng, base, 0.01, 0.003, 0.003) if i % 3 else base
        q = np.concatenate([q, synth.random_genome(rng, 4000 if longer_query else 10)])
        if i % 2:
            t = synth.revcomp(t)
        if i % 4 > 1:
            q = synth.revcomp(q)
        targets.append(t.tobytes())
        queries.append(q.tobytes())
    ts = synth.ReadSet.from_strings(np.arange(1, 25), targets)
    qs = synth.ReadSet.from_strings(np.arange(100, 124), queries)
    params = dict(synth.OVERLAP_PARAMS, min_overlap=100)
    assert _check(gpu, oracle_mod, ts, qs, 15, 1, 100, params, VARIANTS[1:3]) > 0
