"""GPU: the run path where its side tables run out.  What does not fit takes the
hit path; the rows stay those of the hit path and of the oracle."""

import ctypes

import pytest

from test_gpu_parity import oracle_index, overlap_tuples_gpu, overlap_tuples_oracle

pytestmark = pytest.mark.gpu


def _rows(gpu, reads, params):
    """The hit path's rows."""
    gpu.set_sorted_emission(0)
    try:
        return gpu.overlaps(reads, params).tobytes()
    finally:
        gpu.set_sorted_emission(1)


def _launches(be):
    n = ctypes.c_uint64()
    be._L.cuflye_kernel_launches(ctypes.byref(n))
    return n.value


def _tandem(copy_div, seed=21, **kw):
    from cuflye_gb300 import synth
    return synth.tandem_case(seed, genome_len=10_000, coverage=4.0, arrays=1, copy_div=copy_div,
                             **kw)


@pytest.mark.parametrize("copy_div", [0.0, 0.04])
def test_spare_pieces_run_out(gpu, oracle_mod, copy_div):
    """Groups whose runs overlap, with room for the pieces of none, of some and of
    all of them: those without room are left to the hit path, the others go on."""
    from cuflye_gb300.backend import OverlapParams
    wl = _tandem(copy_div)
    p = OverlapParams.make(**wl.params)
    oracle_mod.set_stable(False)
    idx, batch = oracle_index(oracle_mod, wl.reads, wl.k, wl.min_freq, 1000)
    exp = oracle_mod.overlaps(idx, batch, oracle_mod.default_params(**wl.params))
    gpu.build_index(wl.reads, wl.k, wl.min_freq, 1000)
    hits = _rows(gpu, wl.reads, p)
    chained = []
    try:
        for most in (0, 1, 40, 300, 1_000, 3_000, 10_000, None):
            gpu.set_run_limit("spare_pieces", most)
            rows = gpu.overlaps(wl.reads, p)
            assert rows.tobytes() == hits, most
            assert overlap_tuples_gpu(rows) == overlap_tuples_oracle(exp), most
            chained.append(gpu.last_sort_stats()["match_libstdcxx"])
    finally:
        gpu.set_run_limit("spare_pieces", None)
    # without room every such group takes its query's sorted hits
    assert chained[0] == max(chained) > 0


@pytest.mark.parametrize("copies", [2, 4])
def test_tie_list_runs_out(gpu, oracle_mod, copies):
    """More hits at shared positions than the list holds, few beside their
    queries' hits: Flye's order among them decides which one a chain starts at."""
    import numpy as np
    from cuflye_gb300 import synth
    from cuflye_gb300.backend import OverlapParams
    rng = np.random.default_rng(copies)
    targets, queries = [], []
    for i in range(32):
        base = synth.random_genome(rng, int(rng.integers(12_000, 30_000)))
        parts = [base]
        for _ in range(copies - 1):  # copies of its start, before or after it
            copy = base[:int(rng.integers(20, 80))]
            gap = synth.random_genome(rng, int(rng.integers(10, 200)))
            parts = [copy, gap] + parts if rng.random() < 0.5 else parts + [gap, copy]
        targets.append(np.concatenate(parts))
        q = synth.mutate(rng, base, 0.01, 0.003, 0.003) if i % 3 else base
        queries.append(np.concatenate([q, synth.random_genome(rng, 40_000)]))  # the longer one
    ts = synth.ReadSet.from_strings(np.arange(1, 33), [x.tobytes() for x in targets])
    qs = synth.ReadSet.from_strings(np.arange(100, 132), [x.tobytes() for x in queries])
    params = dict(synth.OVERLAP_PARAMS, kmer_size=15, only_max_ext=0, check_overhang=0)
    p = OverlapParams.make(**params)
    idx, _ = oracle_index(oracle_mod, ts, 15, 1, 100)
    b = oracle_mod.SeqBatch(qs.ids, qs.offsets, qs.bases.tobytes())
    exp = {}
    for stable in (True, False):
        oracle_mod.set_stable(stable)
        rows = oracle_mod.overlaps(idx, b, oracle_mod.default_params(**params))
        exp[stable] = overlap_tuples_oracle(rows)
    assert exp[True] != exp[False]  # the order among equal keys shows in the rows
    gpu.build_index(ts, 15, 1, 100)
    try:
        for most in (0, 1, 16, 200, None):
            gpu.set_run_limit("tie_keys", most)
            assert overlap_tuples_gpu(gpu.overlaps(qs, p)) == exp[False], most
            assert gpu.last_sort_stats()["match_libstdcxx"] > 0
    finally:
        gpu.set_run_limit("tie_keys", None)


@pytest.mark.parametrize("most", [None, 0])
def test_open_groups_rows_find_room(gpu, oracle_mod, most):
    """A large pass (above 32,768 runs) whose groups nearly all repeat positions,
    with room for the pieces of some and of none: every group's rows are kept."""
    import numpy as np
    from cuflye_gb300 import synth
    from cuflye_gb300.backend import OverlapParams
    rng = np.random.default_rng(8)
    unit = synth.random_genome(rng, 200)
    read = np.concatenate([synth.random_genome(rng, 300), unit, unit, synth.random_genome(rng, 300)])
    n = 120
    reads = synth.ReadSet.from_strings(
        np.arange(1, n + 1), [(synth.revcomp(read) if i % 3 == 1 else read).tobytes()
                              for i in range(n)])
    params = dict(synth.OVERLAP_PARAMS, kmer_size=15, min_overlap=400)
    p = OverlapParams.make(**params)
    oracle_mod.set_stable(False)
    idx, batch = oracle_index(oracle_mod, reads, 15, 1, 1000)
    exp = overlap_tuples_oracle(
        oracle_mod.overlaps(idx, batch, oracle_mod.default_params(**params)))
    assert len(exp) >= n * (n - 1)
    gpu.build_index(reads, 15, 1, 1000)
    gpu.set_run_limit("spare_pieces", most)
    try:
        rows = gpu.overlaps(reads, p)
        assert gpu.last_timing()[1][1] // 24 > 32_768  # runs (and no other hits) sorted
    finally:
        gpu.set_run_limit("spare_pieces", None)
    assert overlap_tuples_gpu(rows) == exp


def test_open_groups_share_batches_under_a_budget(built_lib):
    """Queries of open groups whose hits take about four times the memory there is
    go through in batches of many queries, not one by one: the launches stay
    within a multiple of an unbounded call's, which takes them in one batch."""
    import numpy as np
    from cuflye_gb300 import synth
    from cuflye_gb300.backend import CudaBackend, OverlapParams
    rng = np.random.default_rng(12)
    unit = synth.random_genome(rng, 250)
    genome = np.concatenate([synth.random_genome(rng, 2500), unit, unit, unit,
                             synth.random_genome(rng, 2500)])
    n = 100
    seqs = []
    for _ in range(n):
        a, b = int(rng.integers(0, 2000)), int(rng.integers(3800, len(genome)))
        s = synth.mutate(rng, genome[a:b], 0.002, 0.0005, 0.0005)
        seqs.append((synth.revcomp(s) if rng.random() < 0.5 else s).tobytes())
    reads = synth.ReadSet.from_strings(np.arange(1, n + 1), seqs)
    p = OverlapParams.make(**dict(synth.OVERLAP_PARAMS, kmer_size=15))
    got, launches, held = [], [], 0
    for budget in (0, 1):
        with CudaBackend(device=0, memory_budget_bytes=budget and held) as be:
            be.build_index(reads, 15, 1, 2000)
            index_bytes = be.memory_stats()[0]
            be.set_run_limit("spare_pieces", 0)  # every group with a repeated position is open
            before = _launches(be)
            got.append(be.overlaps(reads, p).tobytes())
            launches.append(_launches(be) - before)
            assert be.last_sort_stats()["match_libstdcxx"] == n
            if not budget:
                be.set_sorted_emission(0)
                assert be.overlaps(reads, p).tobytes() == got[0]
                hits = be.last_timing()[1][1] // 24
                held = index_bytes + 66 * hits // 4
    assert got[0] == got[1]
    # eight batches (half the memory each, at worst) and as many passes
    assert launches[1] <= 16 * launches[0], launches


def test_open_groups_of_many_rows(gpu, oracle_mod):
    """Open groups of about twenty rows each beside many groups of one: the open
    ones have the room that the others leave."""
    import numpy as np
    from cuflye_gb300 import synth
    from cuflye_gb300.backend import OverlapParams
    rng = np.random.default_rng(6)
    unit = synth.random_genome(rng, 150)
    base = np.concatenate([synth.random_genome(rng, 500), unit, unit, synth.random_genome(rng, 500)])
    other = synth.random_genome(rng, 1000)
    seqs = [synth.mutate(rng, base, 0.006, 0, 0.0015) for _ in range(20)] + [other] * 60
    reads = synth.ReadSet.from_strings(np.arange(1, len(seqs) + 1), [s.tobytes() for s in seqs])
    params = dict(synth.OVERLAP_PARAMS, kmer_size=15, min_overlap=1, max_jump=16, max_gap=1,
                  check_overhang=0, force_local=1, only_max_ext=0)
    p = OverlapParams.make(**params)
    oracle_mod.set_stable(False)
    idx, batch = oracle_index(oracle_mod, reads, 15, 1, 1000)
    exp = overlap_tuples_oracle(
        oracle_mod.overlaps(idx, batch, oracle_mod.default_params(**params)))
    of_open = sum(r[0] <= 20 for r in exp)
    assert 9 * 400 + 1024 < of_open and len(exp) < 8 * (60 * 59 + 380) + 1024
    gpu.build_index(reads, 15, 1, 1000)
    hits = _rows(gpu, reads, p)
    gpu.set_run_limit("spare_pieces", 0)
    try:
        rows = gpu.overlaps(reads, p)
        assert gpu.last_sort_stats()["match_libstdcxx"] >= 20
    finally:
        gpu.set_run_limit("spare_pieces", None)
    assert rows.tobytes() == hits
    assert overlap_tuples_gpu(rows) == exp


@pytest.mark.parametrize("k", [5, 7, 9, 11])
def test_least_k(gpu, oracle_mod, k):
    """k-mers shorter than 11 are chained hit by hit."""
    from cuflye_gb300 import synth
    from cuflye_gb300.backend import OverlapParams
    wl = synth.small_overlap_case(6, genome_len=2_000, coverage=6.0, sub=0.01, ins=0.002,
                                  dele=0.002)
    params = dict(wl.params, kmer_size=k, min_overlap=1000)
    p = OverlapParams.make(**params)
    oracle_mod.set_stable(False)
    idx, batch = oracle_index(oracle_mod, wl.reads, k, 1, 400)
    exp = oracle_mod.overlaps(idx, batch, oracle_mod.default_params(**params))
    gpu.build_index(wl.reads, k, 1, 400)
    rows = gpu.overlaps(wl.reads, p)
    sorted_bytes = gpu.last_timing()[1][1]
    assert overlap_tuples_gpu(rows) == overlap_tuples_oracle(exp)
    assert rows.tobytes() == _rows(gpu, wl.reads, p)
    assert (sorted_bytes < gpu.last_timing()[1][1]) == (k >= 11)
