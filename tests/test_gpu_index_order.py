"""GPU: the index's bucket order.  Windows are sorted by k-mer only, so the
entries of one target within a bucket (both strands of it, several positions)
are put in (stored id, position) order afterwards; candidate records show the
order entry by entry."""

import numpy as np
import pytest

from test_gpu_parity import cand_tuples_gpu, cand_tuples_oracle, oracle_index

pytestmark = pytest.mark.gpu


def _targets(rng, n, k):
    """Targets of about n windows in all whose k-mers repeat within a target on
    both strands: tandem units, inverted copies of them, and unique stretches."""
    from cuflye_gb300 import synth
    unit = synth.random_genome(rng, 3 * k)
    seqs, left = [], n
    while left > 0:
        parts = [synth.random_genome(rng, int(rng.integers(k, 4 * k)))]
        for _ in range(int(rng.integers(1, 6))):
            parts.append(unit if rng.random() < 0.5 else synth.revcomp(unit))
            if rng.random() < 0.3:
                parts.append(synth.random_genome(rng, int(rng.integers(1, 2 * k))))
        s = np.concatenate(parts)[:left + k - 1]
        seqs.append(s.tobytes())
        left -= max(1, len(s) - k + 1)
    order = rng.permutation(len(seqs))  # ids out of order
    return synth.ReadSet.from_strings(order.astype(np.int64) * 3 + 1, seqs)


@pytest.mark.parametrize("n,k", [(40, 7), (4095, 11), (4096, 11), (4097, 12), (20_000, 15),
                                 (70_000, 17)])
def test_bucket_order(gpu, oracle_mod, n, k):
    rng = np.random.default_rng(n + k)
    t = _targets(rng, n, k)
    idx, _ = oracle_index(oracle_mod, t, k, 1, 4000)
    gpu.build_index(t, k, 1, 4000)
    q = t.subset(np.arange(min(t.n, 12)))
    q.ids[::2] *= -1  # a read under its reverse id, and under its own
    b = oracle_mod.SeqBatch(q.ids, q.offsets, q.bases.tobytes())
    rec, filt = gpu.candidates(q)
    exp = oracle_mod.candidates(idx, b)
    assert len(rec) > 0
    assert cand_tuples_gpu(rec) == cand_tuples_oracle(exp)
    assert filt["pos"].tolist() == exp["filtered_pos"].tolist()


@pytest.mark.parametrize("k", [11, 15, 16, 31])
def test_window_records_change_no_result(built_lib, k):
    """An index built at once keeps a record a target window, one built in key
    ranges does not: hits and rows are the same, for targets around a block of
    windows (and shorter than a k-mer), their reverse strands, and sequences
    that differ from the indexed ones."""
    from cuflye_gb300 import synth
    from cuflye_gb300.backend import CudaBackend, OverlapParams
    rng = np.random.default_rng(100 + k)
    genome = synth.random_genome(rng, 1200)
    seqs = [genome[s:s + n] for s in (0, 100) for n in (k - 1, k, k + 1, 255 + k, 256 + k, 600)]
    seqs += [synth.mutate(rng, genome, 0.02, 0.005, 0.005) for _ in range(4)]
    targets = synth.ReadSet.from_strings(np.arange(1, len(seqs) + 1), [x.tobytes() for x in seqs])
    other = [synth.revcomp(x) for x in seqs] + [synth.mutate(rng, x, 0.05, 0.0, 0.0) for x in seqs[-4:]]
    ids = [-i for i in range(1, len(seqs) + 1)] + list(range(len(seqs) - 3, len(seqs) + 1))
    queries = synth.ReadSet.from_strings(np.array(ids), [x.tobytes() for x in other])
    p = OverlapParams.make(**dict(synth.OVERLAP_PARAMS, min_overlap=100, kmer_size=k,
                                  only_max_ext=0))
    got = []
    for ranges in (False, True):
        with CudaBackend(device=0) as be:
            if ranges:
                be.set_index_build_windows(3000)
            be.build_index(targets, k, 2, 1000)
            assert (be.last_index_ranges() > 1) == ranges
            for q in (targets, queries):
                cand, filt = be.candidates(q)
                got.append((cand.tobytes(), filt.tobytes(), be.overlaps(q, p).tobytes()))
    assert got[:2] == got[2:]
    assert all(len(x[0]) and len(x[2]) for x in got)


@pytest.mark.parametrize("room", [0.0, 0.02, 1.0])
def test_rebuilds_reuse_released_buffers(built_lib, room):
    """Index builds of two sizes in turn, and batches on them, give what a fresh
    context gives, within a budget that leaves the released buffers no room,
    little, or enough."""
    from cuflye_gb300 import synth
    from cuflye_gb300.backend import CudaBackend, OverlapParams
    cases = [synth.small_overlap_case(s, genome_len=n, coverage=8.0, sub=0.01, ins=0.002,
                                      dele=0.002) for s, n in ((3, 60_000), (4, 90_000))]
    fresh, peak = [], 0
    for wl in cases:
        with CudaBackend(device=0, memory_budget_bytes=0) as be:
            stats = be.build_index(wl.reads, wl.k, wl.min_freq, wl.max_freq)
            rows = be.overlaps(wl.reads, OverlapParams.make(**wl.params)).tobytes()
            fresh.append((stats, rows))
            peak = max(peak, be.memory_stats()[1])
    budget = int(peak * (1 + room)) + (1 << 20)
    with CudaBackend(device=0, memory_budget_bytes=budget) as be:
        for i in (0, 1, 0, 1, 1, 0):
            wl = cases[i]
            stats = be.build_index(wl.reads, wl.k, wl.min_freq, wl.max_freq)
            rows = be.overlaps(wl.reads, OverlapParams.make(**wl.params)).tobytes()
            assert (stats, rows) == fresh[i]
        assert be.memory_stats()[1] <= budget
        be.trim()
        assert be.overlaps(cases[0].reads, OverlapParams.make(**cases[0].params)).tobytes() == fresh[0][1]


@pytest.mark.parametrize("n", [16, 19, 20, 40, 300, 5_000, 70_000])
def test_lookups_of_absent_kmers(gpu, oracle_mod, n):
    """Queries under ids the index does not have, at indexes of one key up: half
    their k-mers indexed, half not."""
    from cuflye_gb300 import synth
    rng = np.random.default_rng(n)
    genome = synth.random_genome(rng, n)
    t = synth.ReadSet.from_strings(np.array([1]), [genome.tobytes()])
    queries = [genome, synth.revcomp(genome), synth.mutate(rng, genome, 0.1, 0.0, 0.0),
               synth.random_genome(rng, 2 * n)]
    q = synth.ReadSet.from_strings(np.arange(10, 14), [x.tobytes() for x in queries])
    idx, _ = oracle_index(oracle_mod, t, 15, 1, 100)
    gpu.build_index(t, 15, 1, 100)
    b = oracle_mod.SeqBatch(q.ids, q.offsets, q.bases.tobytes())
    cand, _ = gpu.candidates(q)
    exp = oracle_mod.candidates(idx, b)
    assert len(cand) >= 2 * (n - 14)
    assert cand_tuples_gpu(cand) == cand_tuples_oracle(exp)


@pytest.mark.parametrize("n", [15, 31, 32, 33, 63, 64, 200, 1000])
def test_letters_and_other_characters(gpu, oracle_mod, n):
    """Packing: both cases of the four letters, and every other byte as A."""
    from cuflye_gb300 import synth
    rng = np.random.default_rng(n)
    genome = synth.random_genome(rng, n)
    lower = np.frombuffer(genome.tobytes().lower(), dtype=np.uint8).copy()
    odd = genome.copy()
    at = rng.integers(0, n, size=max(1, n // 20))
    odd[at] = rng.integers(1, 256, size=len(at))
    plain = np.array([x if x in b"CGTcgt" else ord("A") for x in odd], dtype=np.uint8)
    t = synth.ReadSet.from_strings(np.array([1, 2]), [genome.tobytes(), odd.tobytes()])
    gpu.build_index(t, 15, 1, 100)
    got = []
    for a, b in ((genome, odd), (lower, plain)):
        q = synth.ReadSet.from_strings(np.array([5, 6]), [a.tobytes(), b.tobytes()])
        got.append(gpu.candidates(q)[0].tobytes())
    assert got[0] == got[1] and len(got[0]) > 0
    t2 = synth.ReadSet.from_strings(np.array([1, 2]), [lower.tobytes(), plain.tobytes()])
    gpu.build_index(t2, 15, 1, 100)
    assert gpu.candidates(q)[0].tobytes() == got[0]
