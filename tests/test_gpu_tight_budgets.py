"""GPU: what a memory budget admits, a larger one admits too.  The index keeps
tables beside its entries when there is room for them; a query that needs that
room gets it back, in the owner's calls and in those that borrow its index."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _call(mode, be, query, p):
    from cuflye_gb300.backend import CudaServer
    if mode == "candidates":
        return be.candidates(query)[0].tobytes()
    if mode == "hits":
        be.set_sorted_emission(0)
    if mode.startswith("server"):
        with CudaServer(be, p, workers=int(mode[-1])) as srv:
            tickets = [srv.submit(query) for _ in range(3)]
            rows = [srv.poll(t, -1).tobytes() for t in tickets]
            assert rows[0] == rows[1] == rows[2]
            return rows[0]
    return be.overlaps(query, p).tobytes()


def _shared(owner, budget):
    """A context that borrows the owner's index."""
    from cuflye_gb300.backend import CudaBackend
    be = CudaBackend.__new__(CudaBackend)
    be._L, be._h, be.k = owner._L, ctypes.c_void_p(), owner.k
    assert owner._L.cuflye_open_shared(owner._h, budget, ctypes.byref(be._h)) == 0
    return be


@pytest.mark.parametrize("length", [5_000, 6_500, 8_500])
@pytest.mark.parametrize("mode,k", [("overlaps", 16), ("hits", 15), ("candidates", 15),
                                    ("server1", 16), ("server2", 16)])
def test_larger_budgets_admit_what_smaller_ones_do(built_lib, mode, k, length):
    from cuflye_gb300 import synth
    from cuflye_gb300.backend import CudaBackend, CuflyeError, OverlapParams
    rng = np.random.default_rng(length)
    unit = synth.random_genome(rng, 3000)
    targets = synth.ReadSet.from_strings(np.arange(1, 301), [unit.tobytes()] * 300)
    query = synth.ReadSet.from_strings(np.array([900]), [np.resize(unit, length).tobytes()])
    p = OverlapParams.make(**dict(synth.OVERLAP_PARAMS, kmer_size=k))
    admitted, rows = [], set()
    for mib in range(60, 420 if mode == "server2" else 260, 4):
        try:
            with CudaBackend(device=0, memory_budget_bytes=mib << 20) as be:
                be.build_index(targets, k, 1, 2000)
                rows.add(_call(mode, be, query, p))
            admitted.append(mib)
        except CuflyeError as e:
            assert "BUDGET" in str(e) or "budget" in str(e), e
            assert not admitted, (admitted[0], mib)  # a smaller one did
    assert admitted and len(rows) == 1


def test_calls_go_on_without_the_tables(built_lib):
    """After a query took the tables' room: the owner, a context that borrows its
    index and a server give the rows that a fresh context gives, and a rebuild has
    the tables again."""
    from cuflye_gb300 import synth
    from cuflye_gb300.backend import CudaBackend, CudaServer, CuflyeError, OverlapParams
    wl = synth.small_overlap_case(5, genome_len=60_000, sub=0.002, ins=0.001, dele=0.001)
    rng = np.random.default_rng(1)
    unit = synth.random_genome(rng, 3000)
    seqs = [wl.reads.seq(i) for i in range(wl.reads.n)] + [unit.tobytes()] * 300
    targets = synth.ReadSet.from_strings(np.arange(1, len(seqs) + 1), seqs)
    big = synth.ReadSet.from_strings(np.array([9000]), [np.resize(unit, 9000).tobytes()])
    p = OverlapParams.make(**dict(wl.params, kmer_size=15))

    def sort_bytes(be):
        return be.last_timing()[1][1]

    with CudaBackend(device=0, memory_budget_bytes=0) as be:
        be.build_index(targets, 15, 1, 2000)
        want = be.overlaps(wl.reads, p).tobytes()
        by_runs = sort_bytes(be)
        want_big = be.candidates(big)[0].tobytes()
    for mib in range(120, 400, 4):
        with CudaBackend(device=0, memory_budget_bytes=mib << 20) as be:
            be.build_index(targets, 15, 1, 2000)
            held = be.memory_stats()[0]
            try:
                assert be.overlaps(wl.reads, p).tobytes() == want
            except CuflyeError:
                continue  # too small a budget for the reads
            if sort_bytes(be) != by_runs:
                continue  # no room for the tables
            with _shared(be, 256 << 20) as other, CudaServer(be, p, workers=1) as srv:
                assert other.overlaps(wl.reads, p).tobytes() == want
                assert srv.poll(srv.submit(wl.reads), -1).tobytes() == want
                try:
                    assert be.candidates(big)[0].tobytes() == want_big
                except CuflyeError:
                    continue  # too small a budget for the query
                be.trim()
                if be.memory_stats()[0] >= held:
                    continue  # room for both
                for _ in range(2):
                    assert other.overlaps(wl.reads, p).tobytes() == want
                    assert sort_bytes(other) > 2 * by_runs
                    assert srv.poll(srv.submit(wl.reads), -1).tobytes() == want
                    assert be.overlaps(wl.reads, p).tobytes() == want
            be.build_index(targets, 15, 1, 2000)
            assert be.overlaps(wl.reads, p).tobytes() == want and sort_bytes(be) == by_runs
            return
    pytest.fail("no budget at which the query took the tables' room")


@pytest.mark.parametrize("mode", ["sort", "server"])
def test_other_calls_get_the_tables_room(built_lib, mode):
    """A sort of arrays that fit beside the entries alone, and a server whose
    workers' least memory does: admitted at every budget above the first."""
    from cuflye_gb300 import synth
    from cuflye_gb300.backend import CudaBackend, CudaServer, CuflyeError, OverlapParams
    rng = np.random.default_rng(3)
    unit = synth.random_genome(rng, 3000)
    targets = synth.ReadSet.from_strings(np.arange(1, 301), [unit.tobytes()] * 300)
    keys = rng.integers(0, 1 << 40, size=3_600_000).astype(np.uint64)
    vals = np.arange(len(keys), dtype=np.uint32)
    offs = np.arange(0, len(keys) + 1, 1000).astype(np.uint64)
    p = OverlapParams.make(**dict(synth.OVERLAP_PARAMS, kmer_size=15))
    admitted = []
    for mib in range(70, 200, 2):
        try:
            with CudaBackend(device=0, memory_budget_bytes=mib << 20) as be:
                be.build_index(targets, 15, 1, 2000)
                if mode == "sort":
                    k2, _ = be.std_sort_segments(keys, vals, offs)
                    assert np.array_equal(k2.reshape(-1, 1000), np.sort(keys.reshape(-1, 1000)))
                else:
                    with CudaServer(be, p, workers=1):
                        pass
            admitted.append(mib)
        except CuflyeError as e:
            assert "BUDGET" in str(e), e
            assert not admitted, (admitted[0], mib)
    assert admitted


def test_run_path_admits_what_the_hit_path_does(built_lib):
    """Reads of a tandem array under every budget around what they need: where the
    hit path gives the rows, so does the run path, twice in a row."""
    from cuflye_gb300 import synth
    from cuflye_gb300.backend import CudaBackend, CuflyeError, OverlapParams
    rng = np.random.default_rng(217)
    unit = synth.random_genome(rng, 200)
    genome = np.concatenate([synth.random_genome(rng, 2000)] + [unit] * 4 +
                            [synth.random_genome(rng, 2000)])
    seqs = []
    for i in range(7):
        a, b = int(rng.integers(0, 1900)), int(rng.integers(2900, len(genome)))
        s = synth.mutate(rng, genome[a:b], 0.01, 0.003, 0.003)
        seqs.append((synth.revcomp(s) if i % 2 else s).tobytes())
    reads = synth.ReadSet.from_strings(np.arange(1, 8), seqs)
    p = OverlapParams.make(**dict(synth.OVERLAP_PARAMS, kmer_size=17, min_overlap=100))
    got, rows = {}, set()
    for kib in range(2500, 8000, 90):
        for mode in (0, 1):
            try:
                with CudaBackend(device=0, memory_budget_bytes=kib << 10) as be:
                    be.build_index(reads, 17, 1, 3000)
                    be.set_sorted_emission(mode)
                    rows |= {be.overlaps(reads, p).tobytes() for _ in range(2)}
                got[kib, mode] = True
            except CuflyeError as e:
                assert "udget" in str(e), e
                got[kib, mode] = False
        assert got[kib, 1] or not got[kib, 0], kib
    assert len(rows) == 1 and not all(got.values())


def test_tables_go_while_others_read_the_index(built_lib):
    """Two borrowing contexts and a server in full use while the owner's query takes
    the tables: every call's rows stay the same."""
    import threading

    from cuflye_gb300 import synth
    from cuflye_gb300.backend import CudaBackend, CudaServer, CuflyeError, OverlapParams
    wl = synth.small_overlap_case(7, genome_len=60_000, sub=0.002, ins=0.001, dele=0.001)
    unit = synth.random_genome(np.random.default_rng(1), 3000)
    seqs = [wl.reads.seq(i) for i in range(wl.reads.n)] + [unit.tobytes()] * 300
    targets = synth.ReadSet.from_strings(np.arange(1, len(seqs) + 1), seqs)
    big = synth.ReadSet.from_strings(np.array([9000]), [np.resize(unit, 9000).tobytes()])
    p = OverlapParams.make(**dict(wl.params, kmer_size=15))
    parts = [wl.reads.subset(np.arange(i, min(i + 9, wl.reads.n)))
             for i in range(0, wl.reads.n, 9)]
    with CudaBackend(device=0, memory_budget_bytes=0) as be:
        be.build_index(targets, 15, 1, 2000)
        want = [be.overlaps(q, p).tobytes() for q in parts]
        want_big = be.candidates(big)[0].tobytes()
    gone = 0
    for mib in range(140, 260, 8):
        with CudaBackend(device=0, memory_budget_bytes=mib << 20) as be:
            be.build_index(targets, 15, 1, 2000)
            be.trim()
            held = be.memory_stats()[0]
            with _shared(be, 128 << 20) as a, _shared(be, 128 << 20) as b, \
                    CudaServer(be, p, workers=1) as srv:
                wrong, started = [], threading.Barrier(4)

                def work(call):
                    started.wait()
                    for _ in range(6):
                        for q, w in zip(parts, want):
                            try:
                                if call(q).tobytes() != w:
                                    wrong.append("rows")
                            except CuflyeError as e:
                                wrong.append(str(e))

                calls = [lambda q: a.overlaps(q, p), lambda q: b.overlaps(q, p),
                         lambda q: srv.poll(srv.submit(q), -1)]
                threads = [threading.Thread(target=work, args=(c,)) for c in calls]
                for t in threads:
                    t.start()
                started.wait()
                try:
                    assert be.candidates(big)[0].tobytes() == want_big
                except CuflyeError as e:
                    assert "udget" in str(e), e  # too small a budget for the query
                for t in threads:
                    t.join()
                assert not wrong, wrong[:3]
                be.trim()
                gone += be.memory_stats()[0] < held
    assert gone
