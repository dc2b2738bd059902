"""GPU: index builds where one target holds a k-mer many times (above 32 its
entries are placed by a block, up to there by a walk each)."""

import time

import numpy as np
import pytest

from test_gpu_parity import cand_tuples_gpu, cand_tuples_oracle, oracle_index

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [15, 16])
@pytest.mark.parametrize("copies", [31, 32, 33, 34, 511, 512, 513, 1025, 4_096, 4_097, 9_000])
def test_bucket_order_of_repeated_kmers(gpu, oracle_mod, k, copies):
    """A word at that many places of one target, on both strands, beside targets
    with it once, a few times, and 33 times on one strand only."""
    from cuflye_gb300 import synth
    rng = np.random.default_rng(copies * k)
    word = synth.random_genome(rng, k)
    words = (word, synth.revcomp(word))

    def target(n, strands):
        parts = []
        for _ in range(n):
            parts += [synth.random_genome(rng, int(rng.integers(1, 12))),
                      words[int(rng.integers(0, 2)) if strands == 2 else strands]]
        return np.concatenate(parts + [synth.random_genome(rng, 40)]).tobytes()

    seqs = [target(3, 2), target(copies, 2), target(1, 1), target(33, 0), target(33, 1),
            target(copies, 2)]
    t = synth.ReadSet.from_strings(np.arange(1, len(seqs) + 1), seqs)
    q = synth.ReadSet.from_strings(
        np.array([50, 51, 2, -4]), [word.tobytes(), words[1].tobytes(), seqs[1][:400], seqs[3]])
    idx, _ = oracle_index(oracle_mod, t, k, 1, 100_000)
    exp = oracle_mod.candidates(idx, oracle_mod.SeqBatch(q.ids, q.offsets, q.bases.tobytes()))
    gpu.build_index(t, k, 1, 100_000)
    got = gpu.candidates(q)[0]
    assert len(got) > 2 * copies
    assert cand_tuples_gpu(got) == cand_tuples_oracle(exp)


def test_build_time_is_linear_in_repeats(built_lib):
    """Two million equal k-mers of one target take a build that long at most 20
    times what as many different ones take (a walk each: 3,500 times)."""
    from cuflye_gb300 import synth
    from cuflye_gb300.backend import CudaBackend
    rng = np.random.default_rng(2)
    n = 2_000_000
    same = np.concatenate([np.full(n // 2, ord("A"), np.uint8), np.full(n // 2, ord("T"), np.uint8)])
    ms = []
    with CudaBackend(device=0, memory_budget_bytes=0) as be:
        for seq in (synth.random_genome(rng, n), same):
            t = synth.ReadSet.from_strings(np.array([1]), [seq.tobytes()])
            best = 1e9
            for _ in range(3):
                t0 = time.perf_counter()
                be.build_index(t, 17, 1, 4_000_000)
                best = min(best, time.perf_counter() - t0)
            ms.append(1e3 * best)
    assert ms[1] <= 20 * ms[0], ms
