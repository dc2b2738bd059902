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
