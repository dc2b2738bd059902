"""GPU: ranges that the segmented sort partitions by a cluster of blocks (longer
than 16,384 elements), alone and beside ranges for one block, against libstdc++."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lengths", [
    [16_384], [16_385], [16_384 + 8 * 32], [65_537], [262_144 + 1],
    [16_385, 16_384, 4_097, 4_096, 40_000, 0, 1, 17_000], [20_000] * 45])
@pytest.mark.parametrize("values", [2, 700, 1 << 20])
def test_long_ranges_match_libstdcxx(gpu, oracle_mod, lengths, values):
    rng = np.random.default_rng(sum(lengths) + values)
    offs = np.concatenate([[0], np.cumsum(lengths)]).astype(np.uint64)
    n = int(offs[-1])
    keys = rng.integers(0, values, size=n).astype(np.uint64) << np.uint64(20)
    a = int(offs[len(lengths) // 2])
    keys[a:a + 9_000] = np.sort(keys[a:a + 9_000])  # a rising stretch
    vals = np.arange(n, dtype=np.uint32)
    k2, v2 = gpu.std_sort_segments(keys, vals, offs)
    for s in range(len(lengths)):
        a, b = int(offs[s]), int(offs[s + 1])
        ek, ev = oracle_mod.std_sort_u64(keys[a:b], vals[a:b])
        assert np.array_equal(k2[a:b], ek) and np.array_equal(v2[a:b], ev), s
