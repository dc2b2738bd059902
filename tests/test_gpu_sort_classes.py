"""GPU: segments of every size class of the segmented sort, in calls of few, of
many short and of many long segments (which decides who sorts the middle class),
against libstdc++."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EDGES = [0, 1, 2, 16, 17, 64, 65, 511, 512, 513, 1024, 2047, 2048, 2049, 4096, 4097]


@pytest.mark.parametrize("lengths", [EDGES, EDGES + [513] * 700, EDGES * 2 + [2048] * 400,
                                     EDGES + [2048] * 300 + [3] * 400, [2048] * 304,
                                     [1024] * 305, [1025] * 305],
                         ids=["few", "short", "long", "mixed", "most-few", "mean", "above-mean"])
def test_classes_match_libstdcxx(gpu, oracle_mod, lengths):
    rng = np.random.default_rng(sum(lengths))
    lengths = rng.permutation(np.array(lengths))
    offs = np.concatenate([[0], np.cumsum(lengths)]).astype(np.uint64)
    n = int(offs[-1])
    keys = rng.integers(0, 300, size=n).astype(np.uint64) << np.uint64(33)
    vals = np.arange(n, dtype=np.uint32)
    k2, v2 = gpu.std_sort_segments(keys, vals, offs)
    for s in range(len(lengths)):
        a, b = int(offs[s]), int(offs[s + 1])
        ek, ev = oracle_mod.std_sort_u64(keys[a:b], vals[a:b])
        assert np.array_equal(k2[a:b], ek) and np.array_equal(v2[a:b], ev), (s, b - a)
