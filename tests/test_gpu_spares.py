"""GPU: the released buffers that a context keeps for its next allocations are
told apart from its buffers, and give way to other contexts."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GB = 1 << 30


def _targets(bases):
    from cuflye_gb300 import synth
    genome = synth.random_genome(np.random.default_rng(4), bases)
    return synth.ReadSet.from_strings(np.array([1]), [genome.tobytes()])


def test_spares_are_reported(built_lib):
    from cuflye_gb300.backend import CudaBackend
    with CudaBackend(device=0, memory_budget_bytes=0) as be:
        assert be.memory_spares() == 0
        be.build_index(_targets(4_000_000), 17, 1, 100)
        used = be.memory_stats()[0]
        assert be.memory_spares() > 4_000_000 * 16  # the build's sort arrays, at least
        be.trim()
        assert be.memory_spares() == 0 and be.memory_stats()[0] <= used


def test_a_failed_allocation_frees_other_contexts_spares(built_lib):
    """A sort that lacks memory on a device that is full but for what an idle
    context keeps."""
    torch = pytest.importorskip("torch")
    from cuflye_gb300.backend import CudaBackend
    rng = np.random.default_rng(5)
    n = 30_000_000
    keys = rng.integers(0, 1 << 40, size=n).astype(np.uint64)
    offs = np.arange(0, n + 1, 1000).astype(np.uint64)
    with CudaBackend(device=0, memory_budget_bytes=0) as idle, \
            CudaBackend(device=0, memory_budget_bytes=0) as be:
        idle.build_index(_targets(20_000_000), 17, 1, 100)
        kept = idle.memory_spares()
        assert kept > 6 * GB // 10
        # 24 bytes an element and tables; .4 GB are left beside what is kept
        free = torch.cuda.mem_get_info(0)[0]
        fill = torch.empty(free - 4 * GB // 10, dtype=torch.uint8, device="cuda:0")
        try:
            k2, _ = be.std_sort_segments(keys, np.arange(n, dtype=np.uint32), offs)
        finally:
            del fill
            torch.cuda.empty_cache()
        assert idle.memory_spares() == 0
        assert np.array_equal(k2.reshape(-1, 1000), np.sort(keys.reshape(-1, 1000)))
