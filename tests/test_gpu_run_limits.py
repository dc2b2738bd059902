"""GPU: the run path where its side tables run out.  What does not fit takes the
hit path; the rows stay those of the hit path and of the oracle."""

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
