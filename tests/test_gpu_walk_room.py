"""The walk when there is no room for the records of its counting pass: within an HBM budget
that the records would break, and for compacted maps with more pieces than they hold.  Both
walk a second time instead; compared with the oracle."""
import pytest

import pakman_plus_gb300 as pk
from gpu_helpers import ctx
from oracle import pk_compact as pc
from pakman_plus_gb300 import synth

pytestmark = pytest.mark.gpu


def _compacted(job, rs, k, cov, threshold, t):
    job.count(rs.fasta, pk.default_params(k=k, coverage=cov))
    job.cutoff(t)
    job.build_macro_nodes(0)
    return job.macro_nodes(cov), job.compact(threshold, cov)


def _walk(mn, k, cov, threshold):
    return pc.walk(pc.compact(pc.initial_nodes(mn.keys, mn.suffix_counts, mn.prefix_counts, k, cov), k, threshold).nodes, k)


@pytest.mark.parametrize("k", [32, 63])
@pytest.mark.parametrize("threshold", [1 << 20, 40])
def test_walk_within_a_budget_that_its_records_would_break(k, threshold):
    rs = synth.small_case(9, genome_len=8000, n_reads=3200, read_len=100, k=k, coverage=20, err=0.003)
    with pk.Context(0, hbm_budget=32 << 30) as c, pk.Job(c) as job:
        mn, res = _compacted(job, rs, k, 20, threshold, 6)
        want = _walk(mn, k, 20, threshold)
        assert job.walk() == want
        used = c.memory()[0]
    # 28 bytes for every piece there is room for: two a wire slot and 1024; the pieces
    # themselves are far fewer, so half of that is more than a second walk takes
    records = 28 * (2 * (len(res.entries) + len(res.keys)) + 1024)
    for part in (0.05, 0.5):  # no room for the outputs beside the records; none for the records
        with pk.Context(0, hbm_budget=int(used - part * records)) as c, pk.Job(c) as job:
            _compacted(job, rs, k, 20, threshold, 6)
            assert job.walk() == want
            assert job.walk() == want  # again, on the buffers that the first one left


@pytest.mark.parametrize("k,genome,reads,err,threshold", [(32, 3000, 8000, 0.01, 400), (63, 300, 4000, 0.005, 100)])
def test_compacted_map_with_more_pieces_than_records(k, genome, reads, err, threshold):
    rs = synth.small_case(9, genome_len=genome, n_reads=reads, read_len=100, k=k, coverage=1, err=err)
    with pk.Job(ctx()) as job:
        mn, res = _compacted(job, rs, k, 1, threshold, 21)
        assert res.rounds > 0
        assert job.walk() == _walk(mn, k, 1, threshold)
