"""A table merged from pieces is partitioned as the same table loaded is: macro-node
construction then has the same units, and asks for the same memory."""
import pytest

import pakman_plus_gb300 as pk
from pakman_plus_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [32, 63])
def test_merged_and_loaded_tables_are_partitioned_alike(k):
    rs = synth.small_case(21, genome_len=60_000, n_reads=24_000, read_len=100, k=k, coverage=20, err=0.002)
    with pk.Context(0, hbm_budget=8 << 30) as c:
        def built(job):  # bytes that macro-node construction adds
            job.cutoff(6)
            before = c.memory()[0]
            job.build_macro_nodes(0)
            return c.memory()[0] - before, job.macro_nodes(20)

        with pk.Job(c) as job:
            job.count(rs.fasta, pk.default_params(k=k, chunking=1, batch_kmers=len(rs.fasta) // 5))
            merged, mn = built(job)
            keys, counts = job.table()
        assert len(keys) > 20_000
        with pk.Job(c) as job:
            job.load_table(keys, counts, pk.default_params(k=k))
            loaded, mn2 = built(job)
    assert merged == loaded
    assert (mn.keys == mn2.keys).all()
