"""The walk where the counting walk has room to record its contigs and where it has not (the
pieces of many deep walks outnumber the map's wires), against the oracle."""
import pytest

import pakman_plus_gb300 as pk
from gpu_helpers import ctx
from oracle import pk_compact as pc
from pakman_plus_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [32, 63])
@pytest.mark.parametrize("cov,threshold,recorded", [(20, 1 << 20, True), (20, 40, True), (1, 1 << 20, False)])
def test_walk_with_and_without_records(k, cov, threshold, recorded):
    rs = synth.small_case(9, genome_len=3000, n_reads=4000, read_len=100, k=k, coverage=cov, err=0.003)
    with pk.Job(ctx()) as job:
        job.count(rs.fasta, pk.default_params(k=k, coverage=cov))
        job.cutoff(21)
        job.build_macro_nodes(0)
        mn = job.macro_nodes(cov)
        res = job.compact(threshold, cov)
        walks = job.walk()
    nodes = pc.compact(pc.initial_nodes(mn.keys, mn.suffix_counts, mn.prefix_counts, k, cov), k, threshold).nodes
    assert walks == pc.walk(nodes, k)
    if res.rounds == 0:  # uncompacted: a piece is one base
        entries = sum(len(nd.suf) + len(nd.pre) for nd in nodes)
        pieces = sum(len(c) - (k - 1) for c in walks)
        assert recorded == (pieces <= 2 * (entries + len(nodes)) + 1024)
