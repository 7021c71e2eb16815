"""Wiring of exactly sized node tables, at the edges of the kernel's CTAs."""
import numpy as np
import pytest

import pakman_plus_gb300 as pk
from gpu_helpers import ctx
from oracle import pk_oracle as po

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 3, 127, 129, 255, 257, 5001])
def test_wiring_at_tile_edges(m):
    """m macro-nodes: (m - 1) / 2 isolated k-mers (two nodes each) and the all-A k-mer,
    whose two nodes are one."""
    k = 31
    rng = np.random.Generator(np.random.PCG64(m))
    keys = np.concatenate([[np.uint64(0)], np.unique(rng.integers(1 << 40, 1 << 62, 4 * m + 8, dtype=np.uint64))])
    keys = np.concatenate([keys[:1], np.sort(rng.permutation(keys[1:])[:(m - 1) // 2])])
    counts = rng.integers(1, 1000, keys.size, dtype=np.uint32)
    with pk.Job(ctx()) as job:
        job.load_table(keys, counts, pk.default_params(k=k, num_buckets=1))
        job.cutoff(1)
        assert job.build_macro_nodes(0) == m
        mn = job.macro_nodes(9)
        w = job.wire(9)
    ref = po.wire(mn.suffix_counts, mn.prefix_counts, 9)
    for f in ("ns", "np", "term_suf", "term_pre", "nw", "wire", "begin"):
        assert np.array_equal(w[f], ref[f]), f
