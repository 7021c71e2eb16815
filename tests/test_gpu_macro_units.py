"""Macro-node units at the edges of the kernel's paths: joined units up to 768 rows a side
with 0 to 32 nodes that only a prefix side names, sorted units of one segment, and units of
several segments counted ahead; against the oracle."""
import numpy as np
import pytest

import pakman_plus_gb300 as pk
from gpu_helpers import assert_mn_equal, ctx
from oracle import pk_oracle as po

pytestmark = pytest.mark.gpu


def _table(k, chain, loose, seed):
    """Rows of `chain` consecutive k-mers of a random sequence and `loose` isolated ones."""
    rng = np.random.Generator(np.random.PCG64(seed))
    mask = (1 << (2 * k)) - 1
    bases = rng.integers(0, 4, chain + k - 1)
    keys, x = set(), 0
    for i, b in enumerate(bases):
        x = ((x << 2) | int(b)) & mask
        if i >= k - 1:
            keys.add(x)
    while len(keys) < chain + loose:
        keys.add(int.from_bytes(rng.bytes(16), "little") & mask)
    rows = sorted(keys)
    out = np.zeros(len(rows), pk.KEY128)
    out["lo"] = np.array([r & ((1 << 64) - 1) for r in rows], np.uint64)
    out["hi"] = np.array([r >> 64 for r in rows], np.uint64)
    return out, rng.integers(1, 200, len(rows), dtype=np.uint32)


@pytest.mark.parametrize("k", [21, 32, 63])
@pytest.mark.parametrize("chain,loose", [(1, 0), (60, 2), (400, 0), (400, 31), (400, 33), (3000, 4), (3060, 0),
                                         (3080, 40), (3080, 120), (3080, 180), (6100, 0), (6300, 9),
                                         (20_000, 50), (0, 700), (0, 9000)])
@pytest.mark.parametrize("units", [0, 1, 2])
def test_units_of_every_size(k, chain, loose, units):
    """Four buckets (2 digits); mn_units 1: four units, 2: one unit of all rows."""
    keys, counts = _table(k, chain, loose, 7 * chain + loose + k)
    p = pk.default_params(k=k, num_buckets=2, bucket_bits=2, mn_units=units)
    with pk.Job(ctx()) as job:
        job.load_table(keys["lo"].copy() if k <= 32 else keys, counts, p)
        job.cutoff(1)
        m = job.build_macro_nodes(0)
        mn = job.macro_nodes(1)
    ref = po.macro_nodes(po.Table(keys, counts, 0, 0), k, 1)
    assert m == ref.keys.size
    assert_mn_equal(mn, ref.keys, ref.suf, ref.pre)
