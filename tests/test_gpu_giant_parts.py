"""A giant bucket is counted by sixteen parts, each a remainder range between quantiles of the
bucket's entries: few entries (one part takes all), just above that, many ranges that split
again, chunks with too many distinct keys, and samples that are one heavy key.  One read per
k-mer window, two partition digits; compared with the oracle."""
import numpy as np
import pytest

from gpu_helpers import assert_mn_equal, assert_table_equal, run_gpu
from oracle import pk_oracle as po

pytestmark = pytest.mark.gpu


def _reads(rows):
    out = np.empty((rows.shape[0], 3 + rows.shape[1] + 1), np.uint8)
    out[:, :3] = np.frombuffer(b">r\n", np.uint8)
    out[:, 3:-1] = np.frombuffer(b"ACTG", np.uint8)[rows]
    out[:, -1] = 10
    return out.tobytes()


@pytest.mark.parametrize("k", [31, 32, 63])
@pytest.mark.parametrize("distinct,heavy", [(1, 0.0), (200, 0.0), (300, 0.5), (4097, 0.0), (30_000, 0.999), (60_000, 0.0),
                                            (300_000, 0.1)])
def test_giant_bucket_parts(k, distinct, heavy):
    rng = np.random.Generator(np.random.PCG64(distinct + k))
    keys = rng.integers(0, 4, (distinct, k), dtype=np.uint8)
    keys[:, 0] = 0  # one of the four buckets
    keys[: distinct // 2, 1:k - 9] = 0  # half of the keys crowd a corner of the key range
    n = 16 * 32768 + 12_345  # windows: sixteen chunks and a tail
    pick = rng.integers(0, distinct, n)
    pick[rng.random(n) < heavy] = distinct - 1
    pick[:distinct] = np.arange(distinct)
    other = rng.integers(0, 4, (5000, k), dtype=np.uint8)
    other[:, 0] = 1 + other[:, 0] % 3
    rows = np.concatenate([keys[pick], other])
    fa = _reads(rows[rng.permutation(rows.shape[0])])
    ora = po.run(fa, k, 21)
    s, tk, tc, hist, mn, err = run_gpu(fa, k, 21, 10, bucket_bits=2)
    assert_table_equal(tk, tc, ora.table.keys, ora.table.counts)
    assert s.cutoff == ora.cutoff
    if ora.mn is not None:
        assert np.array_equal(hist, ora.hist)
        assert_mn_equal(mn, ora.mn.keys, ora.mn.suf, ora.mn.pre)
