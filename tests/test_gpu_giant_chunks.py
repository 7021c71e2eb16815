"""Chunks of a giant bucket around the size from which they stay keys: half a table of distinct
keys, that is 2048 of 8192 keys (k > 32) or 4096 of 32768.  A heavy key and its unique company,
a little fewer, as many and a little more; compared with the oracle."""
import numpy as np
import pytest

from gpu_helpers import assert_table_equal, run_gpu
from oracle import pk_oracle as po

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,limit", [(32, 4096 / 32768), (33, 2048 / 8192), (63, 2048 / 8192)])
@pytest.mark.parametrize("share", [0.9, 1.0, 1.1])
@pytest.mark.parametrize("n", [524_288, 532_479, 700_001])  # whole chunks, all but a key of one, a tail
def test_chunks_around_half_a_table(k, limit, share, n):
    rng = np.random.Generator(np.random.PCG64(n + k))
    rows = rng.integers(0, 4, (n, k), dtype=np.uint8)
    rows[rng.random(n) >= share * limit] = 0
    rows[:, 0] = 0  # one of four buckets
    fa = np.empty((n, 3 + k + 1), np.uint8)
    fa[:, :3] = np.frombuffer(b">r\n", np.uint8)
    fa[:, 3:-1] = np.frombuffer(b"ACTG", np.uint8)[rows]
    fa[:, -1] = 10
    ora = po.run(fa.tobytes(), k, 21)
    s, tk, tc, hist, mn, err = run_gpu(fa.tobytes(), k, 21, 10, bucket_bits=2)
    assert s.n_windows == n
    assert_table_equal(tk, tc, ora.table.keys, ora.table.counts)
