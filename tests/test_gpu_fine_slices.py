"""The fine scatter at the edges of its slices (2048 or 8192 64-bit keys, half as many 128-bit
ones) and of the fan-out at which it changes slice size (2^7 fine buckets per coarse region,
that is 14 partition digits), regions empty, of one slice and of several; compared with the
oracle."""
import numpy as np
import pytest

from gpu_helpers import assert_table_equal, run_gpu
from oracle import pk_oracle as po

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [21, 32, 63])
@pytest.mark.parametrize("bits", [2, 7, 8, 13, 14, 15, 16])
@pytest.mark.parametrize("n", [1, 1023, 1024, 1025, 2048, 2049, 8193, 40_000])
def test_slices(k, bits, n):
    rng = np.random.Generator(np.random.PCG64(n * 64 + bits))
    rows = rng.integers(0, 4, (n + n // 3, k), dtype=np.uint8)
    rows[:n, :4] = 2  # n keys of one coarse region, the others anywhere
    out = np.empty((rows.shape[0], k + 4), np.uint8)
    out[:, :3] = np.frombuffer(b">r\n", np.uint8)
    out[:, 3:-1] = np.frombuffer(b"ACTG", np.uint8)[rows[rng.permutation(rows.shape[0])]]
    out[:, -1] = 10
    fa = out.tobytes()
    ora = po.run(fa, k, 21)
    s, tk, tc, hist, mn, err = run_gpu(fa, k, 21, 10, bucket_bits=bits)
    assert_table_equal(tk, tc, ora.table.keys, ora.table.counts)
    assert s.cutoff == ora.cutoff
