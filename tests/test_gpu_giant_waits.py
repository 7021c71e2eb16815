"""The parts of a giant bucket write their rows one after the other, so the last of many long
parts waits far longer than a wait's poll limit: that limit is for a wait in which nothing
moves.  Two partition digits, all keys of a bucket distinct: each of its sixteen parts has a
dozen sub-ranges or more, some milliseconds, against a limit of 2000 polls (a millisecond or
two)."""
import numpy as np
import pytest

import pakman_plus_gb300 as pk
from gpu_helpers import assert_table_equal, ctx
from oracle import pk_oracle as po

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [32, 63])
@pytest.mark.parametrize("buckets", [1, 4])  # 16 and 64 parts
def test_long_parts_outlast_the_poll_limit(k, buckets):
    rng = np.random.Generator(np.random.PCG64(k + buckets))
    n = 600_000  # windows of a bucket, one a read
    rows = np.empty((n * buckets, 3 + k + 1), np.uint8)
    bases = rng.integers(0, 4, (n * buckets, k), dtype=np.uint8)
    bases[:, 0] = np.arange(n * buckets) % buckets
    rows[:, :3] = np.frombuffer(b">r\n", np.uint8)
    rows[:, 3:-1] = np.frombuffer(b"ACTG", np.uint8)[bases]
    rows[:, -1] = 10
    fa = rows.tobytes()
    ora = po.run(fa, k, 21)
    with pk.Job(ctx()) as job:
        job.set_wait_limit(spins=2000)
        job.count(fa, pk.default_params(k=k, bucket_bits=2))
        keys, counts = job.table()
    assert_table_equal(pk.to_key128(keys), counts, ora.table.keys, ora.table.counts)
