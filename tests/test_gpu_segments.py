"""Counting pass and coarse scatter at the edges of their 16-byte units, 64-byte segments and
64 KiB tiles: records of every length, N and '\\r' bytes anywhere, junk before the first
record; the whole table against the oracle."""
import numpy as np
import pytest

import pakman_plus_gb300 as pk
from gpu_helpers import assert_table_equal, ctx
from oracle import pk_oracle as po

pytestmark = pytest.mark.gpu


def _reads(seed, junk, longest):
    rng = np.random.Generator(np.random.PCG64(seed))
    out, size = [(b"ab\n" * (junk // 3 + 1))[:junk]], junk
    genome = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, 4000)]
    i = 0
    while size < 200_000:
        n = int(rng.integers(0, longest))
        at = int(rng.integers(0, genome.size - n + 1))
        r = genome[at:at + n].copy()
        kind = i % 5
        if kind == 1 and n:  # a run of N
            a = int(rng.integers(0, n))
            r[a:a + int(rng.integers(1, 40))] = ord("N")
        elif kind == 2:  # scattered N and lowercase
            r = np.where(rng.random(n) < 0.05, ord("N"), r | 0x20).astype(np.uint8)
        body = r.tobytes() + (b"\r" if kind == 3 else b"")
        rec = b">" + b"h" * int(rng.integers(0, 70)) + b"\n" + body + b"\n"
        out.append(rec)
        size += len(rec)
        i += 1
    return b"".join(out)[: -1 if seed % 2 else None]


@pytest.mark.parametrize("drop_n", [False, True])
@pytest.mark.parametrize("k", [2, 5, 15, 16, 17, 21, 31, 32, 33, 47, 48, 49, 63, 64])
def test_tables_over_ragged_records(k, drop_n):
    for junk, longest in ((0, 130), (1, 400), (63, 40 + k), (64, 90), (65, 3000), (70_000, 150)):
        fa = _reads(1000 * k + junk, junk, longest)
        ora = po.count(fa, k, drop_n)
        with pk.Job(ctx()) as job:
            job.count(fa, pk.default_params(k=k, drop_n=int(drop_n)))
            keys, counts = job.table()
            assert job.table_info()[1] == ora.n_windows
        assert_table_equal(pk.to_key128(keys), counts, ora.keys, ora.counts)
