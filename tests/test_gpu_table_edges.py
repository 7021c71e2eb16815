"""The table kernel at the edges of its on-chip tables: buckets below, at and above half the
slots (smaller tables retried at full size, then split), bins crowded enough for the
bitonic order, and heavy keys among them.  One read per k-mer window, so the keys and
counts of every bucket are chosen exactly; compared with the oracle."""
import numpy as np
import pytest

import pakman_plus_gb300 as pk
from gpu_helpers import assert_mn_equal, assert_table_equal, run_gpu
from oracle import pk_oracle as po

pytestmark = pytest.mark.gpu


def _fasta(keys, copies, k, rng):
    """One read of exactly k bases per key copy, in random order."""
    sh = [2 * (k - 1 - i) for i in range(k)]
    acgt = np.frombuffer(b"ACTG", np.uint8)  # base codes 0..3
    rows = np.array([[acgt[(int(x) >> s) & 3] for s in sh] for x in keys], np.uint8)
    rows = rows[rng.permutation(np.repeat(np.arange(len(keys)), copies))]
    head = np.frombuffer(b">r\n", np.uint8)
    out = np.empty((rows.shape[0], 3 + k + 1), np.uint8)
    out[:, :3] = head
    out[:, 3:3 + k] = rows
    out[:, -1] = 10
    return out.tobytes()


@pytest.mark.parametrize("k", [15, 32, 63])
@pytest.mark.parametrize("distinct", [1, 2, 511, 513, 2047, 2049, 4095, 4097, 9000])
@pytest.mark.parametrize("dense", [False, True])
def test_distinct_keys_around_the_table_size(k, distinct, dense):
    """Four buckets (2 digits), one with `distinct` keys: spread over the key range, or
    consecutive (one crowded sort bin); a few heavy keys among them."""
    rng = np.random.Generator(np.random.PCG64(distinct * 131 + k + dense))
    top = 1 << (2 * k - 2)
    if dense:
        base = int(rng.integers(0, 1 << 16))
        keys = [base + 3 * i for i in range(distinct)]
    else:
        keys = sorted({int.from_bytes(rng.bytes(16), "little") % top for _ in range(distinct)})
    keys += [top, 2 * top + 5, 4 * top - 1]  # the other buckets hold one key each
    copies = rng.integers(1, 4, len(keys))
    copies[:: max(1, len(keys) // 3)] = 700
    fa = _fasta(keys, copies, k, rng)
    ora = po.run(fa, k, 21)
    s, tk, tc, hist, mn, err = run_gpu(fa, k, 21, 10, bucket_bits=2)
    assert_table_equal(tk, tc, ora.table.keys, ora.table.counts)
    assert s.cutoff == ora.cutoff
    if ora.mn is not None:
        assert np.array_equal(hist, ora.hist)
        assert_mn_equal(mn, ora.mn.keys, ora.mn.suf, ora.mn.pre)


def test_counts_at_the_histogram_edges():
    """Counts on both sides of the on-chip histograms (16 and 512) with a large -t."""
    k, rng = 31, np.random.Generator(np.random.PCG64(5))
    copies = np.array([1, 15, 16, 17, 511, 512, 513, 1023, 1024, 1500])
    keys = sorted(int(x) for x in rng.integers(0, 1 << 62, copies.size, dtype=np.uint64))
    fa = _fasta(keys, copies, k, rng)
    ora = po.run(fa, k, 2000)
    with pk.Job(pk.Context(0)) as job:
        job.count(fa, pk.default_params(k=k, num_buckets=2000))
        cut, hist, kept = job.cutoff(2000)
    assert cut == ora.cutoff and np.array_equal(hist, ora.hist)
