"""Loaded tables (pk_table_load), whose rows are checked and histogrammed on the device."""
import numpy as np
import pytest

import pakman_plus_gb300 as pk
from gpu_helpers import ctx
from oracle import pk_oracle as po

pytestmark = pytest.mark.gpu


def _rows(n, k, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    top = np.unique(rng.integers(1, 1 << 62, n + 8, dtype=np.uint64))[:n]
    counts = rng.integers(1, 40, n, dtype=np.uint32)
    if k <= 32:
        return top, counts
    keys = np.zeros(n, pk.KEY128)  # every other row shares its high word with the row before
    keys["hi"] = top
    keys["hi"][1::2] = keys["hi"][:n - 1:2]
    keys["lo"] = rng.integers(0, 1 << 63, n, dtype=np.uint64)
    keys["lo"][1::2] |= np.uint64(1 << 63)
    return keys, counts


@pytest.mark.parametrize("k", [31, 63])
@pytest.mark.parametrize("n", [1, 2, 255, 256, 257, 4999, 400_003])
def test_loaded_table_histogram_and_bad_rows(k, n):
    """Histogram and window total of a loaded table at every -t, and the first bad row
    named for each rule; a refused table leaves the one before it in place."""
    keys, counts = _rows(n, k, 7 * n + k)
    with pk.Job(ctx()) as job:
        job.load_table(keys, counts, pk.default_params(k=k, num_buckets=21))
        for t in (21, 2, 40, 5000):
            try:
                cut, hist, kept = job.cutoff(t)
            except pk.EmptyAfterCutoff as e:
                cut, hist, kept = e.cutoff, e.hist, e.kept
            ref, rcut = po.cutoff(counts, t)
            assert cut == rcut and np.array_equal(hist, ref) and kept == int((counts >= cut).sum())
        assert job.table_info()[:2] == (n, int(counts.sum()))
        for row in sorted({0, n // 2, n - 1}):
            bad = counts.copy()
            bad[row] = 0
            with pytest.raises(pk.PakmanError, match=f"row {row} has count 0"):
                job.load_table(keys, bad, pk.default_params(k=k))
            if row:
                twice = keys.copy()
                twice[row] = twice[row - 1]
                with pytest.raises(pk.PakmanError, match=rf"ascending and unique \(row {row}\)"):
                    job.load_table(twice, counts, pk.default_params(k=k))
            big = keys.copy()
            if k <= 32:
                big[row] = np.uint64(1) << np.uint64(2 * k)
            else:
                big["hi"][row] = np.uint64(1) << np.uint64(2 * k - 64)
            with pytest.raises(pk.PakmanError, match=f"row {row} is not a k-mer"):
                job.load_table(big, counts, pk.default_params(k=k))
        k2, c2 = job.table()
        assert np.array_equal(k2, keys) and np.array_equal(c2, counts)
