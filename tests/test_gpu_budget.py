"""What a context holds on the device -- blocks in use and idle ones kept for later -- stays
within its HBM budget, whichever part of the library allocates, and what its buffers ask for
exactly fits a budget of just that."""
from contextlib import ExitStack

import numpy as np
import pytest
import torch

import pakman_plus_gb300 as pk
from gpu_helpers import ctx

pytestmark = pytest.mark.gpu

MB = 1 << 20
# what a process allocates besides the buffers (streams, events, graphs) and the granularity
# of the driver's pool; the kernels are loaded before the first reading
SLACK = 96 * MB


def _reads(n, seed=1):
    rng = np.random.Generator(np.random.PCG64(seed))
    rows = np.empty((n, 104), np.uint8)
    rows[:, :3] = np.frombuffer(b">r\n", np.uint8)
    genome = np.frombuffer(b"ACTG", np.uint8)[rng.integers(0, 4, 1_000_000)]
    rows[:, 3:103] = genome[rng.integers(0, genome.size - 100, n)[:, None] + np.arange(100)]
    rows[:, 103] = 10
    return rows.reshape(-1)


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _warm(fasta, p):
    with pk.Job(ctx()) as job:
        job.run(fasta, p)
    with pk.Batch(ctx(), branches=1) as b:
        b.run([(fasta, p)])


def test_batch_after_a_job_stays_within_the_budget():
    p = pk.default_params(k=32, num_buckets=3)
    big, small = _reads(520_000), _reads(40_000)
    _warm(small, p)
    budget = 1024 * MB
    free = _free()
    with pk.Context(0, hbm_budget=budget) as c:
        with pk.Job(c) as job:
            job.count(big, p)
            assert c.memory()[0] > 600 * MB  # most of it idle, and kept, when the job is gone
        with pk.Batch(c, branches=1) as batch:  # input and output of 40 sets: another 600 MB
            res = batch.run([(small, p)] * 40)
            assert all(r.status == 0 for r in res)
            assert 500 * MB < c.memory()[0] <= budget
            assert free - _free() <= budget + SLACK


def test_smaller_jobs_after_larger_ones_stay_within_the_budget():
    p = pk.default_params(k=32, num_buckets=3)
    sizes = [640_000, 585_000]  # buffers a tenth smaller: within what a kept block may be larger
    fa = [_reads(n) for n in sizes]
    _warm(_reads(40_000), p)
    need = []
    for f in fa:  # with a budget, what is in use is what the buffers asked for
        with pk.Context(0, hbm_budget=8192 * MB) as c, pk.Job(c) as job:
            job.count(f, p)
            need.append(c.memory()[0])
    n = 4
    budget = (n + 1) * need[1]
    assert n * need[0] <= budget
    free = _free()
    with pk.Context(0, hbm_budget=budget) as c:
        with ExitStack() as jobs:
            for _ in range(n):
                jobs.enter_context(pk.Job(c)).count(fa[0], p)
        with ExitStack() as jobs:
            for _ in range(n + 1):  # the budget exactly
                jobs.enter_context(pk.Job(c)).count(fa[1], p)
            used, held = c.memory()[0], free - _free()
    assert used == budget
    assert held <= budget + SLACK
