"""Solves on several streams and threads at once -- cooperative launches beside
one another and beside multigrid loops -- end as they do alone."""
import threading

import numpy as np
import pytest
import torch

import test_gpu_coop as coop
from conftest import rng, seed_of
from test_gpu_ops import cells, host, make_grid

pytestmark = pytest.mark.gpu


def double_cg(pg, oracle, dims, out):
    """The reference's CG in doubles: x and the iterations of every solve."""
    g, b = coop.problem(pg, oracle, dims)
    torch.cuda.synchronize()

    def run(times):
        for _ in range(times):
            st, v = coop.solve(pg, g, b, 1, 40, 1e-9)
            out.append((st["status"], st["iterations"], v[0]))

    return run


def multigrid(pg, dims, out):
    g = make_grid(pg, dims)
    b = rng(seed_of(dims, "streams")).standard_normal(dims).astype(np.float32)
    b, x = cells(pg, g, b - b.mean()), g.new_simplex_2()
    torch.cuda.synchronize()
    cfg = pg.SolverConfig(precond=2, rel_stop=True, rel_tol=1e-5, max_iter=50, refine=3)

    def run(times):
        for _ in range(times):
            st = pg.solve_pressure(g, x, b, 0.5, cfg)
            out.append((st["status"], st["iterations"], host(x)))

    return run


def test_threads_with_their_own_streams(pg, oracle):
    jobs, outs = [], []
    for dims, double in (((128, 128), 1), ((384, 380), 1), ((64, 64, 64), 1), ((256, 256), 0), ((64, 64, 64), 0)):
        outs.append([])
        run = double_cg(pg, oracle, dims, outs[-1]) if double else multigrid(pg, dims, outs[-1])
        jobs.append((run, torch.cuda.Stream()))
    for run, stream in jobs:  # alone
        with torch.cuda.stream(stream):
            run(1)
    want = [o.pop() for o in outs]

    def work(run, stream):
        with torch.cuda.stream(stream):
            run(20)

    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    for (status, iterations, x), out in zip(want, outs):
        assert len(out) == 20
        for s, i, v in out:
            assert (s, i) == (status, iterations)
            assert np.array_equal(v, x)
