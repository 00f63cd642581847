"""Counter blocks between jobs that read their own counters back (sample
trees, walks, MDRW), jobs of several kernels, captured batches, host-buffer
jobs and failed jobs on the same contexts: every job's edge count is its own."""
import numpy as np
import pytest

import oracle
from conftest import sort_edges

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def csaw():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("gpu test without a CUDA device")
    import csaw as c
    c.lib()
    return c


def test_counts_across_routes(csaw, skewed_hubs):
    import torch
    g = skewed_hubs
    G = csaw.Graph(g)
    specs = [   # mode, bias, samples, frontier, depth, fan-out, schedule
        (0, 2, 50, 1, 2, [10, 4], 1), (1, 2, 700, 1, 9, None, 1), (2, 1, 90, 5, 6, None, 1), (2, 1, 20, 40, 6, None, 1),
        (1, 0, 300, 1, 12, None, 1), (0, 0, 60, 2, 2, [5, 5], 0), (0, 2, 40, 1, 2, [6, 3], 0), (1, 2, 100, 1, 5, None, 0),
        (0, 1, 9000, 8, 2, [6, 3], 1),
    ]
    jobs, refs, seeds = [], [], []
    for k, (mode, bias, n, F, depth, fan, sched) in enumerate(specs):
        s = oracle.make_seeds(g.rowptr, n * F, 60 + k)
        p = csaw.make_params(mode, bias, n, F, (fan or [1])[0], depth, fan, 900 + k, schedule=sched)
        jobs.append(csaw.BatchJob(p, torch.from_numpy(s).cuda()))
        seeds.append(s)
        refs.append(sort_edges(*oracle.run(g.rowptr, g.col, g.weight, s, mode, bias, n, F, depth, fan, seed=900 + k,
                                           n_threads=8)))

    def same(res, ks):
        for r, k in zip(res, ks):
            got = sort_edges(*[x.cpu().numpy() if hasattr(x, "cpu") else x for x in r])
            assert got.shape == refs[k].shape and np.array_equal(got, refs[k]), k

    order = list(range(len(specs)))
    for k in order + order[::-1] + [0, 0, 1, 1]:            # one context, every route after every other
        same([G.sample(jobs[k].params, jobs[k].seeds)], [k])
    a, b, c = [0, 1, 2], [4, 8, 5], [3, 7, 6]
    for ks in (a, a, a, b, a, c, a, b, b, b, a, c, b):      # eager, captured and replayed batches on the same contexts
        same(G.sample_batch([jobs[k] for k in ks]), ks)
    with pytest.raises(csaw.CsawError):
        G.sample(jobs[1].params, jobs[1].seeds, capacity=3)
    same([G.sample(jobs[4].params, jobs[4].seeds)], [4])
    for k in (1, 0, 8, 4):                                  # host buffers, then device buffers again
        same([G.sample_host(jobs[k].params, seeds[k])], [k])
        same(G.sample_batch([jobs[k]]), [k])
    G.close()
