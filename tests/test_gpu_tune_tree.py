"""The autotuner beside the one-launch route of small neighbor jobs: its
candidates and its choice shape the launches that have a shape, and jobs whose
sample trees run in one launch keep that route."""
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


def job(csaw, g, n, F, fan, seed):
    import torch
    sd = torch.from_numpy(oracle.make_seeds(g.rowptr, n * F, seed)).cuda()
    p = csaw.make_params(0, 2, n, F, fan[0], len(fan), fan, seed, schedule=csaw.SCHED_BATCHED)
    return csaw.BatchJob(p, sd)


def edges(res):
    return [sort_edges(*[x.cpu().numpy() for x in r]) for r in res]


def launches(G, call):
    """Launches by kind of one call."""
    G.profile(True)
    before = {k: G.kernel_stats(k)["launches"] for k in ("tree", "expand")}
    out = call()
    after = {k: G.kernel_stats(k)["launches"] for k in before}
    G.profile(False)
    return out, after["tree"] - before["tree"], after["expand"] - before["expand"]


def test_tuned_shape_leaves_small_jobs_in_one_launch(csaw, rmat12_pareto):
    from csaw import _lib
    g = rmat12_pareto
    G = csaw.Graph(g)
    small, large = job(csaw, g, 300, 2, [10, 5, 3], 31), job(csaw, g, 6000, 2, [10, 5, 3], 32)
    ref = edges(G.sample_batch([small, large]))
    r, tree, expand = launches(G, lambda: G.autotune([small, large]))
    assert tree == 2 * r["candidates"] and expand > 0   # an untimed and a timed run of each
    res, tree, expand = launches(G, lambda: edges(G.sample_batch([small, large])))
    assert tree == 1
    assert all(np.array_equal(a, b) for a, b in zip(res, ref))
    # a shape the caller sets keeps its launches, until it is the default again
    for opt, other, default in ((_lib.OPT_GRID_PCT, 50, 100), (_lib.OPT_PAIR, 0, 1)):
        G.set_option(opt, other)
        res, tree, expand = launches(G, lambda: edges(G.sample_batch([small])))
        assert tree == 0 and np.array_equal(res[0], ref[0])
        G.set_option(opt, default)
        res, tree, expand = launches(G, lambda: edges(G.sample_batch([small])))
        assert tree == 1 and expand == 0 and np.array_equal(res[0], ref[0])
    G.close()


def test_a_batch_without_shaped_launches_keeps_the_default(csaw, rmat12_pareto):
    g = rmat12_pareto
    G = csaw.Graph(g)
    jobs = [job(csaw, g, 300, 2, [10, 5, 3], 33)]
    r, tree, expand = launches(G, lambda: G.autotune(jobs))
    assert tree == 2 * r["candidates"] and expand == 0
    assert (r["grid_pct"], r["pair"], r["persistent"]) == (100, 1, 0) and r["best_ms"] == r["default_ms"]
    G.close()
