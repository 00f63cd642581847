"""Walk kernels at the edges of their routes: a thread per walk (unbiased; many
biased walks) with walks that end inside, at and after the eight kept steps,
the warp walk's search at one tile, up to 1024 edges and beyond, and unbiased
walks that read columns and row offsets instead of records.  Edges equal the
oracle's exactly."""
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


def check(csaw, G, g, bias, n, length, seed, kind):
    import torch
    seeds = oracle.make_seeds(g.rowptr, n, seed)
    p = csaw.make_params(1, bias, n, 1, 1, length, None, seed, schedule=csaw.SCHED_BATCHED, sample_base=3)
    G.profile(True)
    out = [x.cpu().numpy() for x in G.sample(p, torch.from_numpy(seeds).cuda())]
    assert G.kernel_stats(kind)["launches"] == 1
    G.profile(False)
    ref = oracle.run(g.rowptr, g.col, g.weight, seeds, 1, bias, n, 1, length, None, seed=seed, n_threads=8,
                     sample_base=3)
    a, b = sort_edges(*out), sort_edges(*ref)
    assert a.shape == b.shape and np.array_equal(a, b), (bias, n, length)
    return len(out[0])


@pytest.mark.parametrize("rowptr64", [False, True])
@pytest.mark.parametrize("length", [1, 7, 8, 9, 16, 17, 33])
def test_thread_walks_keep_eight_steps(csaw, powerlaw_small, rmat12_pareto, rowptr64, length):
    for g in (powerlaw_small, rmat12_pareto):
        G = csaw.Graph(g, rowptr64=rowptr64)
        check(csaw, G, g, 0, 1037, length, 40 + length, "walk_thread")
        check(csaw, G, g, 2, 15_001, length, 41 + length, "walk_thread")
        check(csaw, G, g, 1, 203, length, 42 + length, "walk")
        G.close()


@pytest.mark.parametrize("rowptr64", [False, True])
@pytest.mark.parametrize("bias", [1, 2, 3])
def test_walks_through_hubs(csaw, skewed_hubs, rowptr64, bias):
    """Rows of 600 to 50,000 edges and walks that die on vertices without
    edges (the power-law base has rows of one edge up)."""
    g = skewed_hubs
    G = csaw.Graph(g, rowptr64=rowptr64)
    check(csaw, G, g, bias, 3001, 40, 7, "walk")
    check(csaw, G, g, bias, 20_000, 12, 8, "walk_thread")
    G.close()


@pytest.mark.parametrize("rowptr64", [False, True])
def test_walks_by_column(csaw, rowptr64):
    """Records above the L2 size, row offsets below, many unbiased walks."""
    from csaw import graphgen
    V, E = 1 << 16, 9_000_000
    rng = np.random.default_rng(5)
    deg = rng.multinomial(E, np.full(V, 1.0 / V))
    deg[:100] = 0   # some walks end
    rowptr = np.concatenate([[0], np.cumsum(deg)])
    g = graphgen.CSR(rowptr, rng.integers(0, V, int(rowptr[-1])), None, name="wide")
    G = csaw.Graph(g, rowptr64=rowptr64)
    check(csaw, G, g, 0, 120_001, 5, 9, "walk_thread")
    G.close()
