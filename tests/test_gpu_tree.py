"""Whole sample trees in one launch (small and middle neighbor jobs): the same
edges as the oracle and as the per-level passes, where the two can differ --
one sample, ragged chunks, levels of one item and of more than a warp's or a
CTA's items, the widest trees it takes, hubs whose first phase fails, 64-bit
row offsets, every bias, the plain unbiased schedule -- and the same errors."""
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


def hub_seeds(g, n, seed):
    hubs = np.argsort(np.diff(g.rowptr))[-min(n, 12):].astype(np.int32)
    return np.concatenate([hubs, oracle.make_seeds(g.rowptr, n - hubs.size, seed)]).astype(np.int32)


SHAPES = [   # samples, frontier, fan-out
    (1, 1, [1]), (1, 1, [32]), (1, 3, [25, 10]), (149, 1, [25, 10]), (1500, 1, [10, 4]), (4003, 1, [3, 2]),
    (37, 33, [16, 3]), (5, 4, [20, 20, 2]), (3, 64, [16, 2, 2]), (40, 1, [2, 2, 2, 2, 2, 2, 2, 2]), (2, 2048, [2]),
]


@pytest.mark.parametrize("which", ["skewed_hubs", "powerlaw_small", "rmat12_pareto"])
@pytest.mark.parametrize("rowptr64", [False, True])
@pytest.mark.parametrize("bias,schedule", [(0, 0), (0, 1), (1, 1), (2, 1), (2, 2), (3, 1)])
def test_tree_equals_oracle_and_levels(csaw, request, which, rowptr64, bias, schedule):
    import torch
    from csaw import _lib
    g = request.getfixturevalue(which)
    G = csaw.Graph(g, rowptr64=rowptr64)
    for k, (n, F, fan) in enumerate(SHAPES):
        seed = 0x7E0 + 16 * k + bias
        seeds = hub_seeds(g, n * F, seed)
        sd = torch.from_numpy(seeds).cuda()
        p = csaw.make_params(0, bias, n, F, fan[0], len(fan), fan, seed, schedule=schedule, sample_base=11)
        G.set_option(_lib.OPT_GRID_PCT, 100)
        G.profile(True)
        out = [x.cpu().numpy() for x in G.sample(p, sd)]
        assert G.kernel_stats("tree")["launches"] == 1, (n, F, fan)
        G.profile(False)
        got = sort_edges(*out)
        ref = oracle.run(g.rowptr, g.col, g.weight, seeds, 0, bias, n, F, len(fan), fan, seed=seed, n_threads=8,
                         sample_base=11)
        want = sort_edges(*ref)
        assert got.shape == want.shape and np.array_equal(got, want), (n, F, fan)
        G.set_option(_lib.OPT_GRID_PCT, 50)   # a launch shape of the per-level passes
        lev = sort_edges(*[x.cpu().numpy() for x in G.sample(p, sd)])
        assert np.array_equal(got, lev), (n, F, fan)
    G.close()


def test_tree_errors_and_limits(csaw, skewed_hubs):
    import torch
    g = skewed_hubs
    G = csaw.Graph(g)
    seeds = torch.from_numpy(hub_seeds(g, 64, 3)).cuda()
    p = csaw.make_params(0, 2, 64, 1, 10, 2, [10, 4], 5, schedule=csaw.SCHED_BATCHED)
    n = G.sample(p, seeds)[0].numel()
    with pytest.raises(csaw.CsawError, match="capacity"):
        G.sample(p, seeds, capacity=n - 1)
    assert G.sample(p, seeds, capacity=n)[0].numel() == n
    bad = seeds.clone()
    bad[5] = g.n_vertices
    with pytest.raises(csaw.CsawError, match="seed vertex"):
        G.sample(p, bad)
    assert G.sample(p, seeds)[0].numel() == n   # the error left nothing behind
    # above the item bound of a chunk or of the job, and with per-sample dedup: the per-level passes
    for q in (csaw.make_params(0, 2, 1, 4097, 2, 1, [2], 5, schedule=1),
              csaw.make_params(0, 2, 262_145, 1, 2, 1, [2], 5, schedule=1),
              csaw.make_params(0, 2, 64, 1, 10, 2, [10, 4], 5, schedule=1, dedup=True)):
        s = torch.from_numpy(oracle.make_seeds(g.rowptr, q.n_samples * q.frontier_size, 9)).cuda()
        G.profile(True)
        G.sample(q, s)
        assert G.kernel_stats("tree")["launches"] == 0 and G.kernel_stats("expand")["launches"] > 0
        G.profile(False)
    G.close()
