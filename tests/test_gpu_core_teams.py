"""Core numbers of a union by teams of blocks: batches of uneven graphs -- one
that takes most blocks, graphs without an edge at the ends and between, more
graphs than teams -- have the answers of each graph alone."""
import numpy as np
import pytest

import kc_cuda_b200 as K
from kc_cuda_b200 import gen

pytestmark = pytest.mark.gpu


def er(n, draws, seed):
    return gen.Graph(gen.GraphSpec(kind=gen.KTG_ER, n=n, draws=draws, seed=seed)).edge_pairs()


def clique(n):
    i, j = np.triu_indices(n, 1)
    return np.stack([i, j], 1)


NONE = np.zeros((0, 2), np.int64)
BATCHES = {
    "two": [clique(900), er(30_000, 400_000, 1)],
    "ends": [NONE, clique(700), NONE, NONE, er(20_000, 500_000, 2), clique(40), NONE],
    "one-large": [clique(30)] * 5 + [gen.Graph(gen.rmat(17, 16, 3, [90])).edge_pairs()] + [clique(50)] * 5,
    "many": [er(400, 12_000 + 100 * i, i) for i in range(150)],
}


@pytest.mark.parametrize("name", sorted(BATCHES))
def test_batch_equals_graphs_alone(name):
    with K.Context(0) as ctx:
        want = []
        for e in BATCHES[name]:
            if len(e):
                d = ctx.load_edges(e)
                want.append(d.kmax_truss())
                d.free()
            else:
                want.append((0, 0))
        b = ctx.batch()
        for e in BATCHES[name]:
            b.add_edges(e)
        b.run()
        k, c = b.results()
        assert list(zip(k.tolist(), c.tolist())) == want


def dense(n, p, seed):
    rng = np.random.default_rng(seed)
    return np.stack(np.nonzero(np.triu(rng.random((n, n)) < p, 1)), 1)


@pytest.mark.parametrize("options", [{}, {"coop_occupancy_pct": 1}, {"batch_lanes": 1, "recount_gamma": 1}])
def test_truss_levels_by_teams(options):
    """Unions whose truss levels are peeled by teams: over 2^19 edges in rows of
    at most 64 words, graphs that end at once, one that dominates, more graphs than
    teams; with few blocks, and with other rounds."""
    sets = [
        [dense(500 + 37 * i, 0.25 + 0.03 * i, i) for i in range(10)] + [clique(64), NONE, dense(90, 0.9, 7)],
        [dense(1900, 0.5, 1), clique(5), dense(200, 0.3, 2), dense(150, 0.5, 3)],
        [dense(180 + i, 0.9, i) for i in range(60)],
    ]
    with K.Context(0) as ctx:
        want = []
        for graphs in sets:
            for e in graphs:
                if len(e):
                    d = ctx.load_edges(e)
                    want.append(d.kmax_truss())
                    d.free()
                else:
                    want.append((0, 0))
        for k, v in options.items():
            ctx.set_option(k, v)
        got = []
        for graphs in sets:
            b = ctx.batch()
            for e in graphs:
                b.add_edges(e)
            b.run()
            k, c = b.results()
            got += list(zip(k.tolist(), c.tolist()))
        assert got == want
