"""Support histograms on both sides of the bins that a block counts in shared
memory (6,144): the truss of a clique of 6,200 vertices is found from its
support bound alone, and in a batch beside smaller graphs."""
import numpy as np
import pytest

import kc_cuda_b200 as K

pytestmark = pytest.mark.gpu


def clique(n):
    i, j = np.triu_indices(n, 1)
    return np.stack([i, j], 1)


def test_bounds_beyond_the_shared_bins():
    sizes = [30, 6200, 200]
    graphs = [np.concatenate([clique(n), [[0, n], [1, n]]]) for n in sizes]  # and a vertex on two of its members
    want = [(n, n * (n - 1) // 2) for n in sizes]
    with K.Context(0) as ctx:
        for e, w in zip(graphs, want):
            d = ctx.load_edges(e)
            assert d.kmax_truss() == w
            d.free()
        b = ctx.batch()
        for e in graphs:
            b.add_edges(e)
        b.run()
        k, c = b.results()
        assert list(zip(k.tolist(), c.tolist())) == want
