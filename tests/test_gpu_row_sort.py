"""Sorted rows of working graphs: lengths around each number of entries that a
warp's lane holds, rows beyond a warp by bitmap and, where those are many in a
wide graph, by the radix sort.  Supports and truss numbers are read off the
sorted rows, so they equal the oracle's only if every row is in order."""
import numpy as np
import pytest

import kt_oracle as O
import kc_cuda_b200 as K
from kc_cuda_b200 import gen

pytestmark = pytest.mark.gpu


def hubs(lengths, n, seed):
    """One vertex of each of these numbers of neighbours among n, and a ring."""
    rng = np.random.default_rng(seed)
    out = [np.stack([np.arange(n), (np.arange(n) + 1) % n], 1)]
    for i, l in enumerate(lengths):
        out.append(np.stack([np.full(l, n + i), rng.choice(n, l, replace=False)], 1))
    return np.concatenate(out)


GRAPHS = {
    "lengths": lambda: hubs([l + d for l in (1, 2, 32, 64, 128, 256, 512) for d in (-1, 0, 1) if l + d > 0], 40_000, 1),
    "long": lambda: hubs([513, 2000, 30_000, 70_000], 300_000, 2),
    "wide": lambda: hubs([600] * 400, 2_000_000, 3),
    "rmat": lambda: gen.Graph(gen.rmat(15, 16, 4, [40])).edge_pairs(),
    "er": lambda: gen.Graph(gen.GraphSpec(kind=gen.KTG_ER, n=20_000, draws=600_000, seed=3)).edge_pairs(),
}


@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_rows_in_order(name):
    e = GRAPHS[name]()
    with K.Context(0) as ctx:
        ctx.set_option("dense_max_n", 0)
        dg = ctx.load_edges(e)
        keys = dg.edges()
        assert np.array_equal(dg.tricount(), O.support(keys))
        if len(keys) < 1_000_000:
            assert np.array_equal(dg.trussness(), O.trussness(keys))
        dg.free()


def test_rows_of_a_union():
    graphs = [hubs([600, 1200], 30_000, 5), hubs([40, 512], 900, 6), GRAPHS["er"]()]
    with K.Context(0) as ctx:
        ctx.set_option("dense_max_n", 0)
        want = []
        for e in graphs:
            d = ctx.load_edges(e)
            want.append(d.kmax_truss())
            d.free()
        b = ctx.batch()
        for e in graphs:
            b.add_edges(e)
        b.run()
        k, c = b.results()
        assert list(zip(k.tolist(), c.tolist())) == want
