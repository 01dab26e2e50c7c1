"""List-mode support counting at the sizes where its kernels meet.

Edges whose larger end has at most 256 neighbours are counted by one warp per
vertex with a hashed filter, the others by the block kernel (a bitmap of the
graph's vertices) or, above support_bitmap_max_n vertices, by binary search.
Every count must equal the oracle's on both sides of that line, for rows of
fewer and more than the 8, 32 and 64 entries a warp step takes, and in unions."""
import numpy as np
import pytest

import kt_oracle as O
import kc_cuda_b200 as K
from kc_cuda_b200 import gen

pytestmark = pytest.mark.gpu


def clique(n, base):
    i, j = np.triu_indices(n, 1)
    return np.stack([i + base, j + base], axis=1)


def wheel(leaves, base):
    """A hub of `leaves` neighbours that form a cycle."""
    r = np.arange(leaves)
    return np.concatenate([np.stack([np.full(leaves, base), base + 1 + r], axis=1),
                           np.stack([base + 1 + r, base + 1 + (r + 1) % leaves], axis=1)])


def pieces(make, sizes):
    out, base = [], 0
    for s in sizes:
        out.append(make(s, base))
        base += s + 1
    return np.concatenate(out)


GRAPHS = {
    "cliques": lambda: pieces(clique, [2, 3, 8, 9, 10, 33, 34, 65, 66, 129, 256, 257, 258, 259]),
    "wheels": lambda: pieces(wheel, [3, 4, 31, 32, 63, 64, 65, 255, 256, 257, 258, 700]),
    "er": lambda: gen.Graph(gen.GraphSpec(kind=gen.KTG_ER, n=3001, draws=190_000, seed=5)).edge_pairs(),
    "rmat": lambda: gen.Graph(gen.rmat(12, 16, 9, [40])).edge_pairs(),
}


@pytest.mark.parametrize("bitmap_max", [1 << 20, 0])
@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_list_support_equals_oracle(name, bitmap_max):
    with K.Context(0) as ctx:
        ctx.set_option("dense_max_n", 0)
        ctx.set_option("support_bitmap_max_n", bitmap_max)
        dg = ctx.load_edges(GRAPHS[name]())
        edges = dg.edges()
        for _ in range(2):
            assert np.array_equal(dg.tricount(), O.support(edges))
        dg.free()


def test_union_without_bitsets_equals_alone():
    graphs = [g() for g in GRAPHS.values()]
    with K.Context(0) as ctx:
        want = []
        for p in graphs:
            dg = ctx.load_edges(p)
            want.append(dg.kmax_truss())
            dg.free()
        ctx.set_option("dense_max_n", 0)
        b = ctx.batch()
        for p in graphs:
            b.add_edges(p)
        b.run()
        k, e = b.results()
        assert [(int(x), int(y)) for x, y in zip(k, e)] == want
        b.free()
