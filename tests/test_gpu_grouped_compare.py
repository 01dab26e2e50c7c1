"""The symmetry check of grouped lines, whose last sorting pass compares: one arc
that lacks its reverse -- early, in the middle and late, in graphs of one tile of
arcs and of many, for numbers of vertices with one to three passes -- sends the
lines to the sorting route, and all its edges are there."""
import numpy as np
import pytest

import kc_cuda_b200 as K
from kc_cuda_b200 import gen

pytestmark = pytest.mark.gpu


def grouped_lines(n, draws, seed):
    keys = gen.Graph(gen.GraphSpec(kind=gen.KTG_ER, n=n, draws=draws, seed=seed)).edge_pairs().astype(np.int64)
    arcs = np.concatenate([keys, keys[:, ::-1]])
    return arcs[np.lexsort((arcs[:, 0], arcs[:, 1]))]  # x, y: by y, then x


def load(ctx, lines):
    g = ctx.load_tsv("".join(f"{x}\t{y}\n" for x, y in lines.tolist()).encode())
    return g, ctx.stats()["csr_grouped"]


@pytest.mark.parametrize("n,draws", [(150, 900), (3_000, 40_000), (70_000, 60_000)])
@pytest.mark.parametrize("where", [0.02, 0.5, 0.98])
def test_one_arc_without_reverse(n, draws, where):
    lines = grouped_lines(n, draws, 7)
    x, y = lines[:, 0], lines[:, 1]
    same = np.concatenate([y[1:] == y[:-1], [False]])
    room = np.flatnonzero((x + 1 < y) & (~same | (np.concatenate([x[1:], [0]]) > x + 1)))
    i = room[int(where * (len(room) - 1))]
    with K.Context(0) as ctx:
        g, grouped = load(ctx, lines)
        assert grouped == 1
        assert np.array_equal(g.edges(), np.unique((np.minimum(x, y) << 32) | np.maximum(x, y)))
        g.free()
        lines[i, 0] += 1
        g, grouped = load(ctx, lines)
        assert grouped == 0
        x, y = lines[:, 0], lines[:, 1]
        assert np.array_equal(g.edges(), np.unique((np.minimum(x, y) << 32) | np.maximum(x, y)))
        g.free()
