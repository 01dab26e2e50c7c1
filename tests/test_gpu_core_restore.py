"""Restoring a core below compacted copies: the vertices of the k-core for
levels at, between and next to the search's probes, where the state goes back to
an earlier graph with some of its probes kept, with all of them, or with none.
Small graphs make copies in host-stepped rounds (kcore_compact 1); the search on
the device makes them only of graphs of millions of edges."""
import numpy as np
import pytest

import kt_oracle as O
import kc_cuda_b200 as K
from kc_cuda_b200 import gen

pytestmark = pytest.mark.gpu


def check(ctx, d, want, levels):
    cmax = int(want.max())
    for k in levels:
        mem, got = d.kmax_core(int(k))
        assert got == cmax
        assert np.array_equal(mem, want >= k), k


@pytest.mark.parametrize("spec", [
    gen.GraphSpec(kind=gen.KTG_CHUNGLU, n=30_000, draws=400_000, seed=5, cl_w_max=3_000.0),
    gen.rmat(13, 24, 5, [60])], ids=["chunglu", "rmat"])
def test_host_stepped_copies(spec):
    with K.Context(0) as ctx:
        ctx.set_option("persistent", 0)
        ctx.set_option("kcore_compact", 1)
        d = ctx.load_pairs(gen.Graph(spec).edges())
        want = O.core_numbers(d.edges(), d.num_vertices)
        check(ctx, d, want, range(1, int(want.max()) + 1))
        d.free()


def test_search_copies():
    """Over 2^22 edges, so the search itself goes on in copies; membership
    against the core numbers of the decomposition (which never copies)."""
    with K.Context(0) as ctx:
        ctx.set_option("kcore_compact", 1)
        d = ctx.load_pairs(gen.Graph(gen.rmat(19, 24, 3, [700])).edges())
        assert d.num_edges > 1 << 22
        want = d.core_numbers()
        cmax = int(want.max())
        near = [cmax, cmax - 1, cmax // 2, cmax // 4]
        check(ctx, d, want, sorted({max(1, k) for k in [1, 2, 3, 4, 7, 8, 9, 16, 33, 64, 65, 128, 200, *near]
                                    if k <= cmax}))
        d.free()
