"""The product kernel's waits run out (timeout_ms = 0): the call either says so
or has the right counts, and the context goes on.  Blocks give up between their
copies, after the last of them was issued (a tile of few columns) and with none
in flight (more blocks than tiles)."""
import numpy as np
import pytest

import kc_cuda_b200 as K

pytestmark = pytest.mark.gpu

KT_ERR_TIMEOUT = 6


@pytest.mark.parametrize("n,p", [(2049, 0.9), (2560, 0.8), (4700, 0.4)])
def test_product_gives_up_then_counts(n, p, capfd):
    rng = np.random.default_rng(n)
    a = np.triu(rng.random((n, n)) < p, 1)
    u, v = np.nonzero(a)
    b = (a | a.T).astype(np.float32)
    square = (b @ b).astype(np.uint32)  # sums below 2^24
    with K.Context(0) as ctx:
        d = ctx.load_edges(np.stack([u, v], 1))
        e = d.edges()
        want = square[e >> 32, e & 0xffffffff]
        ctx.set_option("verbose", 1)
        for timeout in (0, 20000, 0, 0, 20000):
            ctx.set_option("timeout_ms", timeout)
            try:
                got = d.tricount()
            except K.KtError as x:
                assert timeout == 0 and x.status == KT_ERR_TIMEOUT
                continue
            assert np.array_equal(got, want)
        assert "support (products)" in capfd.readouterr().err
        d.free()


def test_product_of_a_union_gives_up_then_counts():
    rng = np.random.default_rng(5)
    graphs = []
    for n, p in [(2100, 0.7), (220, 0.95), (256, 0.98), (3000, 0.5)]:
        graphs.append(np.stack(np.nonzero(np.triu(rng.random((n, n)) < p, 1)), 1))
    with K.Context(0) as ctx:
        want = []
        for g in graphs:
            d = ctx.load_edges(g)
            want.append(d.kmax_truss())
            d.free()
        for timeout in (0, 20000):
            ctx.set_option("timeout_ms", timeout)
            b = ctx.batch()
            for g in graphs:
                b.add_edges(g)
            if timeout:
                b.run()
                k, m = b.results()
                assert [(int(x), int(y)) for x, y in zip(k, m)] == want
            else:
                with pytest.raises(K.KtError) as ei:
                    b.run()
                assert ei.value.status == KT_ERR_TIMEOUT
            b.free()
