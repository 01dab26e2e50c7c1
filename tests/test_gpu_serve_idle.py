"""Requests that find the server idle: whichever lane takes one, its wave runs
cooperative launches (the small lane holds them for the wave while the other
lane has none in flight), and a burst after them is answered as ever."""
import pytest

import kc_cuda_b200 as K
from kc_cuda_b200 import gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("small_coop", [0, 1])
def test_requests_one_at_a_time_then_a_burst(small_coop):
    idx = [i for i in range(400, 460) if gen.mix_graph(i).draws <= 400_000][:12]
    with K.Context(0) as ctx:
        alone = {}
        for i in idx:
            g = ctx.load_mix_graph(i)
            alone[i] = g.kmax_truss()
            g.free()
        ctx.set_option("serve_small_coop", small_coop)
        with ctx.server() as srv:
            rs = [(i, srv.wait(srv.submit_mix(i))) for i in idx]
            burst = [(i, srv.submit_mix(i)) for i in idx * 2]
            rs += [(i, srv.wait(r)) for i, r in burst]
        ctx.set_option("serve_small_coop", 0)
        assert ctx.get_option("persistent") == 1
    for i, r in rs:
        assert r["status"] == 0 and (r["kmax"], r["edges"]) == alone[i], i
