"""A server whose budget holds little more than one request takes a request's
memory from what an equal one before it left, without asking CUDA for any."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
DIMS = (8, 8, 8, 16)


@pytest.mark.parametrize("prec", ["F64", "F16"])
def test_second_request_asks_for_no_memory(wd, prec):
    with wd.Context(0) as ctx:
        gauge = wd.gen_gauge(DIMS, seed=94)

        def server(**kw):
            sv = wd.Server(ctx, prec=getattr(wd, prec), **kw)
            return sv, sv.add_lattice(DIMS, gauge)

        def serve(sv, lat):
            rid = sv.submit(lat, 2, mass=0.2, tol=1e-6, seeds=[1, 2])
            for _ in range(400):
                sv.step()
                if sv.poll(rid)[0]:
                    return
            raise AssertionError("request unfinished")

        sv, lat = server()
        links = sv.status()[2]
        rid = sv.submit(lat, 2, mass=0.2, tol=1e-6, seeds=[1, 2])
        sv.step()
        request = sv.status()[2] - links
        while not sv.poll(rid)[0]:
            sv.step()
        sv.close()

        sv, lat = server(hbm_budget_bytes=links + 1.1 * request)
        serve(sv, lat)
        serve(sv, lat)
        ctx.exhaust_memory_after(1000)
        serve(sv, lat)
        assert ctx.exhaust_memory_after(-1) == 1000
        sv.close()
