"""What the server and the propagator hold on the device once their requests
are done: the work-buffer cache keeps a bounded part of the fields' memory,
and the server's budget bounds cached blocks of earlier requests too."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
GB = 1 << 30


def used(ctx):
    import torch

    ctx.sync()
    free, total = torch.cuda.mem_get_info()
    return total - free


def field(dims):
    return int(np.prod(dims)) * 12 * 16


def drain(sv, rids):
    peak, todo = 0, list(rids)
    for _ in range(400):
        sv.step()
        peak = max(peak, used(sv.ctx))
        for r in list(todo):
            done, _, stats, _ = sv.poll(r)
            if done:
                assert all(s.converged for s in stats)
                todo.remove(r)
        if not todo:
            return peak
    raise AssertionError("requests unfinished")


def test_burst_is_not_kept(wd):
    dims = (16, 16, 16, 64)  # fields of 50 MB
    nsrc = 24                # 48 of them: 2.4 GB
    with wd.Context(0) as ctx:
        sv = wd.Server(ctx, prec=wd.F64)
        lat = sv.add_lattice(dims, wd.gen_gauge(dims, seed=91))
        drain(sv, [sv.submit(lat, 1, mass=0.2, tol=1e-6, seeds=[1])])
        before = used(ctx)  # a solve's work buffers are cached
        drain(sv, [sv.submit(lat, nsrc, mass=0.2, tol=1e-6, seeds=list(range(nsrc)))])
        assert used(ctx) - before <= GB
        sv.close()


def test_budget_bounds_cached_blocks(wd):
    small, large = (16, 16, 16, 16), (16, 16, 16, 64)  # fields of 12.6 and 50 MB: no block serves both
    with wd.Context(0) as ctx:
        start = used(ctx)
        sv = wd.Server(ctx, prec=wd.F64)
        ids = [sv.add_lattice(d, wd.gen_gauge(d, seed=92)) for d in (small, large)]
        links = sv.status()[2]
        sv.close()
        request = 6 * field(large)  # two fields and the solver's eight halves
        budget = links + 1.1 * request
        sv = wd.Server(ctx, prec=wd.F64, hbm_budget_bytes=budget)
        ids = [sv.add_lattice(d, wd.gen_gauge(d, seed=92)) for d in (small, large)]
        peak = 0
        for _ in range(2):
            n = 4
            peak = max(peak, drain(sv, [sv.submit(ids[0], n, mass=0.2, tol=1e-6, seeds=list(range(n)))]))
            peak = max(peak, drain(sv, [sv.submit(ids[1], 1, mass=0.2, tol=1e-6, seeds=[7])]))
        # beside the budget: the staging buffer of link uploads and small buffers
        assert peak - start <= budget + 9 * 16 * int(np.prod(large)) + (16 << 20)
        sv.close()


def test_plain_server_outlives_its_context(wd):
    """A server whose finished request was not collected, closed after its context."""
    dims = (4, 4, 4, 4)
    ctx = wd.Context(0)
    sv = wd.Server(ctx, prec=wd.F64)
    lat = sv.add_lattice(dims, wd.gen_gauge(dims, seed=93))
    for seed in (1, 2):
        sv.submit(lat, 1, mass=0.2, tol=1e-8, seeds=[seed])
    for _ in range(4):
        sv.step()
    ctx.close()
    sv.close()
    with wd.Context(0) as other:
        f = other.lattice(dims, wd.gen_gauge(dims, seed=93)).field(wd.gen_source(dims, seed=1))
        assert abs(f.norm2() - 1.0) < 1e-12
