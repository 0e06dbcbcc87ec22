"""One lattice used beside several contexts, whose copy of the links in fixed
point any of them may take back when device memory runs short.

Tolerances as in the operator and solver tests: 1e-13 for an operator, 1e-9
between a solution of true residual 1e-10 and the oracle's."""
import ctypes as C
import threading

import numpy as np
import pytest

from oracle import rel_l2

pytestmark = pytest.mark.gpu
DIMS = (4, 4, 4, 8)
MASS = 0.1


@pytest.fixture(scope="module")
def problem(wd, oracle):
    gauge, src = wd.gen_gauge(DIMS, seed=61), wd.gen_source(DIMS, seed=61)
    return gauge, src


class Borrowed:
    """Fields and calls of one context on a lattice another one made."""

    def __init__(self, wd, ctx, lat, src):
        self.wd, self.ctx, self.lat = wd, ctx, lat
        self.f = []
        for host in (src, None):
            h = C.c_void_p()
            ctx.check(wd.lib.wd_field_create(ctx.handle, lat.handle, C.byref(h)))
            if host is not None:
                ctx.check(wd.lib.wd_field_upload(ctx.handle, h, wd._ptr(host)))
            self.f.append(h)

    def full(self, dag):
        self.ctx.check(self.wd.lib.wd_dslash_full(self.ctx.handle, self.lat.handle, self.f[0], self.f[1], MASS, dag, 0))
        return self.result()

    def solve(self):
        p, st = self.wd.solver_params(mass=MASS, tol=1e-10), self.wd.SolverStats()
        self.ctx.check(self.wd.lib.wd_solve(self.ctx.handle, self.lat.handle, self.f[0], self.f[1], C.byref(p),
                                            C.byref(st)))
        assert st.converged and st.true_residual <= 1e-10
        return self.result()

    def result(self):
        out = np.empty(self.lat.V * 12, np.complex128)
        self.ctx.check(self.wd.lib.wd_field_download(self.ctx.handle, self.f[1], self.wd._ptr(out)))
        return out

    def exhaust(self):
        self.ctx.exhaust_memory_after(0)
        h = C.c_void_p()
        st = self.wd.lib.wd_field_create(self.ctx.handle, self.lat.handle, C.byref(h))
        self.ctx.exhaust_memory_after(-1)
        self.wd.lib.wd_field_destroy(h)
        return st

    def close(self):
        for h in self.f:
            self.wd.lib.wd_field_destroy(h)


@pytest.mark.parametrize("owner_first", [True, False])
def test_update_through_another_context(wd, oracle, problem, owner_first):
    gauge, src = problem
    a, b = wd.Context(0), wd.Context(0)
    lat = a.lattice(DIMS, [np.ascontiguousarray(3.0 * g) for g in gauge])  # links that the copy cannot hold
    u = Borrowed(wd, b, lat, src)
    b.check(wd.lib.wd_lattice_update(b.handle, lat.handle, wd._gauge_ptrs(gauge)))
    want = oracle.dslash_full(src, gauge, DIMS, MASS, 1)
    assert rel_l2(u.full(1), want) < 1e-13
    assert u.exhaust() == wd.OK  # the copy is given back, whichever context built it
    assert u.exhaust() == wd.OOM
    assert rel_l2(u.full(1), want) < 1e-13
    if owner_first:
        a.close()
        b.check(wd.lib.wd_lattice_update(b.handle, lat.handle, wd._gauge_ptrs(gauge)))
        assert rel_l2(u.full(1), want) < 1e-13
        u.close()
        lat.close()
        b.close()
    else:
        u.close()
        b.close()
        lat.close()
        a.close()


def test_another_context_takes_the_links_back(wd, oracle, problem):
    gauge, src = problem
    with wd.Context(0) as a, wd.Context(0) as b:
        lat = a.lattice(DIMS, gauge)
        u, v = Borrowed(wd, a, lat, src), Borrowed(wd, b, lat, src)
        want = oracle.dslash_full(src, gauge, DIMS, MASS, 0)
        assert rel_l2(u.full(0), want) < 1e-13
        assert v.exhaust() == wd.OK
        assert rel_l2(u.full(0), want) < 1e-13
        for w in (u, v, lat):
            w.close()


def test_taken_back_while_another_thread_solves(wd, oracle, problem):
    gauge, src = problem
    want = oracle.cg_eo(src, gauge, DIMS, MASS)[0]
    stop, seen, errors = threading.Event(), [], []
    with wd.Context(0) as a, wd.Context(0) as b:
        lat = a.lattice(DIMS, gauge)
        other = a.lattice(DIMS, gauge)
        u, v = Borrowed(wd, a, other, src), Borrowed(wd, b, lat, src)

        def work():
            try:
                while not stop.is_set():
                    seen.append(rel_l2(v.solve(), want))
            except Exception as e:  # noqa: BLE001
                errors.append(e)

        t = threading.Thread(target=work)
        t.start()
        for _ in range(40):
            u.exhaust()  # OK or, with every copy already gone, OOM
            other.update(gauge)
            u.full(0)
        stop.set()
        t.join()
        assert not errors and seen and max(seen) < 1e-9
        for w in (u, v, lat, other):
            w.close()
