"""Device memory that runs short inside a call: the library gives back what it
holds for speed only (cached work buffers, fixed-point links) and the call
goes on without it.

Tolerances: a solve's FP64 true residual meets its 1e-10 and its solution lies
within 1e-9 of the oracle's, as in the other solver tests; operators 1e-13."""
import numpy as np
import pytest

from oracle import rel_l2

pytestmark = pytest.mark.gpu
DIMS = (4, 4, 4, 8)
MASS = 0.1


@pytest.fixture(scope="module")
def problem(wd, oracle):
    gauge, src = wd.gen_gauge(DIMS, seed=51), wd.gen_source(DIMS, seed=51)
    return gauge, src, oracle.cg_eo(src, gauge, DIMS, MASS)[0]


def plans(wd):
    return {"eo_f64": (wd.CG_EO, wd.F64, wd.F64), "ref_f64": (wd.CGNR_REF, wd.F64, wd.F64),
            "eo_df64": (wd.CG_EO, wd.DF64, wd.F64), "f32_f64": (wd.CG_EO, wd.F32, wd.F64),
            "f16_df64": (wd.CG_EO, wd.F16, wd.DF64)}


@pytest.mark.parametrize("plan", ["eo_f64", "ref_f64", "eo_df64", "f32_f64", "f16_df64"])
def test_memory_runs_short_at_every_request_of_a_solve(wd, problem, plan):
    gauge, src, want = problem
    kind, prec, rel = plans(wd)[plan]
    params = wd.solver_params(kind=kind, mass=MASS, tol=1e-12 if kind == wd.CGNR_REF else 1e-10, max_iter=2000,
                              prec=prec, prec_reliable=rel)
    hit = 0
    for n in range(60):
        with wd.Context(0) as ctx:
            lat = ctx.lattice(DIMS, gauge)
            b, x, t = lat.field(src), lat.field(), lat.field()
            lat.dslash_full(b, t, MASS, 0)
            x.zero()
            ctx.exhaust_memory_after(n)
            st = lat.solve(b, x, params)
            left = ctx.exhaust_memory_after(-1)
            assert st.converged and st.true_residual <= 1e-10, n
            assert rel_l2(x.download(), want) < 1e-9, n
            for o in (b, x, t, lat):
                o.close()
        if left >= 0:  # the solve asks for memory fewer than n times
            break
        hit += 1
    assert hit >= 1 and left >= 0


def test_operators_after_the_links_are_given_back(wd, problem, oracle):
    gauge, src, _ = problem
    with wd.Context(0) as ctx:
        lat = ctx.lattice(DIMS, gauge)
        b, x = lat.field(src), lat.field()
        want = oracle.dslash_full(src, gauge, DIMS, MASS, 1)
        for _ in range(2):
            lat.dslash_full(b, x, MASS, 1)
            assert rel_l2(x.download(), want) < 1e-13
            ctx.exhaust_memory_after(0)
            extra = lat.field()  # finds memory exhausted
            assert ctx.exhaust_memory_after(-1) == -1
            lat.dslash_offd(b, x, 0, 1)
            assert rel_l2(x.download(), oracle.dslash_offd(src, gauge, DIMS, 0, 1)) < 1e-13
            extra.close()
            lat.update(gauge)
        for o in (b, x, lat):
            o.close()


def test_exhausted_with_nothing_to_give_back_is_oom(wd, problem):
    gauge, _, _ = problem
    with wd.Context(0) as ctx:
        lat = ctx.lattice(DIMS, [np.ascontiguousarray(3.0 * g) for g in gauge])  # links without a second copy
        ctx.exhaust_memory_after(0)
        with pytest.raises(wd.WilsonError) as e:
            lat.field()
        assert e.value.status == wd.OOM
        lat.field().close()
        lat.close()
