"""The FP64-pipe kernels, which run where the links have no fixed-point copy
(not of unitary size, no room) and where their launch shape is pinned: solvers
and operators against the oracle.

Tolerances as in the other operator and solver tests: 1e-13 for operators; a
true residual of 1e-10 and 1e-9 to the oracle's solution."""
import numpy as np
import pytest

from oracle import rel_l2

pytestmark = pytest.mark.gpu
DIMS = (8, 6, 4, 8)


@pytest.fixture(scope="module")
def unitary(wd):
    return wd.gen_gauge(DIMS, seed=95), wd.gen_source(DIMS, seed=95)


@pytest.fixture(scope="module")
def scaled(wd, oracle, unitary):
    """Links with entries above one, and a mass that keeps M's spectrum away from zero."""
    gauge = [np.ascontiguousarray(1.2 * g) for g in unitary[0]]
    return gauge, unitary[1], 1.0, oracle.cg_eo(unitary[1], gauge, DIMS, 1.0)[0]


def test_pinned_shape_runs_the_pipe_kernel(wd, ctx, oracle, unitary):
    gauge, src = unitary
    lat = ctx.lattice(DIMS, gauge)
    a, b = lat.field(src), lat.field()
    vh = int(np.prod(DIMS)) // 2
    want = oracle.dslash_full(src, gauge, DIMS, 0.1, 1)
    lat.dslash_full(a, b, 0.1, 1)
    fixed = b.download()
    pinned = []
    try:
        for v in range(wd.tune_variants("hop_f64")):
            wd.tune_pin("hop_f64", vh, v)
            lat.dslash_full(a, b, 0.1, 1)
            pinned.append(b.download())
    finally:
        wd.tune_pin("hop_f64", vh, -1)
    lat.dslash_full(a, b, 0.1, 1)
    assert len(pinned) == 3 and np.array_equal(b.download(), fixed)
    for p in pinned:
        assert rel_l2(p, want) < 1e-13
        assert np.array_equal(p, pinned[0]) and not np.array_equal(p, fixed)
    assert rel_l2(fixed, want) < 1e-13


@pytest.fixture
def pinned(wd, request):
    """The FP64-pipe kernel of the shape in the test's parameters, for this lattice size."""
    vh = int(np.prod(DIMS)) // 2
    wd.tune_pin("hop_f64", vh, request.param)
    yield request.param
    wd.tune_pin("hop_f64", vh, -1)


@pytest.mark.parametrize("prec", ["F64", "DF64"])
def test_even_odd_cg_on_scaled_links(wd, ctx, scaled, prec):
    gauge, src, mass, want = scaled
    lat = ctx.lattice(DIMS, gauge)
    b, x = lat.field(src), lat.field()
    st = lat.solve(b, x, wd.solver_params(mass=mass, tol=1e-10, max_iter=2000, prec=getattr(wd, prec)))
    assert st.converged and st.true_residual <= 1e-10
    assert rel_l2(x.download(), want) < 1e-9


# (FP32 and FP16 links are two rows of an SU(3) matrix, so these solve on unitary links)
@pytest.mark.parametrize("pinned", [0, 1, 2], indirect=True)
@pytest.mark.parametrize("prec", ["F64", "F32", "F16"])
def test_fp64_reliable_updates_on_the_pipe(wd, ctx, oracle, unitary, pinned, prec):
    gauge, src = unitary
    lat = ctx.lattice(DIMS, gauge)
    b, x = lat.field(src), lat.field()
    params = wd.solver_params(mass=0.1, tol=1e-10, max_iter=2000, prec=getattr(wd, prec), prec_reliable=wd.F64)
    want = oracle.cg_eo(src, gauge, DIMS, 0.1)[0]
    st = lat.solve(b, x, params)
    assert st.converged and st.true_residual <= 1e-10
    assert rel_l2(x.download(), want) < 1e-9
    if prec != "F64":
        y = lat.field()
        stats = ctx.solve_batch([(lat, b, x, 0.1), (lat, b, y, 0.1)], params)
        for s, f in zip(stats, (x, y)):
            assert s.converged and s.true_residual <= 1e-10
            assert rel_l2(f.download(), want) < 1e-9


@pytest.mark.parametrize("prec", ["F64", "DF64"])
def test_reference_cg_on_scaled_links(wd, ctx, oracle, scaled, prec):
    gauge, src, mass, _ = scaled
    x0 = oracle.rand_guess(src.size, 3)
    want, its, _ = oracle.cg_ref(src, gauge, DIMS, mass, 2000, 1e-9, x0)
    x = x0.copy()
    st = ctx.host_cg(DIMS, gauge, src, x, wd.solver_params(kind=wd.CGNR_REF, mass=mass, tol=1e-9, max_iter=2000,
                                                           prec=getattr(wd, prec)))
    assert st.converged and abs(st.iterations - its) <= 1
    assert rel_l2(x, want) < 1e-9


def test_check_on_scaled_links(wd, ctx, oracle, scaled):
    gauge, src, mass, want = scaled
    lat = ctx.lattice(DIMS, gauge)
    got = lat.check(lat.field(src), lat.field(want), mass)
    ref = oracle.check(src, want, gauge, DIMS, mass)
    for i in (0, 1, 2, 4, 6, 8):
        assert abs(got[i] - ref[i]) <= 1e-12 * abs(ref[i])
