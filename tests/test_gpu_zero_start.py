"""A solve from zero takes its first residual from the source alone, one from
an initial guess from the operator.

Tolerance: none.  With a guess of zeros both form the same residual, entry by
entry, and only the sum |s|^2 (which sets the stopping target, not the
iterates) is added in another order, so two iterations from either start give
the same numbers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# sites of a parity: 8 (less than a warp), 108 (no multiple of 32), 256 (one
# block), 1080 (a ragged last block)
@pytest.mark.parametrize("dims", [(2, 2, 2, 2), (6, 6, 6, 2), (8, 4, 4, 4), (6, 6, 10, 6)])
@pytest.mark.parametrize("prec, reliable", [("F64", "F64"), ("DF64", "DF64"), ("F32", "F64"), ("F32", "DF64"),
                                            ("F16", "F64"), ("F16", "DF64")])
def test_zero_start_is_a_guess_of_zeros(ctx, wd, dims, prec, reliable):
    lat = ctx.lattice(dims, wd.gen_gauge(dims, 5))
    src = lat.field(wd.gen_source(dims, 6))
    sols = []
    for guess in (0, 1):
        x = lat.field()
        x.zero()
        p = wd.solver_params(kind=wd.CG_EO, mass=0.1, tol=1e-12, max_iter=2, prec=getattr(wd, prec),
                             prec_reliable=getattr(wd, reliable))
        p.use_initial_guess = guess
        lat.solve(src, x, p, allow_unconverged=True)
        sols.append(x.download())
    assert np.abs(sols[0]).max() > 0
    np.testing.assert_array_equal(sols[0], sols[1])
