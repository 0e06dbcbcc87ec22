"""A residual of exactly zero meets every positive tolerance, also one whose
square is below the smallest double.

With zero links M is 4 + m; at m = 0 and a source of one entry every number
of the reference CG is a power of two, so its first iteration ends at zero.
Tolerance: none, the arithmetic is exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
DIMS = (4, 2, 2, 4)


@pytest.mark.parametrize("prec", ["F64", "DF64"])
@pytest.mark.parametrize("tol", [1e-100, 1e-170, 5e-324])
def test_zero_residual_converges(wd, ctx, prec, tol):
    n = int(np.prod(DIMS))
    lat = ctx.lattice(DIMS, [np.zeros(9 * n, np.complex128) for _ in range(4)])
    src = np.zeros(12 * n, np.complex128)
    src[17] = 1.0
    b, x = lat.field(src), lat.field()
    st = lat.solve(b, x, wd.solver_params(kind=wd.CGNR_REF, mass=0.0, tol=tol, max_iter=10, prec=getattr(wd, prec)))
    assert st.converged and st.iterations == 1 and st.residual == 0 and st.true_residual == 0
    assert np.array_equal(x.download(), src / 4)
    for o in (b, x, lat):
        o.close()
