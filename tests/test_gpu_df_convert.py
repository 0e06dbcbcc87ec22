"""FP64 <-> double-float conversion of whole fields.

Tolerance: none.  h = fl32(x), l = fl32(x - h) and h + l are what the
conversions are defined as; NumPy forms the same roundings."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def values(kind, n):
    rng = np.random.default_rng(n)
    sign = rng.choice([-1.0, 1.0], n)
    if kind == "unit":
        return sign * rng.random(n)
    if kind == "wide":  # high part normal; low part normal, subnormal or zero
        return sign * np.ldexp(1 + rng.random(n), rng.integers(-126, 127, n))
    if kind == "subnormal":  # high part subnormal or zero
        return sign * np.ldexp(1 + rng.random(n), rng.integers(-160, -120, n))
    if kind == "tiny":  # zero as a float, FP64 subnormals among them
        return sign * np.ldexp(1 + rng.random(n), rng.integers(-1074, -150, n))
    if kind == "mixed":  # zeros and ordinary values in one warp
        return np.where(rng.random(n) < 0.5, 0.0 * sign, sign * np.ldexp(rng.random(n), rng.integers(-140, 100, n)))
    # "ties": at and next to the midpoints of neighbouring floats, and where h carries into the next power of two
    m = rng.integers(1 << 23, 1 << 24, n).astype(np.int64)
    m[::3] = (1 << 24) - 1
    rem = rng.choice([(1 << 28) - 1, 1 << 28, (1 << 28) + 1, (1 << 29) - 1, 1, 0], n).astype(np.int64)
    return sign * np.ldexp((m * (1 << 29) + rem).astype(np.float64), rng.integers(-120, 40, n) - 52)


@pytest.mark.parametrize("kind", ["unit", "wide", "subnormal", "tiny", "mixed", "ties"])
def test_field_round_trip(ctx, wd, kind):
    dims = (4, 4, 6, 2)
    lat = ctx.lattice(dims, wd.gen_gauge(dims, 3))
    x = values(kind, int(np.prod(dims)) * 24)
    with np.errstate(under="ignore"):
        h = x.astype(np.float32)
        want = h.astype(np.float64) + (x - h.astype(np.float64)).astype(np.float32).astype(np.float64)
    got = lat.field(x.view(np.complex128), prec=wd.DF64).download().view(np.float64)
    np.testing.assert_array_equal(got, want)
