"""The FP64 hopping term component by component: a component that is small
because its own terms are small (one colour or spin beside another, a small
link entry, a real part beside an imaginary one) is as accurate as the large
ones, and one without terms is exactly zero.

Tolerance.  S = sum |U| |h| over the products behind one real of the result (h:
the projected half-spinor).  FP64 arithmetic (the oracle) is within 20 x 2^-53
S: 6 products and sums per direction, 8 directions, a factor.  Fixed point
is within 90 units of 2^-58 of the block scale (8 directions x 10: cut
operands 2.5, rounded links 0.75, dropped low products 6, a shift 1; and
rescaling), and the kernel uses it only where S is at least 2^-7 of that scale:
360 x 2^-53 S.  Together below 384 x 2^-53 S.  The same holds for M with the
mass term's size added."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
BAR = 384 * 2.0 ** -53
SMALL, LARGE = (8, 4, 4, 6), (16, 16, 16, 10)  # a direction pair per warp; two threads a site


def order(dims):
    lx, ly, lz, lt = dims
    i = np.arange(lx * ly * lz * lt)
    odd = (i % lx + i // lx % ly + i // (lx * ly) % lz + i // (lx * ly * lz)) % 2
    return np.argsort(odd * i.size + i, kind="stable")


def sums(src, gauge, dims, dag):
    """S of both reals of every component of D src / 2 (both parities)."""
    lx, ly, lz, lt = dims
    o = order(dims)

    def grid(a, *k):
        lex = np.empty((o.size,) + k, np.complex128)
        lex[o] = a.reshape((o.size,) + k)
        return lex.reshape((lt, lz, ly, lx) + k)

    psi, out = grid(src, 4, 3), np.zeros((lt, lz, ly, lx, 4, 3, 2))
    for mu in range(4):
        ax, U = 3 - mu, grid(gauge[mu], 3, 3)
        for fwd in (True, False):
            sg = (-1 if fwd else 1) * (-1 if dag else 1)
            s = np.moveaxis(np.roll(psi, -1 if fwd else 1, ax), -2, 0)
            h = {0: (s[0] + sg * 1j * s[3], s[1] + sg * 1j * s[2]), 1: (s[0] - sg * s[3], s[1] + sg * s[2]),
                 2: (s[0] + sg * 1j * s[2], s[1] - sg * 1j * s[3]), 3: (s[0] + sg * s[2], s[1] + sg * s[3])}[mu]
            W = U if fwd else np.roll(U, 1, ax).swapaxes(-1, -2)
            wr, wi = np.abs(W.real), np.abs(W.imag)
            for k, v in enumerate(h):
                hr, hi = np.abs(v.real)[..., None], np.abs(v.imag)[..., None]
                t = np.stack([wr @ hr + wi @ hi, wr @ hi + wi @ hr], -1)[..., 0, :]
                out[..., k, :, :] += t
                low = (3 - k) if mu < 2 else 2 + k
                out[..., low, :, :] += t[..., ::-1] if mu in (0, 2) else t
    return 0.5 * out.reshape(o.size, 12, 2)[o]


def reals(v):
    return v.view(np.float64).reshape(-1, 12, 2)


def check(got, want, S, what):
    g, w = reals(got), reals(want)
    assert np.all(g[S == 0] == 0), what
    err = np.abs(g - w) / np.where(S > 0, S, 1.0)
    assert err.max() <= BAR, (what, err.max() / 2.0 ** -53)


def links(wd, dims, kind):
    V = int(np.prod(dims))
    rng = np.random.default_rng(5)
    if kind == "su3":
        return wd.gen_gauge(dims, seed=31)
    if kind == "near_unit":
        return wd.gen_gauge(dims, seed=31, eps=1e-9)
    out = []
    for _ in range(4):
        d = np.ones((V, 3)) if kind == "unit" else np.exp(2j * np.pi * rng.random((V, 3)))
        out.append(np.ascontiguousarray((d[:, :, None] * np.eye(3)).astype(np.complex128).reshape(-1)))
    return out


def source(wd, dims, kind):
    V = int(np.prod(dims))
    rng = np.random.default_rng(6)
    src = wd.gen_source(dims, seed=32).reshape(V, 4, 3)
    r = src.view(np.float64).reshape(V, 4, 3, 2)
    if kind == "colours":
        r *= np.array([1.0, 1e-10, 1e-20])[:, None]
    elif kind == "spins":
        r *= np.array([1.0, 1e-18, 1e-18, 1e-7])[:, None, None]
    elif kind == "imaginary":
        r[..., 1] *= 1e-12
    elif kind == "spread":
        r *= 10.0 ** rng.uniform(-15, 15, (1, 4, 3, 2))
    elif kind == "spread_everywhere":
        r *= 10.0 ** rng.uniform(-12, 0, r.shape)
    elif kind == "zeros":
        r[:, :, 1:] = 0.0
        r[:, 1:] *= -0.0
    elif kind == "point":
        r[:] = -0.0
        for site in (0, V // 2 + 3, V // 3):
            r[site, site % 4, site % 3, 0] = 1.0
    elif kind == "negative_zero":
        r[:] = -0.0
    return np.ascontiguousarray(src.reshape(-1))


CASES = [("unit", "colours"), ("unit", "spins"), ("unit", "imaginary"), ("unit", "spread"), ("unit", "zeros"),
         ("unit", "point"), ("unit", "negative_zero"), ("diagonal", "colours"), ("diagonal", "zeros"),
         ("near_unit", "colours"), ("su3", "spread"), ("su3", "spread_everywhere"), ("su3", "point"), ("su3", "spins"),
         ("su3", "dense")]


@pytest.mark.parametrize("dims", [SMALL, LARGE], ids=["small", "large"])
@pytest.mark.parametrize("link,kind", CASES)
def test_components(wd, ctx, oracle, dims, link, kind):
    gauge, src = links(wd, dims, link), source(wd, dims, kind)
    V = int(np.prod(dims))
    lat = ctx.lattice(dims, gauge)
    fi, fo = lat.field(src), lat.field()
    for dag in (0, 1):
        S = sums(src, gauge, dims, dag)
        for cb in (0, 1):
            part = S.copy()
            part[(1 - cb) * V // 2:(2 - cb) * V // 2] = 0
            lat.dslash_offd(fi, fo, dag, cb)
            want = oracle.dslash_offd(src, gauge, dims, dag, cb)
            check(fo.download(), want, part, ("offd", dag, cb))
            check(ctx.host_dslash_offd(dims, gauge, src, dag, cb), want, part, ("host", dag, cb))
        lat.dslash_full(fi, fo, 0.1, dag)
        check(fo.download(), oracle.dslash_full(src, gauge, dims, 0.1, dag), S + 4.1 * np.abs(reals(src)), ("full", dag))
