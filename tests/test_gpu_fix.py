"""The FP64 hopping term in fixed point: where its block scale, its ranges and
its routing can go wrong.

Tolerances.  Oracle and kernel each round a sum of 8 x 12 products; both stay
within a few dozen units of 2^-53 of the largest neighbour value of a site,
so site by site |difference| <= 128 x 2^-53 x (largest |component| among the
site's eight neighbours) -- also when the neighbours' sizes differ by more
than a block scale holds, where the small ones are rounded off.  Over a whole
field the relative L2 bar of the FP64 operators applies."""
import numpy as np
import pytest

from oracle import rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-13
EPS = 2.0 ** -53


def neighbour_max(oracle, src, dims, cb):
    """Largest |re|, |im| among the neighbours of every output site (the hop of
    |src| with unit links and all components equal cannot be below it / 8)."""
    V = int(np.prod(dims))
    a = np.maximum(np.abs(src.real), np.abs(src.imag)).reshape(V, 12).max(1)
    lx, ly, lz, lt = dims
    i = np.arange(V)
    odd = (i % lx + i // lx % ly + i // (lx * ly) % lz + i // (lx * ly * lz)) % 2
    order = np.argsort(odd * V + i, kind="stable")
    lex = np.empty(V)
    lex[order] = a
    g = lex.reshape(lt, lz, ly, lx)
    m = np.max([np.roll(g, s, ax) for ax in range(4) for s in (1, -1)], axis=0).reshape(-1)[order]
    return m.reshape(2, V // 2)[cb]


def check_sites(got, want, nbmax, cb):
    V = nbmax.size * 2
    g, w = got.reshape(V, 12), want.reshape(V, 12)
    sl = slice(cb * V // 2, (cb + 1) * V // 2)
    err = np.maximum(np.abs((g - w)[sl].real), np.abs((g - w)[sl].imag)).max(1)
    # FP64 below its normal range loses digits in both
    assert np.all(err <= 128 * EPS * nbmax + 1e-306)


@pytest.mark.parametrize("scale", [0, 40, 700, -600, -880, -960, -1030])
def test_uniform_scales(wd, ctx, oracle, scale):
    """Values far above and below one, through the block exponents' limits."""
    dims = (6, 4, 6, 4)
    gauge = wd.gen_gauge(dims, seed=21)
    src = np.ldexp(wd.gen_source(dims, seed=21).view(np.float64), scale).view(np.complex128)
    lat = ctx.lattice(dims, gauge)
    fi, fo = lat.field(src), lat.field()
    for dag in (0, 1):
        for cb in (0, 1):
            lat.dslash_offd(fi, fo, dag, cb)
            want = oracle.dslash_offd(src, gauge, dims, dag, cb)
            check_sites(fo.download(), want, neighbour_max(oracle, src, dims, cb), cb)
    host = ctx.host_dslash_full(dims, gauge, src, 0.1, 1)
    full = oracle.dslash_full(src, gauge, dims, 0.1, 1)
    for cb in (0, 1):
        check_sites(host, full, np.maximum(neighbour_max(oracle, src, dims, cb),
                                           np.abs(src).reshape(2, -1, 12)[cb].max(1)) * 5, cb)


@pytest.mark.parametrize("spread", [5, 40, 300])
def test_neighbours_of_different_sizes(wd, ctx, oracle, spread):
    dims = (8, 4, 4, 6)
    rng = np.random.default_rng(spread)
    gauge = wd.gen_gauge(dims, seed=22)
    src = wd.gen_source(dims, seed=22).reshape(-1, 12)
    src = np.ascontiguousarray((src * 10.0 ** rng.uniform(-spread, spread, src.shape[0])[:, None]).reshape(-1))
    lat = ctx.lattice(dims, gauge)
    fi, fo = lat.field(src), lat.field()
    for cb in (0, 1):
        lat.dslash_offd(fi, fo, 1, cb)
        check_sites(fo.download(), oracle.dslash_offd(src, gauge, dims, 1, cb), neighbour_max(oracle, src, dims, cb), cb)


def test_zeros_stay_zero(wd, ctx, oracle):
    dims = (4, 4, 2, 6)
    gauge = wd.gen_gauge(dims, seed=23)
    src = np.zeros(int(np.prod(dims)) * 12, np.complex128)
    src[5] = 1.0 - 2.0j
    lat = ctx.lattice(dims, gauge)
    fo = lat.field()
    for cb in (0, 1):
        lat.dslash_offd(lat.field(src), fo, 0, cb)
        got, want = fo.download(), oracle.dslash_offd(src, gauge, dims, 0, cb)
        assert np.array_equal(got == 0, want == 0)
        assert rel_l2(got, want) < TOL if want.any() else not got.any()


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf, 1.5e308])
def test_non_finite_and_overflowing_values(wd, ctx, oracle, bad):
    """One bad value: the sites it reaches come out as FP64 arithmetic gives
    them, every other site is untouched."""
    dims = (6, 4, 4, 4)
    gauge = wd.gen_gauge(dims, seed=24)
    src = wd.gen_source(dims, seed=24)
    clean = src.copy()
    V = int(np.prod(dims))
    src[(V // 2 + 17) * 12 + 4] = complex(bad, 0.25)
    lat = ctx.lattice(dims, gauge)
    fo = lat.field()
    lat.dslash_offd(lat.field(src), fo, 0, 0)
    got = fo.download().reshape(V, 12)
    lat.dslash_offd(lat.field(clean), fo, 0, 0)
    ref = fo.download().reshape(V, 12)
    want = oracle.dslash_offd(src, gauge, dims, 0, 0).reshape(V, 12)
    wclean = oracle.dslash_offd(clean, gauge, dims, 0, 0).reshape(V, 12)
    with np.errstate(all="ignore"):
        hit = ~(np.abs(want - wclean).max(1) < 1e-10)
    assert hit.sum() == 8
    assert np.array_equal(got[~hit], ref[~hit])
    assert np.array_equal(np.isfinite(got[hit]).all(1), np.isfinite(want[hit]).all(1))


@pytest.mark.parametrize("scale,shift", [(3.0, 0.0), (1.0, 1e-3), (1e-8, 0.0)])
def test_links_outside_the_fixed_point_range(wd, ctx, oracle, scale, shift):
    """Links that are not unitary take the FP64-pipe kernels, or the fixed-point
    ones where their entries still fit; an update with other links reroutes."""
    dims = (10, 6, 6, 6)
    gauge = wd.gen_gauge(dims, seed=25)
    other = [np.ascontiguousarray(g * scale + shift) for g in gauge]
    src = wd.gen_source(dims, seed=25)
    lat = ctx.lattice(dims, gauge)
    fi, fo = lat.field(src), lat.field()
    lat.dslash_full(fi, fo, 0.1, 0)
    assert rel_l2(fo.download(), oracle.dslash_full(src, gauge, dims, 0.1, 0)) < TOL
    lat.update(other)
    for dag in (0, 1):
        lat.dslash_offd(fi, fo, dag, 1)
        # entries of size 1e-8 keep 60 - 27 bits of a fixed-point link: such
        # lattices must not lose precision either
        assert rel_l2(fo.download(), oracle.dslash_offd(src, other, dims, dag, 1)) < TOL
    lat.update(gauge)
    lat.dslash_full(fi, fo, 0.1, 1)
    assert rel_l2(fo.download(), oracle.dslash_full(src, gauge, dims, 0.1, 1)) < TOL


def test_more_accurate_than_fp64_rounding(wd, ctx, oracle):
    """Error against extended precision no larger than the FP64 oracle's own."""
    if np.finfo(np.longdouble).eps > 1e-18:
        pytest.skip("no extended precision on this machine")
    dims = (4, 4, 4, 4)
    gauge, src = wd.gen_gauge(dims, seed=26), wd.gen_source(dims, seed=26)
    lat = ctx.lattice(dims, gauge)
    fo = lat.field()
    lat.dslash_offd(lat.field(src), fo, 0, 0)
    exact = longdouble_offd(src, gauge, dims)
    n = np.linalg.norm(src)
    mine = np.linalg.norm((fo.download() - exact).astype(np.complex128)) / n
    fp64 = np.linalg.norm((oracle.dslash_offd(src, gauge, dims, 0, 0) - exact).astype(np.complex128)) / n
    assert mine <= fp64


def longdouble_offd(src, gauge, dims):
    """out[even] = -1/2 D src[odd] in extended precision (no dagger)."""
    lx, ly, lz, lt = dims
    V = lx * ly * lz * lt
    i = np.arange(V)
    odd = (i % lx + i // lx % ly + i // (lx * ly) % lz + i // (lx * ly * lz)) % 2
    order = np.argsort(odd * V + i, kind="stable")

    def grid(a, k):
        lex = np.empty((V, k), np.clongdouble)
        lex[order] = a.reshape(V, k)
        return lex.reshape(lt, lz, ly, lx, k)

    psi = grid(src, 12).reshape(lt, lz, ly, lx, 4, 3)
    U = [grid(g, 9).reshape(lt, lz, ly, lx, 3, 3) for g in gauge]
    out = np.zeros_like(psi)
    I = np.clongdouble(1j)
    for mu in range(4):
        ax = 3 - mu
        for fwd in (True, False):
            sg = -1 if fwd else 1
            nb = np.roll(psi, -1 if fwd else 1, ax)
            s = [nb[..., k, :] for k in range(4)]
            h = {0: (s[0] + sg * I * s[3], s[1] + sg * I * s[2]), 1: (s[0] - sg * s[3], s[1] + sg * s[2]),
                 2: (s[0] + sg * I * s[2], s[1] - sg * I * s[3]), 3: (s[0] + sg * s[2], s[1] + sg * s[3])}[mu]
            W = U[mu] if fwd else np.conj(np.roll(U[mu], 1, ax).swapaxes(-1, -2))
            t = [sum(W[..., :, b] * v[..., b:b + 1] for b in range(3)) for v in h]
            out[..., 0, :] += t[0]
            out[..., 1, :] += t[1]
            lo = {0: (-sg * I * t[1], -sg * I * t[0]), 1: (sg * t[1], -sg * t[0]),
                  2: (-sg * I * t[0], sg * I * t[1]), 3: (sg * t[0], sg * t[1])}[mu]
            out[..., 2, :] += lo[0]
            out[..., 3, :] += lo[1]
    out = (out.reshape(V, 12)[order] * np.longdouble(-0.5)).reshape(2, -1)
    out[1] = 0
    return out.reshape(-1)
