"""Field and link transfers from every kind of host memory: pinned arrays are
read and written by the layout kernels themselves, pageable ones and arrays
that are only 8-byte aligned go through the staging copies.  All give the
same bytes."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
DIMS = (6, 4, 6, 4)  # Vh = 288: a partial tile of 64 sites


def buffer(kind, n):
    """n complex doubles of the given kind of host memory, and its owner."""
    import torch

    if kind == "pageable":
        return np.zeros(n, np.complex128), None
    off = 1 if kind == "pinned8" else 0
    t = torch.zeros(2 * n + 1, dtype=torch.float64, pin_memory=True)
    return t.numpy()[off:off + 2 * n], t


@pytest.mark.parametrize("prec", ["F64", "DF64", "F32", "F16"])
@pytest.mark.parametrize("kind", ["pageable", "pinned", "pinned8"])
def test_transfers(wd, ctx, prec, kind):
    n = int(np.prod(DIMS)) * 12
    src = wd.gen_source(DIMS, seed=31)
    plain = wd.gen_gauge(DIMS, seed=31)
    bufs = []
    for g in plain:
        b, own = buffer(kind, g.size)
        b[...] = g if kind == "pageable" else g.view(np.float64)
        bufs.append((b, own))
    lat = C.c_void_p()
    ptrs = (C.c_void_p * 4)(*[b.ctypes.data for b, _ in bufs])
    assert all((b.ctypes.data % 16 == 8) == (kind == "pinned8") for b, _ in bufs)
    ctx.check(wd.lib.wd_lattice_create(ctx.handle, wd._dims(DIMS), ptrs, C.byref(lat)))
    ref = ctx.lattice(DIMS, plain)
    p = getattr(wd, prec)
    f = ref.field(prec=p)
    s, own_s = buffer(kind, n)
    d, own_d = buffer(kind, n)
    s[...] = src if kind == "pageable" else src.view(np.float64)
    ctx.check(wd.lib.wd_field_upload(ctx.handle, f.handle, C.c_void_p(s.ctypes.data)))
    want = ref.field(src, prec=p).download()  # numpy arrays are pageable
    ctx.check(wd.lib.wd_field_download(ctx.handle, f.handle, C.c_void_p(d.ctypes.data)))
    assert np.array_equal(d.view(np.complex128) if kind == "pageable" else d.view(np.float64),
                          want if kind == "pageable" else want.view(np.float64))
    # the links: one hop on each lattice
    a, b = ref.field(prec=p), ref.field(prec=p)
    ref.dslash_offd(f, a, 1, 0, p)
    ctx.check(wd.lib.wd_dslash_offd(ctx.handle, lat, f.handle, b.handle, 1, 0, p))
    assert np.array_equal(a.download(), b.download())
    wd.lib.wd_lattice_destroy(lat)


def test_host_operator_on_arrays_of_8_byte_alignment(wd, ctx, oracle):
    n = int(np.prod(DIMS)) * 12
    gauge, src = wd.gen_gauge(DIMS, seed=32), wd.gen_source(DIMS, seed=32)
    s, d = np.zeros(2 * n + 1)[1:], np.zeros(2 * n + 1)[1:]
    s[...] = src.view(np.float64)
    ctx.check(wd.lib.wd_host_dslash_full(ctx.handle, wd._dims(DIMS), wd._gauge_ptrs(gauge),
                                         C.c_void_p(s.ctypes.data), C.c_void_p(d.ctypes.data), 0.1, 0))
    want = oracle.dslash_full(src, gauge, DIMS, 0.1, 0).view(np.float64)
    assert np.linalg.norm(d - want) <= 1e-13 * np.linalg.norm(want)
