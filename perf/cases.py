"""What the speed of this framework is measured on.

Every case is a call, or a short chain of calls, that a program using the
library makes through its public entry points (the C ABI as bound by
`wilson_gb300`), with inputs of the kind it meets in earnest: smooth SU(3)
links (Gram-Schmidt of 1 + i eps H, eps = 0.5) and unit-norm Gaussian or
point sources.

Results are fetched into page-locked arrays that the program keeps, as a
program that fetches results again and again does; the fetch is part of the
call.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "ipcc2021-final_gb300"))
import wilson_gb300 as wd  # noqa: E402

PREC = {"f64": wd.F64, "df64": wd.DF64, "f32": wd.F32, "f16": wd.F16}
# bytes per site of links (4 directions) and of a spinor in each storage
LINK_BYTES = {"f64": 4 * 144, "df64": 4 * 144, "f32": 4 * 48, "f16": 4 * 24}
SPINOR_BYTES = {"f64": 192, "df64": 192, "f32": 96, "f16": 52}
HOP_FLOPS = 1320  # of one site's hopping term
EPS = 0.5

_CTX = []


def _ctx():
    # one context per process and device, as a program keeps it
    if not _CTX:
        _CTX.append(wd.Context(0))
    return _CTX[0]


# ------------------------------------------------------------------- cases
def listed():
    return [
        # one hopping term on the reference's own small lattice: latency and launches
        {"name": "offd_f64_8c16", "kind": "op", "op": "offd", "prec": "f64", "dims": "8x8x8x16", "reps": 1,
         "mass": 0.1},
        # the full operator (DslashNew and its adjoint) applied in turn on the resident benchmark
        # lattice, as a Krylov or polynomial method of the user's own does
        {"name": "full_f64_32c64", "kind": "op", "op": "full", "prec": "f64", "dims": "32x32x32x64", "reps": 8,
         "mass": 0.05},
        # the same in double-float arithmetic on an odd-shaped lattice
        {"name": "full_df64_ragged", "kind": "op", "op": "full", "prec": "df64", "dims": "20x18x26x30", "reps": 8,
         "mass": 0.05},
        # even-odd hopping terms in FP32 storage, mid-size lattice
        {"name": "eo_f32_24c48", "kind": "op", "op": "eo", "prec": "f32", "dims": "24x24x24x48", "reps": 16,
         "mass": 0.05},
        # the drop-in DslashoffdNew on host arrays (page-locked), benchmark lattice
        {"name": "host_offd_32c64", "kind": "host", "op": "offd", "dims": "32x32x32x64", "pinned": True,
         "mass": 0.05},
        # the drop-in DslashNew on malloc'ed host arrays, as the reference allocates them
        {"name": "host_full_24c48", "kind": "host", "op": "full", "dims": "24x24x24x48", "pinned": False,
         "mass": 0.05},
        # the reference's own job: CGinvert on host arrays at 8^3x16, mass 0.1
        {"name": "host_cg_ref_8c16", "kind": "hostcg", "dims": "8x8x8x16", "mass": 0.1, "tol": 1e-11},
        # even-odd CG in plain FP64 on resident fields, ordinary size
        {"name": "cg_f64_16c32", "kind": "cg", "prec": "f64", "reliable": "f64", "dims": "16x16x16x32",
         "mass": 0.05, "tol": 1e-10},
        # the fastest plan on the largest benchmark lattice: FP16 inner, double-float reliable updates
        {"name": "cg_f16_df64_48c96", "kind": "cg", "prec": "f16", "reliable": "df64", "dims": "48x48x48x96",
         "mass": 0.01, "tol": 1e-10},
        # a propagator: 12 point sources batched on one lattice (FP32 inner, FP64 reliable updates)
        {"name": "propagator_16c32", "kind": "prop", "prec": "f32", "reliable": "f64", "dims": "16x16x16x32",
         "mass": 0.05, "tol": 1e-10},
        # lattices of uneven volume solved together, L = 8, 12, 16, 24
        {"name": "batch_uneven", "kind": "batch", "prec": "f16", "reliable": "df64", "sizes": "8,12,16,24",
         "each": 2, "tol": 1e-10},
        # the solve server taking a burst of requests on two resident lattices
        {"name": "server_burst", "kind": "server", "prec": "f16", "reliable": "df64", "sizes": "8,16",
         "requests": 6, "nsrc": 3, "tol": 1e-10},
    ]


def _draw_dims(rng, lo, hi):
    """Even extents, volume between lo and hi sites (spread over its logarithm)."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    while True:
        side = (v / 2) ** 0.25
        d = [max(2, 2 * round(side * math.exp(rng.uniform(-0.35, 0.35)) / 2)) for _ in range(3)]
        t = 2 * round(v / (d[0] * d[1] * d[2]) / 2)
        if 2 <= t <= 6 * side and d[0] >= 4 and lo <= d[0] * d[1] * d[2] * t <= hi:
            return "x".join(str(k) for k in d + [t])


def draw(rng):
    mass = round(rng.uniform(0.02, 0.2), 4)
    kind = rng.choice(["op", "op", "host", "hostcg", "cg", "cg", "prop", "batch", "server"])
    if kind == "op":
        return {"kind": "op", "op": rng.choice(["offd", "eo", "full"]), "prec": rng.choice(["f64", "f64", "df64", "f32"]),
                "dims": _draw_dims(rng, 256, 2097152), "reps": rng.choice([1, 2, 4, 8]), "mass": mass}
    if kind == "host":
        return {"kind": "host", "op": rng.choice(["offd", "full"]), "dims": _draw_dims(rng, 256, 2097152),
                "pinned": rng.choice([True, False]), "mass": mass}
    if kind == "hostcg":
        return {"kind": "hostcg", "dims": _draw_dims(rng, 256, 131072), "mass": mass, "tol": 1e-11}
    if kind == "cg":
        prec, rel = rng.choice([("f64", "f64"), ("df64", "df64"), ("f32", "f64"), ("f32", "df64"), ("f16", "f64"),
                                ("f16", "df64")])
        return {"kind": "cg", "prec": prec, "reliable": rel, "dims": _draw_dims(rng, 1024, 1048576), "mass": mass,
                "tol": 1e-10}
    prec, rel = rng.choice([("f32", "f64"), ("f32", "df64"), ("f16", "df64")])
    if kind == "prop":
        return {"kind": "prop", "prec": prec, "reliable": rel, "dims": _draw_dims(rng, 2048, 262144), "mass": mass,
                "tol": 1e-10}
    if kind == "batch":
        sizes = sorted(rng.sample([6, 8, 10, 12, 14, 16, 20, 24], rng.choice([2, 3, 4])))
        return {"kind": "batch", "prec": prec, "reliable": rel, "sizes": ",".join(map(str, sizes)),
                "each": rng.choice([1, 2, 3]), "tol": 1e-10}
    sizes = sorted(rng.sample([6, 8, 10, 12, 16], 2))
    return {"kind": "server", "prec": "f16", "reliable": "df64", "sizes": ",".join(map(str, sizes)),
            "requests": rng.choice([2, 4, 8]), "nsrc": rng.choice([1, 2, 4]), "tol": 1e-10}


# ------------------------------------------------------------------ inputs
def _dims(case):
    return tuple(int(v) for v in case["dims"].split("x"))


def _vol(dims):
    return dims[0] * dims[1] * dims[2] * dims[3]


def _randn(shape, gen):
    return torch.view_as_complex(torch.randn(*shape, 2, generator=gen, device="cuda", dtype=torch.float64))


def _unit(v):
    return v / torch.sqrt((v.abs() ** 2).sum(1, keepdim=True))


def _gauge(dims, gen):
    """Four device tensors of V*9 entries: SU(3) links near 1."""
    V, out = _vol(dims), []
    one = torch.eye(3, device="cuda", dtype=torch.complex128)
    for _ in range(4):
        a = _randn((V, 3, 3), gen)
        a = (a + a.conj().transpose(1, 2)) / 2
        w = one + 1j * EPS * a
        r0 = _unit(w[:, 0])
        r1 = w[:, 1]
        r1 = _unit(r1 - (r0.conj() * r1).sum(1, keepdim=True) * r0)
        r2 = torch.stack([r0[:, 1] * r1[:, 2] - r0[:, 2] * r1[:, 1], r0[:, 2] * r1[:, 0] - r0[:, 0] * r1[:, 2],
                          r0[:, 0] * r1[:, 1] - r0[:, 1] * r1[:, 0]], 1).conj()
        out.append(torch.stack([r0, r1, r2], 1).reshape(-1))
    return out


def _source(dims, gen):
    s = _randn((_vol(dims) * 12,), gen)
    return s / torch.linalg.vector_norm(s)


def _gen(seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 1000 + salt)
    return g


def _pinned(n):
    return torch.empty(n, dtype=torch.complex128, pin_memory=True)


def _host(t, pinned=True):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=pinned)
    h.copy_(t)
    return h


def _lattice(dims, gen):
    return _ctx().lattice(dims, [_host(g).numpy() for g in _gauge(dims, gen)])


def _ptr(t):
    return C.c_void_p(t.data_ptr())


def _fetch(field, out):
    field.lat.ctx.check(wd.lib.wd_field_download(field.lat.ctx.handle, field.handle, _ptr(out)))
    return out


def _batch_lats(case):
    """(dims, mass) of every system of a batch of lattices."""
    out = []
    for i, L in enumerate(int(v) for v in case["sizes"].split(",")):
        for k in range(case["each"]):
            out.append(((L, L, L, 2 * L), 0.05 + 0.15 * ((3 * i + 5 * k) % 8) / 8))
    return out


def _server_requests(case, seed):
    """(lattice index, mass, source seeds) of every request of a burst."""
    return [(r % 2, 0.02 + 0.18 * ((5 * r) % 8) / 8, [seed * 7919 + 100 * r + k + 1 for k in range(case["nsrc"])])
            for r in range(case["requests"])]


def prepare(case, seed):
    kind, ctx, gen = case["kind"], _ctx(), _gen(seed)
    s = {"case": case, "ctx": ctx}
    if kind in ("op", "cg", "hostcg", "host", "prop"):
        dims = _dims(case)
        s["dims"] = dims
        n = _vol(dims) * 12
    if kind == "op":
        p = PREC[case["prec"]]
        s["lat"] = lat = _lattice(dims, gen)
        s["f"] = [lat.field(_host(_source(dims, gen)).numpy(), prec=p), lat.field(prec=p), lat.field(prec=p)]
        s["out"] = _pinned(n)
    elif kind == "host":
        s["ctx"] = wd.Context(0)  # a context keeps one configuration's links for the host-buffer calls
        s["gauge"] = [_host(g, case["pinned"]).numpy() for g in _gauge(dims, gen)]
        s["src"] = _host(_source(dims, gen), case["pinned"])
        s["out"] = _host(torch.zeros(n, dtype=torch.complex128), case["pinned"])
        s["args"] = (wd._dims(dims), wd._gauge_ptrs(s["gauge"]), _ptr(s["src"]), _ptr(s["out"]))
    elif kind == "hostcg":
        s["ctx"] = wd.Context(0)
        s["gauge"] = [_host(g, False).numpy() for g in _gauge(dims, gen)]
        s["src"] = _host(_source(dims, gen), False).numpy()
        s["out"] = np.empty(n, np.complex128)
        s["params"] = wd.solver_params(kind=wd.CGNR_REF, mass=case["mass"], tol=case["tol"], max_iter=2000)
    elif kind == "cg":
        s["lat"] = lat = _lattice(dims, gen)
        s["b"], s["x"] = lat.field(_host(_source(dims, gen)).numpy()), lat.field()
        s["out"] = _pinned(n)
        s["params"] = wd.solver_params(mass=case["mass"], tol=case["tol"], max_iter=5000, prec=PREC[case["prec"]],
                                       prec_reliable=PREC[case["reliable"]])
    elif kind == "prop":
        s["lat"] = lat = _lattice(dims, gen)
        s["props"] = [lat.field() for _ in range(12)]
        s["arr"] = (C.c_void_p * 12)(*[f.handle.value for f in s["props"]])
        s["out"] = [_pinned(n) for _ in range(12)]
        s["ct"] = np.zeros(dims[3])
        s["params"] = wd.solver_params(mass=case["mass"], tol=case["tol"], max_iter=5000, prec=PREC[case["prec"]],
                                       prec_reliable=PREC[case["reliable"]])
    elif kind == "batch":
        s["systems"], s["out"] = [], []
        for dims, mass in _batch_lats(case):
            lat = _lattice(dims, gen)
            s["systems"].append((lat, lat.field(_host(_source(dims, gen)).numpy()), lat.field(), mass))
            s["out"].append(_pinned(_vol(dims) * 12))
        s["params"] = wd.solver_params(tol=case["tol"], max_iter=5000, prec=PREC[case["prec"]],
                                       prec_reliable=PREC[case["reliable"]])
    else:
        s["server"] = sv = wd.Server(ctx, prec=PREC[case["prec"]], prec_reliable=PREC[case["reliable"]])
        sizes = [(L, L, L, 2 * L) for L in (int(v) for v in case["sizes"].split(","))]
        s["ids"] = [sv.add_lattice(d, [_host(g).numpy() for g in _gauge(d, gen)]) for d in sizes]
        s["requests"] = _server_requests(case, seed)
        s["out"] = [[_pinned(_vol(sizes[l]) * 12) for _ in seeds] for l, _, seeds in s["requests"]]
    torch.cuda.synchronize()
    return s


# --------------------------------------------------------------------- run
def _apply(case, lat, src, dst, i):
    """Application i of a chain: the operator and its adjoint in turn."""
    p = PREC[case["prec"]]
    if case["op"] == "full":
        lat.dslash_full(src, dst, case["mass"], i & 1, p)
    elif case["op"] == "offd":
        lat.dslash_offd(src, dst, (i >> 1) & 1, i & 1, p)
    else:
        lat.dslash_eo(src, dst, (i >> 1) & 1, i & 1, p)


def run(s):
    case, ctx = s["case"], s["ctx"]
    kind = case["kind"]
    if kind == "op":
        src, a, b = s["f"]
        if case["op"] == "eo":  # leaves the other parity as it is: start from zero
            a.zero()
            b.zero()
        for i in range(case["reps"]):
            _apply(case, s["lat"], src, a, i)
            src, a, b = a, b, a
        return _fetch(src, s["out"])
    if kind == "host":
        if case["op"] == "offd":
            ctx.check(wd.lib.wd_host_dslash_offd(ctx.handle, *s["args"], 0, 0))
        else:
            ctx.check(wd.lib.wd_host_dslash_full(ctx.handle, *s["args"], case["mass"], 0))
        return s["out"]
    if kind == "hostcg":
        s["out"][:] = 0
        ctx.host_cg(s["dims"], s["gauge"], s["src"], s["out"], s["params"])
        return s["out"]
    if kind == "cg":
        s["lat"].solve(s["b"], s["x"], s["params"])
        return _fetch(s["x"], s["out"])
    if kind == "prop":
        stats = (wd.SolverStats * 12)()
        ctx.check(wd.lib.wd_propagator(ctx.handle, s["lat"].handle, (C.c_int * 4)(1, 0, 0, 0), C.byref(s["params"]),
                                       s["arr"], stats))
        ct = s["lat"].pion_correlator(s["props"])
        return {"pion": ct, "props": [_fetch(f, o) for f, o in zip(s["props"], s["out"])]}
    if kind == "batch":
        ctx.solve_batch(s["systems"], s["params"])
        return [_fetch(x, o) for (_, _, x, _), o in zip(s["systems"], s["out"])]
    sv = s["server"]
    rids = [sv.submit(s["ids"][l], len(seeds), mass, case["tol"], seeds=seeds) for l, mass, seeds in s["requests"]]
    todo = set(range(len(rids)))
    while todo:
        sv.step()
        for r in sorted(todo):
            n = len(s["out"][r])
            done, stats, lat_s = C.c_int(), (wd.SolverStats * n)(), C.c_double()
            sols = (C.c_void_p * n)(*[o.data_ptr() for o in s["out"][r]])
            ctx.check(wd.lib.wd_server_poll(sv.handle, rids[r], C.byref(done), sols, stats, C.byref(lat_s)))
            if done.value:
                todo.remove(r)
    return s["out"]


# -------------------------------------------------------------------- work
_ITERS = 30  # CG iterations that a solve of these masses takes, to a few


def work(case):
    kind = case["kind"]
    if kind == "op":
        V, r = _vol(_dims(case)), case["reps"]
        sites = V * (1.0 if case["op"] == "full" else 0.5)
        p = case["prec"]
        # every application reads the links and a spinor and writes one; the result comes down in FP64
        per = V * LINK_BYTES[p] + (2 * V if case["op"] == "full" else V) * SPINOR_BYTES[p]
        return {"bytes": r * per, "flops": r * sites * HOP_FLOPS}
    if kind == "host":
        V = _vol(_dims(case))
        full = case["op"] == "full"
        return {"bytes": V * LINK_BYTES["f64"] + (2 * V if full else V) * 192, "flops": V * (1 if full else 0.5) * HOP_FLOPS}
    if kind in ("hostcg", "cg", "prop"):
        V = _vol(_dims(case))
        p = case.get("prec", "f64")
        hops = _ITERS * (4 if kind != "hostcg" else 10)  # half-lattice hopping terms (the full-lattice CG takes more iterations)
        nsys = 12 if kind == "prop" else 1
        return {"bytes": hops * (V * LINK_BYTES[p] + nsys * V * SPINOR_BYTES[p]),
                "flops": hops * nsys * V * 0.5 * HOP_FLOPS}
    if kind == "batch":
        vols = [_vol(d) for d, _ in _batch_lats(case)]
    else:
        L = [int(v) for v in case["sizes"].split(",")]
        vols = [2 * L[l] ** 4 for l, _, seeds in _server_requests(case, 0) for _ in seeds]
    p, hops = case["prec"], 4 * _ITERS
    return {"bytes": hops * sum(vols) * (LINK_BYTES[p] * (1 if kind == "batch" else 0) + SPINOR_BYTES[p]),
            "flops": hops * sum(vols) * 0.5 * HOP_FLOPS}


# ------------------------------------------------------------------- exact
def _order(dims):
    """Lexicographic index of every entry of the even-odd order."""
    x, y, z, t = dims
    i = torch.arange(_vol(dims), device="cuda")
    c = (i % x + (i // x) % y + (i // (x * y)) % z + i // (x * y * z)) & 1
    return torch.argsort(c * _vol(dims) + i)  # even sites first, each parity in lexicographic order


class _Wilson:
    """The operator in plain torch, FP64, on (t, z, y, x, spin, colour) grids."""

    def __init__(self, dims, gauge):
        self.dims, self.order = dims, _order(dims)
        self.grid = (dims[3], dims[2], dims[1], dims[0])
        self.U = [self._lex(g.reshape(-1, 9)).reshape(*self.grid, 3, 3) for g in gauge]

    def _lex(self, v):
        out = torch.empty_like(v)
        out[self.order] = v
        return out

    def lex(self, psi):
        return self._lex(psi.reshape(-1, 12)).reshape(*self.grid, 4, 3)

    def eo(self, g):
        return g.reshape(-1, 12)[self.order].reshape(-1)

    def mask(self, cb):
        m = torch.zeros(_vol(self.dims), 1, device="cuda", dtype=torch.float64)
        m[self.order[cb * (_vol(self.dims) // 2):(cb + 1) * (_vol(self.dims) // 2)]] = 1.0
        return m.reshape(*self.grid, 1, 1)

    def hop(self, psi, dag):
        out = torch.zeros_like(psi)
        for mu in range(4):
            ax = 3 - mu
            for fwd in (True, False):
                sg = (-1.0 if fwd else 1.0) * (-1.0 if dag else 1.0)
                nb = torch.roll(psi, -1 if fwd else 1, ax)
                s0, s1, s2, s3 = (nb[..., k, :] for k in range(4))
                if mu == 0:
                    h = (s0 + sg * 1j * s3, s1 + sg * 1j * s2)
                elif mu == 1:
                    h = (s0 - sg * s3, s1 + sg * s2)
                elif mu == 2:
                    h = (s0 + sg * 1j * s2, s1 - sg * 1j * s3)
                else:
                    h = (s0 + sg * s2, s1 + sg * s3)
                U = self.U[mu] if fwd else torch.roll(self.U[mu], 1, ax)
                t = []
                for v in h:
                    if fwd:
                        t.append(sum(U[..., :, b] * v[..., b:b + 1] for b in range(3)))
                    else:
                        t.append(sum(U[..., b, :].conj() * v[..., b:b + 1] for b in range(3)))
                out[..., 0, :] += t[0]
                out[..., 1, :] += t[1]
                if mu == 0:
                    out[..., 2, :] -= sg * 1j * t[1]
                    out[..., 3, :] -= sg * 1j * t[0]
                elif mu == 1:
                    out[..., 2, :] += sg * t[1]
                    out[..., 3, :] -= sg * t[0]
                elif mu == 2:
                    out[..., 2, :] -= sg * 1j * t[0]
                    out[..., 3, :] += sg * 1j * t[1]
                else:
                    out[..., 2, :] += sg * t[0]
                    out[..., 3, :] += sg * t[1]
        return -0.5 * out

    def full(self, psi, mass, dag):
        return (4.0 + mass) * psi + self.hop(psi, dag)

    def solve(self, b, mass, tol=1e-13):
        x = torch.zeros_like(b)
        r = self.full(b, mass, 1)
        p, rr = r.clone(), (r.abs() ** 2).sum()
        stop = tol * tol * rr
        for _ in range(1000):
            q = self.full(p, mass, 0)
            al = rr / (q.abs() ** 2).sum()
            x += al * p
            r -= al * self.full(q, mass, 1)
            new = (r.abs() ** 2).sum()
            if new <= stop:
                break
            p = r + (new / rr) * p
            rr = new
        return x


def exact(case, seed):
    kind, gen = case["kind"], _gen(seed)
    if kind in ("op", "host"):
        dims = _dims(case)
        W = _Wilson(dims, _gauge(dims, gen))
        v = W.lex(_source(dims, gen))
        if kind == "host":
            v = W.mask(0) * W.hop(v, 0) if case["op"] == "offd" else W.full(v, case["mass"], 0)
        else:
            for i in range(case["reps"]):
                if case["op"] == "full":
                    v = W.full(v, case["mass"], i & 1)
                else:
                    v = W.mask(i & 1) * W.hop(v, (i >> 1) & 1)
        return W.eo(v).cpu()
    if kind in ("cg", "hostcg"):
        dims = _dims(case)
        if _vol(dims) > 1 << 18:
            return None
        W = _Wilson(dims, _gauge(dims, gen))
        return W.eo(W.solve(W.lex(_source(dims, gen)), case["mass"])).cpu()
    if kind == "prop":
        dims = _dims(case)
        if _vol(dims) > 1 << 15:
            return None
        W = _Wilson(dims, _gauge(dims, gen))
        props, ct = [], torch.zeros(dims[3], dtype=torch.float64, device="cuda")
        for k in range(12):
            b = torch.zeros(*W.grid, 4, 3, dtype=torch.complex128, device="cuda")
            b[0, 0, 0, 1, k // 3, k % 3] = 1.0
            x = W.solve(b, case["mass"])
            ct += (x.abs() ** 2).sum((1, 2, 3, 4, 5))
            props.append(W.eo(x).cpu())
        return {"pion": ct.cpu(), "props": props}
    if kind == "batch":
        out = []
        for dims, mass in _batch_lats(case):
            W = _Wilson(dims, _gauge(dims, gen))
            b = W.lex(_source(dims, gen))
            out.append(W.eo(W.solve(b, mass)).cpu() if _vol(dims) <= 1 << 18 else None)
        return out
    return None  # the server draws its own sources
