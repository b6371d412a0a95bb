"""Timed calls of the framework, one per way it is used.

A case is one call a program makes through the public Python entry points:

  apply  opr * x, mul!(out, opr, x, a, b) or a stack of vectors through
         apply_into, on a resident operator and device vectors (the inner
         call of every iterative solve);
  build  an operator built from its geometry and applied once (the start of
         every program that has no kernel cache);
  solve  (1 - chi G) t = i, ComplexF32 Krylov with FP64 reliable updates.

Operators of `apply` and `solve` are created from a Fourier kernel held by
the caller (egoFur, what the kernel caches store): the dyadic free-space Green
function sampled on the circulant separations, embedded and transformed here
with torch, so that `exact` can apply the same kernel with torch alone.
Cell counts are even (the framework evens odd ones) and every circulant
length srcCel + trgCel is a product of 2, 3, 5 and 7 (what it accepts).
"""
from __future__ import annotations

import importlib.util
import math
import os
import sys
from fractions import Fraction

import numpy as np
import torch

PKG = os.path.join("gilaelectromagnetics.jl_b200", "__init__.py")
DT = {"c128": (torch.complex128, np.complex128), "c64": (torch.complex64, np.complex64)}
SOLVE_TOL = 1e-11
ALPHA, BETA = 0.5 - 2j, 0.5 + 0.25j  # |beta| < 1: repeated passes on one output stay finite


def _gila():
    """The package (its folder's name is not an importable identifier)."""
    if "gila_b200" in sys.modules:
        return sys.modules["gila_b200"]
    path = os.path.abspath(PKG)
    spec = importlib.util.spec_from_file_location("gila_b200", path,
                                                  submodule_search_locations=[os.path.dirname(path)])
    mod = importlib.util.module_from_spec(spec)
    sys.modules["gila_b200"] = mod
    spec.loader.exec_module(mod)
    return mod


# ------------------------------------------------------------------- cases
def _case(kind, trg, src=None, off=0, dt="c128", nrhs=1, form="mul"):
    """src None: a self operator; else source cells and the target's offset
    along x in cells.  form (apply): "mul" is opr * x, "axpby" is mul! with
    alpha and beta, "stack" is apply_into on nrhs stacked vectors."""
    c = {"kind": kind, "nx": trg[0], "ny": trg[1], "nz": trg[2], "dt": dt, "nrhs": nrhs, "form": form,
         "self": src is None}
    s = trg if src is None else src
    c.update({"sx": s[0], "sy": s[1], "sz": s[2], "off": off})
    return c


def listed():
    def named(name, *a, **kw):
        return dict(_case(*a, **kw), name=name)

    return [
        # the volumes of the reference's own tests: latency and launches
        named("self_16x16x16_c128", "apply", (16, 16, 16)),
        # a small scatterer at a ragged size, inside an iterative solver
        named("axpby_50x40x30_c128", "apply", (50, 40, 30), form="axpby"),
        # ordinary user volumes whose sizes are not powers of two
        named("self_100x84x60_c128", "apply", (100, 84, 60)),
        named("self_180x140x90_c64", "apply", (180, 140, 90), dt="c64"),
        # two volumes apart (the benchmark's external operator)
        named("ext_64x64x64_to_64x64x32_c128", "apply", (64, 64, 32), (64, 64, 64), 80),
        # the benchmark's volumes, both precisions, and a block of vectors
        named("self_128x128x64_c128", "apply", (128, 128, 64)),
        named("stack8_96x96x48_c64", "apply", (96, 96, 48), dt="c64", nrhs=8, form="stack"),
        named("self_192x192x96_c64", "apply", (192, 192, 96), dt="c64"),
        named("self_256x256x128_c128", "apply", (256, 256, 128)),
        # an operator from its geometry, then its first product
        named("build_self_32x32x32", "build", (32, 32, 32)),
        named("build_ext_24x20x16_to_16x16x12", "build", (16, 16, 12), (24, 20, 16), 30),
        # scattering by a lossy inhomogeneous inclusion, two incident fields
        named("solve_64x64x32_x2", "solve", (64, 64, 32), nrhs=2),
    ]


def _smooth(n):
    for q in (2, 3, 5, 7):
        while n % q == 0:
            n //= q
    return n == 1


def _axis(rng, lo, hi):
    """An even 7-smooth cell count, spread over the logarithm of [lo, hi]."""
    while True:
        n = 2 * int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / 2))
        if lo <= n <= hi and _smooth(n):
            return n


def _cells(rng, lo, hi, most, div=1):
    while True:
        c = tuple(_axis(rng, lo, hi) for _ in range(3))
        if c[0] * c[1] * c[2] * div <= most:
            return c


def draw(rng):
    """Volumes of 8 to 256 cells an axis (a thinner third axis where 256^3
    would be left), any shape that the framework takes."""
    u = rng.random()
    if u < 0.5:
        dt, form = rng.choice(("c128", "c64")), rng.choice(("mul", "mul", "axpby", "stack"))
        nrhs = rng.randint(2, 8) if form == "stack" else 1
        return _case("apply", _cells(rng, 8, 256, 256 * 256 * 128, nrhs), dt=dt, nrhs=nrhs, form=form)
    if u < 0.7:
        dt = rng.choice(("c128", "c64"))
        while True:
            t, s = _cells(rng, 8, 128, 128 * 128 * 128), _cells(rng, 8, 128, 128 * 128 * 128)
            if all(_smooth(a + b) for a, b in zip(t, s)):
                return _case("apply", t, s, (t[0] + s[0]) // 2 + rng.randint(2, 40), dt=dt)
    if u < 0.8:
        return _case("build", _cells(rng, 8, 48, 32 * 32 * 32))
    if u < 0.9:
        while True:
            t, s = _cells(rng, 8, 24, 16 * 16 * 16), _cells(rng, 8, 24, 16 * 16 * 16)
            if all(_smooth(a + b) for a, b in zip(t, s)):
                return _case("build", t, s, (t[0] + s[0]) // 2 + rng.randint(2, 40))
    return _case("solve", _cells(rng, 12, 96, 64 * 64 * 32, 1), nrhs=rng.randint(1, 2))


# ------------------------------------------------------------------ inputs
def _gen(seed, salt):
    return torch.Generator(device="cuda").manual_seed(1000003 * (seed % 1000003) + salt)


def _randn(shape, dtype, seed, salt):
    return torch.randn(shape, dtype=dtype, device="cuda", generator=_gen(seed, salt))


def _scl(seed):
    """Cells of about 1/32 wavelength, another size for each seed."""
    return Fraction(1, 28 + seed % 9)


def _sizes(c):
    t, s = (c["nx"], c["ny"], c["nz"]), (c["sx"], c["sy"], c["sz"])
    return t, s, tuple(a + b for a, b in zip(t, s))


def _stored(c):
    """Stored kernel entries per parity branch and axis: half of them where
    the two volumes have the same extent and centre on the axis."""
    t, s, P = _sizes(c)
    half = [t[d] == s[d] and not (d == 0 and c["off"]) for d in range(3)]
    return [max(n // 2 + 1, 2) if h else p // 2 for n, p, h in zip(t, P, half)]


def _separations(c, scl, d):
    """Separation of target and source cell at each circulant index of axis
    d; index trgCel is not a separation (its entries are zero)."""
    t, s, P = _sizes(c)
    m = torch.arange(P[d], dtype=torch.float64, device="cuda")
    t0 = (c["off"] if d == 0 else 0) - (t[d] - 1) / 2 + (s[d] - 1) / 2
    return torch.where(m < t[d], m, m - P[d]).add(t0).mul(float(scl))


def _green(c, scl, dtype):
    """The six transformed circulant components (xx, yy, zz, xy, xz, yz),
    each [Pz, Py, Px], rounded to dtype."""
    t, _, P = _sizes(c)
    x, y, z = (_separations(c, scl, d) for d in range(3))
    r = (x[None, None, :], y[None, :, None], z[:, None, None])
    k = 2 * math.pi
    rr = (r[0] * r[0] + r[1] * r[1] + r[2] * r[2]).sqrt()
    far = rr > 0
    kr = torch.where(far, rr, torch.ones_like(rr)).mul(k)
    g = torch.polar(float(scl) ** 3 * k ** 3 / (4 * math.pi * kr), kr)
    one = 1 + torch.complex(-1 / kr ** 2, 1 / kr)
    two = g * torch.complex(3 / kr ** 2 - 1, -3 / kr)
    one = g * one
    del g
    dead = [torch.arange(P[d], device="cuda") == t[d] for d in range(3)]
    zero = dead[0][None, None, :] | dead[1][None, :, None] | dead[2][:, None, None]
    for a, b in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)):
        v = two * (r[a] * r[b] * (k * k) / kr ** 2)
        if a == b:
            v += one
            v = torch.where(far, v, torch.full_like(v, -1 / 3))
        v.masked_fill_(zero, 0)
        yield torch.fft.fftn(v).to(dtype)


def _operator(c, seed, dtype, ndt):
    """The operator on egoFur: for each parity branch (4 px + 2 py + pz) the
    array (x, y, z, 6, 1, 1) of its stored entries."""
    gila = _gila()
    t, s, _ = _sizes(c)
    scl = _scl(seed)
    parts = [[] for _ in range(8)]
    keep = _stored(c)
    for comp in _green(c, scl, dtype):
        for e in range(8):
            b = comp[e & 1::2, (e >> 1) & 1::2, (e >> 2) & 1::2]
            parts[e].append(b[:keep[2], :keep[1], :keep[0]].contiguous().cpu().numpy())
    fur = [np.stack(p).transpose(3, 2, 1, 0)[..., None, None] for p in parts]
    sc = (scl, scl, scl)
    trg = gila.GlaVol(t, sc, (c["off"] * scl, 0, 0) if not c["self"] else (0, 0, 0))
    src = None if c["self"] else gila.GlaVol(s, sc, (0, 0, 0))
    return gila.GlaOpr(gila.GlaOprMem(gila.GlaKerOpt(True), trg, src, egoFur=fur, setTyp=ndt))


def _vectors(c, seed):
    """Currents (nrhs, 3, z, y, x) with normal real and imaginary parts."""
    lead = (c["nrhs"],) if c["nrhs"] > 1 else ()
    dtype = DT[c["dt"]][0]
    x = _randn((*lead, 3, c["sz"], c["sy"], c["sx"]), dtype, seed, 1)
    y = _randn((*lead, 3, c["nz"], c["ny"], c["nx"]), dtype, seed, 2)
    return x, y


def _medium(c, seed):
    """An inclusion in the middle half of the volume, susceptibility uniform
    in [0, 1.5] with some loss."""
    shp = (c["nz"], c["ny"], c["nx"])
    chi = torch.zeros(shp, dtype=torch.complex128, device="cuda")
    box = tuple(slice(n // 4, n - n // 4) for n in shp)
    u = torch.rand(shp, dtype=torch.float64, device="cuda", generator=_gen(seed, 3))
    chi[box] = torch.complex(1.5 * u, torch.full_like(u, 0.1))[box]
    return chi


def prepare(case, seed):
    c = case
    dtype, ndt = DT[c["dt"]]
    x, y = _vectors(c, seed)
    st = {"case": c, "x": x, "out": y}
    if c["kind"] == "build":
        gila = _gila()
        sc = (_scl(seed),) * 3
        t, s, _ = _sizes(c)
        st["trg"] = gila.GlaVol(t, sc, (c["off"] * sc[0], 0, 0) if not c["self"] else (0, 0, 0))
        st["src"] = None if c["self"] else gila.GlaVol(s, sc, (0, 0, 0))
        return st
    st["opr"] = _operator(c, seed, dtype, ndt)
    if c["kind"] == "solve":
        st["ls"] = _gila().LippmannSchwinger(st["opr"], _medium(c, seed))
        st["ls"].g32()
    torch.cuda.synchronize()
    return st


def run(state):
    gila, c = _gila(), state["case"]
    if c["kind"] == "build":
        mem = gila.GlaOprMem(gila.GlaKerOpt(True), state["trg"], state["src"])
        return gila.GlaOpr(mem) * state["x"]
    if c["kind"] == "solve":
        # tight enough that the field itself, not its last correction, is
        # what two runs have in common
        t, _ = gila.solve(state["ls"], state["x"], tol=SOLVE_TOL, mixed=True)
        return t
    if c["form"] == "stack":
        return state["opr"].mem.apply_into(state["x"], state["out"], nrhs=c["nrhs"])
    if c["form"] == "axpby":
        return gila.mul(state["out"], state["opr"], state["x"], ALPHA, BETA)
    return state["opr"] * state["x"]


def work(case):
    """Bytes: the transforms of a matvec that keeps one z line of the padded
    spectrum on chip at a time (input, x/y-transformed planes out and in,
    kernel, planes out and in, output); a build writes its kernel; a solve
    is counted as 60 matvecs a field.  Flops: 5 n log2 n a transform of
    length n, 66 a frequency for the 3 x 3 product; an integrand of the
    build's quadratures as 100."""
    c = case
    t, s, P = _sizes(c)
    b = 16 if c["dt"] == "c128" else 8
    vt, vs, vp = t[0] * t[1] * t[2], s[0] * s[1] * s[2], P[0] * P[1] * P[2]
    ker = 8 * math.prod(_stored(c))
    byt = b * (3 * vs + 6 * P[0] * P[1] * s[2] + 6 * P[0] * P[1] * t[2] + 3 * vt)

    def fft(n):
        return 5 * n * math.log2(n)

    flops = 66 * vp + 6 * P[0] * P[1] * fft(P[2])
    for v in (s, t):
        flops += 3 * v[2] * (v[1] * fft(P[0]) + P[0] * fft(P[1]))
    if c["kind"] == "build":
        # one 57-point rule for each of 24 face pairs of each separation, the
        # six circulant transforms
        pairs = vt if c["self"] else vp
        return {"bytes": byt + b * 6 * ker + 2 * 6 * b * vp,
                "flops": flops + pairs * 24 * 57 * 100 + 6 * vp * 5 * math.log2(vp)}
    n = c["nrhs"]
    if c["kind"] == "solve":
        return {"bytes": 60 * n * byt / 2 + 60 * b * 6 * ker / 2, "flops": 60 * n * flops}
    if c["form"] == "axpby":
        byt += b * 3 * vt
    return {"bytes": n * byt + b * 6 * ker, "flops": n * flops}


# ------------------------------------------------------------------- exact
def _apply_exact(c, green, x):
    """The circular convolution, one source component's transform at a time."""
    t, s, P = _sizes(c)
    X = [torch.fft.fftn(x[k], s=(P[2], P[1], P[0])) for k in range(3)]
    at = ((0, 3, 4), (3, 1, 5), (4, 5, 2))
    out = []
    for i in range(3):
        Y = sum(green[at[i][k]] * X[k] for k in range(3))
        out.append(torch.fft.ifftn(Y)[:t[2], :t[1], :t[0]])
    return torch.stack(out)


def _solve_exact(mul, b):
    """Restarted GMRES to the last digits of FP64."""
    x, r, m = torch.zeros_like(b), b.clone(), 60
    want = 1e-14 * float(torch.linalg.vector_norm(b))
    for _ in range(8):
        beta = torch.linalg.vector_norm(r)
        if float(beta) <= want:
            break
        V, H = [r / beta], torch.zeros(m + 1, m, dtype=b.dtype, device=b.device)
        for j in range(m):
            w = mul(V[j])
            for _ in range(2):  # orthogonalised twice
                for i in range(j + 1):
                    h = torch.vdot(V[i].reshape(-1), w.reshape(-1))
                    H[i, j] += h
                    w = w - h * V[i]
            H[j + 1, j] = torch.linalg.vector_norm(w)
            V.append(w / H[j + 1, j])
        e = torch.zeros(m + 1, dtype=b.dtype, device=b.device)
        e[0] = beta
        y = torch.linalg.lstsq(H, e[:, None]).solution[:, 0]
        for j in range(m):
            x = x + y[j] * V[j]
        r = b - mul(x)
    return x


def exact(case, seed):
    """None for a build: its integrals are defined by their quadrature."""
    c = case
    if c["kind"] == "build":
        return None
    green = [g.to(torch.complex128) for g in _green(c, _scl(seed), DT[c["dt"]][0])]
    x, y = (v.to(torch.complex128) for v in _vectors(c, seed))
    xs = x if c["nrhs"] > 1 else x[None]
    if c["kind"] == "solve":
        chi = _medium(c, seed)
        got = torch.stack([_solve_exact(lambda v: v - chi * _apply_exact(c, green, v), f) for f in xs])
    else:
        got = torch.stack([_apply_exact(c, green, f) for f in xs])
    got = got if c["nrhs"] > 1 else got[0]
    if c["form"] == "axpby":
        got = ALPHA * got + BETA * y
    return got
