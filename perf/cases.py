"""The work a user of this library has it do, as cases that can be timed and compared.

Each case is one call pattern of the public interface (the Python package and, where results go to
device buffers of the caller, the C ABI beneath it) on a periodic lattice of lx*ly*lz*lt sites with
Ls fifth-dimension slices and nrhs right-hand sides.  Inputs are random SU(3) links and Gaussian
spinors, the distributions that the reference's table generator documents.  Results come back as the
user reads them: every output spinor, whole, in the reference layout.

Kinds:
  hop      a chain of hopping terms, alternating Dhop and DhopDag (polynomial filters, spectral
           estimates, the reference's own repetition loop)
  mdagm    Shamir M^dag M, the operator of every normal-equation solve
  schur    the even-odd Schur operator Mpc^dag Mpc
  mobius   Mobius M^dag M
  lanczos  Krylov steps written by the user from the operator and the vector operations
  seam     the drop-in dslash_kernel call on host buffers, as GridBench's drivers make it
  cg       a whole solve (full lattice or even-odd; plain, or mixed precision with FP16 or FP32 inside)
  batch    independent instances of different sizes in one call

"tune": the program ran the library's autotuner once for its shapes, as a long production run does;
short programs don't.
"""
import ctypes

import numpy as np
import torch

import gridbench_gb300 as gb

M5, MF = 1.8, 0.05          # domain-wall height and mass
MOBIUS_B, MOBIUS_C = 1.5, 0.5
TOL = 1e-10                 # solves: relative true residual, as the solver's own default

SPINOR = {"f64": 192, "f32": 96, "f16": 52}   # bytes of one 5D site
LINK = {"f64": 144, "f32": 72, "f16": 24}     # bytes of one link
PREC = {"f64": gb.F64, "f32": gb.F32, "f16": gb.F16}


def _case(name, kind, dims, Ls, **more):
    c = {"kind": kind, "lx": dims[0], "ly": dims[1], "lz": dims[2], "lt": dims[3], "Ls": Ls}
    if name:
        c["name"] = name
    c.update(more)
    return c


def listed():
    return [
        # the smallest call: one application on a test-sized lattice, where the launches count
        _case("hop_f32_4x4x4x4_Ls8", "hop", (4, 4, 4, 4), 8, prec="f32", nrhs=1, steps=1, tune=False),
        # the benchmark's lattice, in the chain that filters and spectral estimates make of it
        _case("hop_f32_16x16x16x16_Ls16", "hop", (16, 16, 16, 16), 16, prec="f32", nrhs=1, steps=6, tune=True),
        # twelve right-hand sides at once (the spin-colour components of a propagator)
        _case("hop_f32_24x24x24x24_Ls12_12rhs", "hop", (24, 24, 24, 24), 12, prec="f32", nrhs=12, steps=4, tune=True),
        # extents that are no powers of two, some odd, odd Ls, untuned: a local volume as it falls
        _case("hop_f32_15x9x21x14_Ls7", "hop", (15, 9, 21, 14), 7, prec="f32", nrhs=1, steps=4, tune=False),
        # the solver-sized lattice of the benchmark: the operator of a normal-equation solve
        _case("mdagm_f32_32x32x32x32_Ls16", "mdagm", (32, 32, 32, 32), 16, prec="f32", tune=True),
        # the even-odd operator of production solves on an elongated lattice
        _case("schur_f32_16x16x16x32_Ls12", "schur", (16, 16, 16, 32), 12, prec="f32", tune=True),
        # Mobius fermions with a short fifth dimension that is no power of two
        _case("mobius_f32_16x16x16x32_Ls10", "mobius", (16, 16, 16, 32), 10, prec="f32", tune=False),
        # eigenvector code on a small lattice: operator, dot products and vector updates in turn
        _case("lanczos_f32_12x12x12x12_Ls8", "lanczos", (12, 12, 12, 12), 8, prec="f32", steps=5, tune=False),
        # GridBench's bench_simple flow: host buffers in, host buffers out, doubles
        _case("seam_f64_8x8x8x8_Ls8", "seam", (8, 8, 8, 8), 8, prec="f64"),
        # a propagator solve through the even-odd operator, FP16 inside, FP64 true residuals
        _case("cg_eo_f16_16x16x16x16_Ls16", "cg", (16, 16, 16, 16), 16, system="eo", inner="f16", tune=True),
        # a normal-equation solve with FP64 vectors on a small lattice
        _case("cg_full_plain_12x12x12x12_Ls8", "cg", (12, 12, 12, 12), 8, system="full", inner="plain", tune=True),
        # many small instances at once: volumes and Ls of the benchmark's batch
        _case("batch_f32_20_up_to_16_Ls16", "batch", (16, 16, 16, 16), 16, n=20, spec=7),
    ]


def _extent(rng, lo, hi, even=False):
    n = int(round(2 ** rng.uniform(np.log2(lo), np.log2(hi))))
    return max(2, n + (n & 1)) if even else n


def _volume(rng, Ls, lo, hi, even=False, nrhs=1):
    """Extents whose 5D volume (times right-hand sides) is spread over lo..hi on its logarithm."""
    target = 2 ** rng.uniform(np.log2(lo), np.log2(hi)) / (Ls * nrhs)
    side = target ** 0.25
    dims = [_extent(rng, max(2, side * 0.7), max(3, side * 1.4), even) for _ in range(3)]
    lt = max(2, int(round(target / (dims[0] * dims[1] * dims[2]))))
    return dims + [max(2, lt + (lt & 1)) if even else lt]


def draw(rng):
    kind = rng.choice(["hop", "hop", "hop", "mdagm", "schur", "mobius", "lanczos", "seam", "cg", "batch"])
    Ls = rng.choice([4, 6, 8, 10, 12, 16, 16, 20, 24, 32, rng.randint(3, 24)])
    tune = rng.random() < 0.5
    if kind == "hop":
        prec = rng.choice(["f32", "f32", "f32", "f64"])
        nrhs = rng.choice([1, 1, 1, 2, 3, 4, 8, 12])
        dims = _volume(rng, Ls, 2e3, 1.2e7 if prec == "f32" else 1.5e6, nrhs=nrhs)
        return _case(None, kind, dims, Ls, prec=prec, nrhs=nrhs, steps=rng.randint(1, 6), tune=tune)
    if kind in ("mdagm", "mobius"):
        prec = rng.choice(["f32", "f32", "f32", "f64"])
        return _case(None, kind, _volume(rng, Ls, 2e3, 1.2e7 if prec == "f32" else 1.5e6), Ls, prec=prec, tune=tune)
    if kind == "schur":
        return _case(None, kind, _volume(rng, Ls, 4e3, 1.2e7, even=True), Ls, prec="f32", tune=tune)
    if kind == "lanczos":
        return _case(None, kind, _volume(rng, Ls, 2e3, 4e6), Ls, prec="f32", steps=rng.randint(2, 6), tune=tune)
    if kind == "seam":
        return _case(None, kind, _volume(rng, Ls, 2e3, 4e5), Ls, prec=rng.choice(["f64", "f32"]))
    if kind == "cg":
        system = rng.choice(["full", "eo"])
        most = 5e5 if system == "eo" else 1.4e5
        return _case(None, kind, _volume(rng, Ls, 8e3, most, even=system == "eo"), Ls, system=system,
                     inner=rng.choice(["f16", "f32", "plain"]), tune=tune)
    side = rng.choice([8, 10, 12, 14, 16])
    return _case(None, kind, [side] * 4, rng.choice([8, 12, 16]), n=rng.randint(2, 24), spec=rng.randint(0, 10 ** 6))


# ------------------------------------------------------------------ inputs
def _dims(case):
    return case["lx"], case["ly"], case["lz"], case["lt"]


def _vol(dims):
    return dims[0] * dims[1] * dims[2] * dims[3]


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _links(dims, gen, dtype):
    """Doubled random SU(3) links [site, 8, 3, 3] (complex): Gaussian rows made orthonormal, det 1;
    link mu + 4 is the adjoint of link mu one step back."""
    V = _vol(dims)
    a = torch.randn(V, 4, 2, 3, 2, generator=gen, device="cuda", dtype=torch.float64)
    a = torch.view_as_complex(a)
    r0 = a[:, :, 0] / torch.linalg.vector_norm(a[:, :, 0], dim=-1, keepdim=True)
    r1 = a[:, :, 1] - (r0.conj() * a[:, :, 1]).sum(-1, keepdim=True) * r0
    r1 = r1 / torch.linalg.vector_norm(r1, dim=-1, keepdim=True)
    r2 = torch.linalg.cross(r0, r1, dim=-1).conj()
    fwd = torch.stack((r0, r1, r2), dim=2)  # [site, 4, row, col]
    U = torch.empty(V, 8, 3, 3, device="cuda", dtype=torch.complex128)
    U[:, :4] = fwd
    for mu in range(4):
        back = fwd[:, mu].reshape(dims[3], dims[2], dims[1], dims[0], 3, 3).roll(1, dims=3 - mu)
        U[:, 4 + mu] = back.reshape(V, 3, 3).transpose(-1, -2).conj()
    return U.to(dtype)


def _spinor(dims, Ls, gen, dtype):
    """Gaussian spinor [site, Ls, 4, 3] (complex)."""
    real = torch.float64 if dtype == torch.complex128 else torch.float32
    return torch.view_as_complex(torch.randn(_vol(dims), Ls, 4, 3, 2, generator=gen, device="cuda", dtype=real))


def _cdtype(case):
    return torch.complex128 if case.get("prec") == "f64" or case["kind"] == "cg" else torch.complex64


def _inputs(case, seed):
    """Links and source spinors of a case, in the reference layout."""
    gen = _generator(seed)
    dims, Ls, dt = _dims(case), case["Ls"], _cdtype(case)
    U = _links(dims, gen, dt)
    sdims = (dims[0] // 2,) + tuple(dims[1:]) if case["kind"] == "schur" else dims
    return U, [_spinor(sdims, Ls, gen, dt) for _ in range(case.get("nrhs", 1))]


def _instances(case, seed):
    """Sizes of a batch's instances (by the case alone) and their inputs' seeds."""
    rng = np.random.default_rng(case["spec"])
    most, most_ls = case["lx"], case["Ls"]
    sides = [s for s in range(8, most + 1, 2)]
    out = []
    for k in range(case["n"]):
        s = int(rng.choice(sides))
        out.append(((s, s, s, s), int(rng.choice([n for n in (8, 12, 16) if n <= most_ls])), seed * 1000 + k))
    return out


def _host(t):
    return torch.view_as_real(t).reshape(-1).cpu().numpy()


def _ctype(t):
    return gb.F64 if t.dtype in (torch.float64, torch.complex128) else gb.F32


def _take(field, t, rhs=0):
    """A device tensor in the reference layout into one right-hand side of a field."""
    gb.check(gb.load().gbdw_field_import(field.h, rhs, ctypes.c_void_p(t.data_ptr()), _ctype(t)))
    return field


def _give(field, t, rhs=0):
    """One right-hand side of a field into a device tensor, queued behind what computes it."""
    gb.check(gb.load().gbdw_field_export_async(field.h, rhs, ctypes.c_void_p(t.data_ptr()), _ctype(t)))


_tuned = {}  # what the tuner's cache was last filled for: it is kept by precision and extent


def _tune(case, g, out, inp):
    """The autotuner, once for a shape, as a program runs it at its start."""
    if not case.get("tune"):
        return
    key = (g.prec, inp.prec, inp.nrhs * inp.lat.info()["Ls"], getattr(g.lat, "parity", -1) >= 0)
    if _tuned.get(key) != _dims(case):
        gb.tune_dhop(g, out, inp)
        _tuned[key] = _dims(case)


def _buffer(V, Ls, n, dtype):
    real = torch.float64 if dtype in (gb.F64, torch.complex128) else torch.float32
    return torch.empty(n, V * Ls * 24, device="cuda", dtype=real)


# ------------------------------------------------------------------ what a program has in hand
def prepare(case, seed):
    kind, dims, Ls = case["kind"], _dims(case), case["Ls"]
    V = _vol(dims)
    s = {"case": case}
    if kind == "batch":
        s["fields"], s["out"], G, O, I = [], [], [], [], []
        for d, ls, sd in _instances(case, seed):
            gen = _generator(sd)
            lat = gb.Lattice.periodic(d, ls)
            U, phi = _links(d, gen, torch.complex64), _spinor(d, ls, gen, torch.complex64)
            torch.cuda.synchronize()
            G.append(gb.Gauge(lat, _host(U), gb.F32))
            I.append(_take(gb.Field(lat, gb.F32), phi))
            O.append(gb.Field(lat, gb.F32))
            s["out"].append(_buffer(_vol(d), ls, 1, gb.F32)[0])
            gb.synchronize()
        s["outs"] = O
        s["batch"] = gb.Batch(G, O, I)
        gb.synchronize()
        return s
    U, phi = _inputs(case, seed)
    torch.cuda.synchronize()
    if kind == "seam":
        nbr, prm, nsite = gb.generate_table(dims, Ls)
        s.update(U=_host(U), phi=_host(phi[0]), nbr=nbr, prm=prm, nsite=nsite)
        s["out"] = np.empty_like(s["phi"])
        return s
    lat = s["lat"] = gb.Lattice.periodic(dims, Ls)
    if kind == "cg":
        host = _host(U)
        inner = case["inner"]
        low = gb.F16 if inner == "f16" else gb.F32
        g64, glow = gb.Gauge(lat, host, gb.F64), gb.Gauge(lat, host, low)
        x, y = gb.Field(lat, low).gaussian(1), gb.Field(lat, low)
        _tune(case, glow, y, x)
        if case["system"] == "eo":
            even, odd = lat.checkerboard()
            g64 = (g64.checkerboard(even), g64.checkerboard(odd))
            glow = (glow.checkerboard(even), glow.checkerboard(odd))
            _tune(case, glow[0], gb.Field(even, low), gb.Field(odd, low).gaussian(1))
        s["g64"], s["glow"] = g64, glow
        s["b"], s["x"] = _take(gb.Field(lat, gb.F64), phi[0]), gb.Field(lat, gb.F64)
        s["out"] = _buffer(V, Ls, 1, gb.F32)  # propagators are kept in single precision
        gb.synchronize()
        return s
    prec = PREC[case["prec"]]
    g = gb.Gauge(lat, _host(U), prec)
    if kind == "schur":
        even, odd = lat.checkerboard()
        s["ge"], s["go"] = g.checkerboard(even), g.checkerboard(odd)
        s["in"] = _take(gb.Field(odd, prec), phi[0])
        s["tmp"] = [gb.Field(odd, prec), gb.Field(even, prec), gb.Field(even, prec)]
        s["res"] = gb.Field(odd, prec)
        s["out"] = _buffer(V // 2, Ls, 1, prec)
        _tune(case, s["ge"], s["tmp"][1], s["in"])
        gb.synchronize()
        return s
    s["g"] = g
    nrhs = case.get("nrhs", 1)
    s["in"] = gb.Field(lat, prec, nrhs)
    for r in range(nrhs):
        _take(s["in"], phi[r], r)
    s["tmp"] = [gb.Field(lat, prec, nrhs) for _ in range(3 if kind == "lanczos" else 2)]
    s["res"] = gb.Field(lat, prec, nrhs)
    s["out"] = _buffer(V, Ls, nrhs, prec)
    _tune(case, g, s["res"], s["in"])
    gb.synchronize()
    return s


# ------------------------------------------------------------------ one pass
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "hop":
        src, bufs = s["in"], s["tmp"]
        for k in range(case["steps"]):
            gb.dhop(s["g"], bufs[k & 1], src, k & 1)
            src = bufs[k & 1]
        for r in range(case["nrhs"]):
            _give(src, s["out"][r], r)
        return s["out"]
    if kind == "mdagm":
        pap = gb.dwf_mdagm(s["g"], s["res"], s["tmp"][0], s["in"], M5, MF)
        _give(s["res"], s["out"][0])
        return {"psi": s["out"], "pap": pap}
    if kind == "schur":
        pap = gb.dwf_mpcdagmpc(s["go"], s["ge"], s["res"], *s["tmp"], s["in"], M5, MF)
        _give(s["res"], s["out"][0])
        return {"psi": s["out"], "pap": pap}
    if kind == "mobius":
        pap = gb.mobius_mdagm(s["g"], s["res"], s["tmp"][0], s["tmp"][1], s["in"], MOBIUS_B, MOBIUS_C, M5, MF)
        _give(s["res"], s["out"][0])
        return {"psi": s["out"], "pap": pap}
    if kind == "lanczos":
        t, (v, prev, w) = s["res"], s["tmp"]
        v.copy_from(s["in"])
        v.axpby(0.0, s["in"], 1.0 / v.norm2() ** 0.5)
        alpha, beta = [], []
        for k in range(case["steps"]):
            alpha.append(gb.dwf_mdagm(s["g"], w, t, v, M5, MF))
            w.axpby(-alpha[-1], v, 1.0)
            if k:
                w.axpby(-beta[-1], prev, 1.0)
            beta.append(w.norm2() ** 0.5)
            w.axpby(0.0, v, 1.0 / beta[-1])
            prev, v, w = v, w, prev
        _give(v, s["out"][0])
        overlap = prev.dot(v)
        return {"alpha": alpha, "beta": beta, "v": s["out"], "orthogonal": abs(overlap) < 1e-3}
    if kind == "seam":
        gb.dslash_kernel(1, s["U"], s["out"], s["phi"], s["nbr"], s["nsite"], case["Ls"], s["prm"])
        return s["out"]
    if kind == "cg":
        s["x"].zero()
        how = dict(tol=TOL, max_iter=5000)
        if case["inner"] == "plain":
            how.update(mode=gb.CG_PLAIN, delta=1e-4, g32=s["glow"])
        elif case["inner"] == "f32":
            how.update(mode=gb.CG_MIXED, delta=1e-4, gsloppy=s["glow"], sloppy_prec=gb.F32)
        else:
            how.update(mode=gb.CG_MIXED, delta=0.03, gsloppy=s["glow"], sloppy_prec=gb.F16, sloppy_residual=1)
        solve = gb.cg_solve_eo if case["system"] == "eo" else gb.cg_solve
        solve(s["g64"], s["x"], s["b"], M5, MF, **how)
        _give(s["x"], s["out"][0])
        return s["out"]
    s["batch"].run()
    for f, t in zip(s["outs"], s["out"]):
        _give(f, t)
    return s["out"]


# ------------------------------------------------------------------ what a pass cannot do without
def _hop_work(prec, V, Ls, nrhs=1):
    return V * Ls * nrhs * 2 * SPINOR[prec] + V * 8 * LINK[prec], 1320 * V * Ls * nrhs


def work(case):
    kind, Ls = case["kind"], case["Ls"]
    V = _vol(_dims(case))
    if kind == "batch":
        b = f = 0
        for d, ls, _ in _instances(case, 0):
            hb, hf = _hop_work("f32", _vol(d), ls)
            b, f = b + hb + 2 * 96 * _vol(d) * ls, f + hf
        return {"bytes": b, "flops": f}
    if kind == "cg":
        # about this many steps at this mass and tolerance; each is M^dag M and the vector updates
        steps = 200 if case["system"] == "eo" else 340
        inner = "f32" if case["inner"] == "plain" else case["inner"]
        hb, hf = _hop_work(inner, V, Ls)
        vec = 5 * 192 if case["inner"] == "plain" else 2 * 96 + 4 * SPINOR[inner]
        sites = V * Ls // 2 if case["system"] == "eo" else V * Ls
        return {"bytes": steps * (2 * hb + vec * sites), "flops": steps * 2 * (hf + 96 * V * Ls)}
    prec, nrhs = case["prec"], case.get("nrhs", 1)
    hb, hf = _hop_work(prec, V, Ls, nrhs)
    S = SPINOR[prec]
    read = V * Ls * nrhs * (S + (192 if prec == "f64" else 96))  # handing the result over
    if kind == "hop":
        return {"bytes": case["steps"] * hb + read, "flops": case["steps"] * hf}
    if kind in ("mdagm", "mobius"):
        return {"bytes": 2 * hb + read, "flops": 2 * (hf + 96 * V * Ls)}
    if kind == "schur":  # four hopping terms on half the sites, two of them with a diagonal part
        return {"bytes": 2 * hb + V * Ls * S + read // 2, "flops": 2 * (hf + 200 * V * Ls)}
    if kind == "lanczos":
        return {"bytes": case["steps"] * (2 * hb + 9 * S * V * Ls) + read, "flops": case["steps"] * 2 * (hf + 160 * V * Ls)}
    nbr = V * Ls * 8 * 9  # seam: the neighbour and permute tables
    return {"bytes": hb + nbr + V * 8 * LINK[prec] + 2 * S * V * Ls, "flops": hf}


# ------------------------------------------------------------------ the same in 64 bits, plain torch
_UNIT = {0: (-1j, -1j), 1: (1, -1), 2: (-1j, 1j), 3: (-1, -1)}  # per direction: projector coefficients


def _dhop64(U, psi, dims, dag):
    shape = (dims[3], dims[2], dims[1], dims[0])
    out = torch.zeros_like(psi)
    for leg in range(8):
        d, forward = leg & 3, leg < 4
        nb = psi.reshape(shape + psi.shape[1:]).roll(-1 if forward else 1, dims=3 - d).reshape(psi.shape)
        sign = 1 if forward != bool(dag) else -1
        c0, c1 = (sign * c for c in _UNIT[d])
        a, b = (3, 2) if d < 2 else (2, 3)
        h = torch.stack((nb[:, :, 0] + c0 * nb[:, :, a], nb[:, :, 1] + c1 * nb[:, :, b]), dim=2)
        del nb
        u = torch.zeros_like(h)
        for j in range(3):
            u += U[:, leg, :, j][:, None, None, :] * h[..., j:j + 1]
        out[:, :, 0] += u[:, :, 0]
        out[:, :, 1] += u[:, :, 1]
        out[:, :, a] += complex(c0).conjugate() * u[:, :, 0]
        out[:, :, b] += complex(c1).conjugate() * u[:, :, 1]
    return out


def _fifth64(psi, diag, off, mf, dag):
    """diag psi(s) + off [P- psi(s+1) + P+ psi(s-1)] with walls -mf off; the adjoint for dag."""
    up, down = psi.roll(-1, dims=1), psi.roll(1, dims=1)
    up[:, -1] *= -mf
    down[:, 0] *= -mf
    out = diag * psi
    lo, hi = (slice(2, 4), slice(0, 2)) if dag else (slice(0, 2), slice(2, 4))
    out[:, :, lo] += off * down[:, :, lo]
    out[:, :, hi] += off * up[:, :, hi]
    return out


def _m64(U, psi, dims, dag):
    return _fifth64(psi, 5 - M5, -1.0, MF, dag) - 0.5 * _dhop64(U, psi, dims, dag)


def _mobius64(U, psi, dims, dag):
    b, c = MOBIUS_B, MOBIUS_C
    diag = _fifth64(psi, 1 + b * (4 - M5), -(1 - c * (4 - M5)), MF, dag)
    if dag:
        return diag - 0.5 * _fifth64(_dhop64(U, psi, dims, 1), b, c, MF, 1)
    return diag - 0.5 * _dhop64(U, _fifth64(psi, b, c, MF, 0), dims, 0)


def _fifth_inv64(psi, dag):
    Ls = psi.shape[1]
    eye = torch.eye(Ls, dtype=torch.complex128, device=psi.device).reshape(Ls, Ls, 1, 1).expand(Ls, Ls, 4, 3)
    cols = _fifth64(eye.clone(), 5 - M5, -1.0, MF, dag)  # [column, row, spin, colour]
    out = torch.empty_like(psi)
    for spin in range(4):
        inv = torch.linalg.inv(cols[:, :, spin, 0].T)
        out[:, :, spin] = torch.einsum("st,vtc->vsc", inv, psi[:, :, spin])
    return out


def _schur64(U, psi, dims, dag):
    """Mpc on the odd half: the full operator on fields that are zero on the other parity."""
    n = torch.arange(_vol(dims), device=psi.device)
    x, y = n % dims[0], n // dims[0] % dims[1]
    z, t = n // (dims[0] * dims[1]) % dims[2], n // (dims[0] * dims[1] * dims[2])
    odd = (x + y + z + t) % 2 == 1
    full = torch.zeros((_vol(dims),) + psi.shape[1:], dtype=psi.dtype, device=psi.device)
    full[odd] = psi
    even = _dhop64(U, full, dims, dag)
    even[~odd] = _fifth_inv64(even[~odd], dag)
    even[odd] = 0
    return _fifth64(psi, 5 - M5, -1.0, MF, dag) - 0.25 * _dhop64(U, even, dims, dag)[odd]


def _norm2(v):
    return float(torch.linalg.vector_norm(v)) ** 2


def _cg64(A, b):
    x, r = torch.zeros_like(b), b.clone()
    p, rr, stop = r.clone(), _norm2(r), 1e-26 * _norm2(b)
    for _ in range(5000):
        if rr <= stop:
            break
        q = A(p)
        a = rr / float(torch.sum(p.conj() * q).real)
        x += a * p
        r -= a * q
        new = _norm2(r)
        p = r + (new / rr) * p
        rr = new
    return x


def _flat(psi):
    return torch.view_as_real(psi.contiguous()).reshape(-1)


def exact(case, seed):
    kind, dims = case["kind"], _dims(case)
    if kind == "batch":
        out = []
        for d, ls, sd in _instances(case, seed):
            gen = _generator(sd)
            U, phi = _links(d, gen, torch.complex64), _spinor(d, ls, gen, torch.complex64)
            out.append(_flat(_dhop64(U.to(torch.complex128), phi.to(torch.complex128), d, 0)))
        return out
    U, phi = _inputs(case, seed)
    U = U.to(torch.complex128)
    if kind == "hop":
        out = torch.empty(len(phi), phi[0].numel() * 2, device="cuda", dtype=torch.float64)
        for r, v in enumerate(phi):
            v = v.to(torch.complex128)
            for k in range(case["steps"]):
                v = _dhop64(U, v, dims, k & 1)
            out[r] = _flat(v)
        return out
    psi = phi[0].to(torch.complex128)
    if kind == "seam":
        return _flat(_dhop64(U, psi, dims, 0)).cpu().numpy()
    if kind == "lanczos":
        v, prev = psi / _norm2(psi) ** 0.5, None
        alpha, beta = [], []
        for k in range(case["steps"]):
            w = _m64(U, _m64(U, v, dims, 0), dims, 1)
            alpha.append(float(torch.sum(v.conj() * w).real))
            w = w - alpha[-1] * v
            if k:
                w = w - beta[-1] * prev
            beta.append(_norm2(w) ** 0.5)
            prev, v = v, w / beta[-1]
        return {"alpha": alpha, "beta": beta, "v": _flat(v)[None], "orthogonal": True}
    if kind == "cg":
        # every inner precision converges to the same solution
        if case["system"] == "eo":
            psi = _m64(U, psi, dims, 1)
        return _flat(_cg64(lambda v: _m64(U, _m64(U, v, dims, 0), dims, 1), psi))[None]
    op = {"mdagm": _m64, "mobius": _mobius64, "schur": _schur64}[kind]
    t = op(U, psi, dims, 0)
    return {"psi": _flat(op(U, t, dims, 1))[None], "pap": _norm2(t)}
