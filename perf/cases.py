"""The work that is timed: mat-vecs, rigorous solves, ragged batches and microscope images through the public entry
points of the ifdda package, over the lattices that its tests and its benchmark use, small, odd and large.

A case is a dict of plain values. `kind` says which entry point it calls:

  matvec      GreenSpectrum.matvec_device: nrhs vectors, FFB <- FFB - conv(FFX) in place, complex128 or complex64
  solve       GreenSpectrum.recompute (where `spectrum` is set: a new object, as one cdmlib call) and the rigorous solve
              of nrhs plane waves, on device arrays (inverserig_device) or host arrays (inverserig)
  ragged      Context.inverserig_ragged_device: uneven objects of one common box in one batch
  microscope  GreenSpectrum.microscope: every illumination solved, then the bright-field image

Lattices: `full` boxes (produitfftmatvectopt / inverserigopt) or inside-only ellipsoids with a Tabdip
(produitfftmatvect3 / inverserig). Sides that are no compiled FFT length run padded.

Mixed solves are asked for 1e-11, the accuracy of a converged FP64 solve: at looser tolerances two correct
FP32 inner solves leave fields that differ by as much as the tolerance.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if os.path.join(ROOT, "if-dda_b200") not in sys.path:
    sys.path.insert(0, os.path.join(ROOT, "if-dda_b200"))

import ifdda  # noqa: E402

LAMBDA = 632.8e-9
K0 = 2 * math.pi / LAMBDA
PRECISION = {"f64": ifdda.IFDDA_FP64, "f32": ifdda.IFDDA_FP32, "mixed": ifdda.IFDDA_MIXED}
_ctx = []


def _context():
    """One context for the process, as a program keeps it."""
    if not _ctx:
        _ctx.append(ifdda.Context(0))
    return _ctx[0]


# ------------------------------------------------------------------- cases --
def _matvec(name, nx, ny, nz, prec, nrhs, full):
    return {"name": name, "kind": "matvec", "nx": nx, "ny": ny, "nz": nz, "prec": prec, "nrhs": nrhs, "full": full}


def _solve(name, nx, ny, nz, prec, nrhs, full, host, spectrum, method="GPBICG1"):
    return {"name": name, "kind": "solve", "nx": nx, "ny": ny, "nz": nz, "prec": prec, "nrhs": nrhs, "full": full,
            "host": host, "spectrum": spectrum, "method": method, "tol": 1e-11 if prec == "mixed" else 1e-4}


def listed():
    return [
        # the product inside a caller's own Krylov loop on a small sphere: launches and latency count
        _matvec("matvec f64 sphere 16^3", 16, 16, 16, "f64", 1, False),
        # the same on the benchmark's cube, in both precisions
        _matvec("matvec f32 cube 64^3", 64, 64, 64, "f32", 1, True),
        _matvec("matvec f64 cube 64^3", 64, 64, 64, "f64", 1, True),
        # a microscope sweep's product: several incidences on one object
        _matvec("matvec f32 96x96x64 x8", 96, 96, 64, "f32", 8, True),
        # the largest object of the benchmark
        _matvec("matvec f32 cube 192^3", 192, 192, 192, "f32", 1, True),
        # a user's own discretisation: odd sides, padded, an inside-only object, two polarisations
        _matvec("matvec f64 75x45x29 x2", 75, 45, 29, "f64", 2, False),
        # a whole cdmlib call on a small sphere from host arrays
        _solve("solve f64 sphere 16^3 host", 16, 16, 16, "f64", 1, False, True, True),
        # a whole cdmlib call on the benchmark's cube, arrays resident: spectrum and solve
        _solve("solve f64 cube 64^3", 64, 64, 64, "f64", 1, True, False, True),
        _solve("solve mixed cube 64^3", 64, 64, 64, "mixed", 1, True, False, True),
        # an incidence sweep on a spectrum that stays
        _solve("sweep f64 48x40x32 x12", 48, 40, 32, "f64", 12, False, False, False),
        # a server's batch: four uneven objects, three incidences each, on one 32^3 box
        {"name": "ragged f64 32^3 4 objects", "kind": "ragged", "box": 32, "objects": 4, "nrhs": 3, "prec": "f64",
         "method": "GPBICG1", "tol": 1e-4},
        # a bright-field image: illuminations solved in batches, lens, image
        {"name": "microscope f64 24^3", "kind": "microscope", "nx": 24, "ny": 24, "nz": 24, "prec": "f64",
         "nfft2d": 128, "method": "GPBICG1", "tol": 1e-4},
    ]


def _side(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["matvec"] * 4 + ["solve"] * 3 + ["ragged"] + ["microscope"])
    if kind == "matvec":
        nx, ny, nz = (_side(rng, 6, 192) for _ in range(3))
        nrhs = rng.choice([1, 1, 1, 2, 3, 5, 8, 12])
        while nx * ny * nz * nrhs > 192 ** 3 // 2:
            nrhs = max(1, nrhs // 2)
            nx, ny, nz = max(6, nx * 7 // 8), max(6, ny * 7 // 8), max(6, nz * 7 // 8)
        c = _matvec("", nx, ny, nz, rng.choice(["f64", "f32"]), nrhs, rng.random() < 0.6)
    elif kind == "solve":
        nx, ny, nz = (_side(rng, 8, 80) for _ in range(3))
        nrhs = rng.choice([1, 1, 1, 2, 4, 9])
        while nx * ny * nz * nrhs > 64 ** 3:
            nrhs = max(1, nrhs // 2)
            nx, ny, nz = max(8, nx * 7 // 8), max(8, ny * 7 // 8), max(8, nz * 7 // 8)
        prec = rng.choice(["f64", "mixed"])
        method = rng.choice(["GPBICG1"] * 4 + ["GPBICG2", "BICGSTAB"]) if prec == "f64" else "GPBICG1"
        c = _solve("", nx, ny, nz, prec, nrhs, rng.random() < 0.6, rng.random() < 0.3, rng.random() < 0.5, method)
    elif kind == "ragged":
        c = {"kind": "ragged", "box": rng.choice([16, 24, 32, 40, 48]), "objects": rng.randint(2, 6),
             "nrhs": rng.randint(1, 4), "prec": rng.choice(["f64", "mixed"]), "method": "GPBICG1"}
        c["tol"] = 1e-11 if c["prec"] == "mixed" else 1e-4
    else:
        n = rng.choice([10, 12, 16, 20, 24])
        c = {"kind": "microscope", "nx": n, "ny": n, "nz": rng.choice([n, n // 2, n - 1]), "prec": "f64",
             "nfft2d": 128, "method": "GPBICG1", "tol": 1e-4}
    c.pop("name", None)
    return c


# ------------------------------------------------------------------ inputs --
def _lattice(nx, ny, nz, d):
    """Site positions (x fastest), centred."""
    ax = [(torch.arange(n, device="cuda", dtype=torch.float64) + 0.5 - n / 2) * d for n in (nx, ny, nz)]
    z, y, x = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    return x.reshape(-1), y.reshape(-1), z.reshape(-1)


def _permittivity(nx, ny, nz, gen):
    """A smooth random field: mean 2.25, standard deviation 0.1, correlation length of five sites."""
    w = torch.randn((nz, ny, nx), generator=gen, device="cuda", dtype=torch.float64)
    k = [torch.fft.fftfreq(n, device="cuda", dtype=torch.float64) * 2 * math.pi for n in (nz, ny, nx)]
    k2 = k[0][:, None, None] ** 2 + k[1][None, :, None] ** 2 + k[2][None, None, :] ** 2
    f = torch.fft.ifftn(torch.fft.fftn(w) * torch.exp(-k2 * 25 / 8)).real
    f = (f - f.mean()) / f.std().clamp_min(1e-30)
    return 2.25 + 0.1 * f.reshape(-1)


def _object(nx, ny, nz, d, full, gen):
    """Positions, polarisability per dipole (Clausius-Mossotti with radiative reaction) and Tabdip (None: full box)."""
    x, y, z = _lattice(nx, ny, nz, d)
    eps = _permittivity(nx, ny, nz, gen)
    tab = keep = None
    if not full:
        keep = (x / nx) ** 2 + (y / ny) ** 2 + (z / nz) ** 2 < (d / 2) ** 2
        tab = torch.where(keep, torch.cumsum(keep, 0), 0).to(torch.int32)
        x, y, z, eps = x[keep], y[keep], z[keep], eps[keep]
    pola = (eps - 1) / (eps + 2) * (d ** 3 * 0.75 / math.pi)
    alpha = pola / (1 - 2 / 3 * 1j * K0 ** 3 * pola)
    return x.contiguous(), y.contiguous(), z.contiguous(), alpha, tab


def _polarisa(alpha, nmax):
    """The reference's (nmax,3,3) column-major tensor."""
    p = torch.zeros((3, 3, nmax), dtype=torch.complex128, device="cuda")
    for a in range(3):
        p[a, a, : alpha.numel()] = alpha
    return p.reshape(-1)


def _incident(x, y, z, nrhs, gen):
    """Plane waves of incidences on the NA 0.9 cone, s and p in turn: (nrhs, 3 dipoles)."""
    out = torch.empty((nrhs, x.numel(), 3), dtype=torch.complex128, device="cuda")
    u = torch.rand((nrhs, 2), generator=gen, device="cuda", dtype=torch.float64).cpu()
    for r in range(nrhs):
        th, ph = math.asin(0.9 * math.sqrt(float(u[r, 0]))), 2 * math.pi * float(u[r, 1])
        k = (math.sin(th) * math.cos(ph), math.sin(th) * math.sin(ph), math.cos(th))
        e = (math.cos(th) * math.cos(ph), math.cos(th) * math.sin(ph), -math.sin(th)) if r % 2 == 0 else \
            (-math.sin(ph), math.cos(ph), 0.0)
        wave = torch.exp(1j * K0 * (k[0] * x + k[1] * y + k[2] * z))
        for a in range(3):
            out[r, :, a] = 1e3 * e[a] * wave
    return out.reshape(nrhs, -1).contiguous()


def _spacing(case):
    """10 nm, the benchmark's; small lattices take the 12.5 nm and 25 nm of its small sphere and microscope."""
    if case["kind"] == "microscope":
        return 25e-9
    n = max(case.get(s, 0) for s in ("nx", "ny", "nz", "box"))
    return 12.5e-9 if n <= 24 else 10e-9


def _inputs(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    d = _spacing(case)
    if case["kind"] == "ragged":
        box, objs = case["box"], []
        for i in range(case["objects"]):
            # sides from three quarters of the box to the box, one of them the box's own
            sides = [max(4, box - (i * (a + 2)) % (box // 4 + 1)) for a in range(3)]
            objs.append((sides, _object(*sides, d, i % 2 == 0, gen)))
        return d, [(s, o, _incident(o[0], o[1], o[2], case["nrhs"], gen)) for s, o in objs]
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    obj = _object(nx, ny, nz, d, case.get("full", True), gen)
    nd = obj[0].numel()
    if case["kind"] == "matvec":
        t = torch.complex64 if case["prec"] == "f32" else torch.complex128
        x, b = (torch.randn((case["nrhs"], 3 * nd), generator=gen, device="cuda", dtype=torch.complex128)
                for _ in range(2))
        # moments of the size that a field of order one induces
        alpha = obj[3].repeat_interleave(3)
        return d, obj, (x * alpha).to(t), b.to(t)
    if case["kind"] == "solve":
        return d, obj, _incident(obj[0], obj[1], obj[2], case["nrhs"], gen)
    return d, obj


# ----------------------------------------------------------------- prepare --
def prepare(case, seed):
    ctx = _context()
    inp = _inputs(case, seed)
    d, s = inp[0], {"kind": case["kind"], "d": inp[0], "prec": PRECISION[case["prec"]]}
    if case["kind"] == "ragged":
        s["objects"] = []
        items = []
        for sides, (x, y, z, alpha, tab), ff0 in inp[1]:
            g = ctx.green_box(*sides, (case["box"],) * 3, d, K0)
            nmax = sides[0] * sides[1] * sides[2]
            pol = _polarisa(alpha, nmax)
            ff, loc = torch.empty_like(ff0), torch.empty_like(ff0)
            s["objects"].append((pol, tab, ff0, ff, loc))
            items.append((g, x.numel(), nmax, None if tab is None else tab.data_ptr(), pol.data_ptr(), ff0.data_ptr(),
                          ff.data_ptr(), loc.data_ptr(), case["nrhs"]))
        s.update(items=items, method=case["method"], tol=case["tol"])
    else:
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        x, y, z, alpha, tab = inp[1]
        s.update(green=ctx.green(nx, ny, nz, d, K0), nd=x.numel(), nmax=nx * ny * nz, tab=tab)
        if case["kind"] == "matvec":
            s.update(x=inp[2], b=inp[3], nrhs=case["nrhs"])
        else:
            s.update(method=case["method"], tol=case["tol"], pol=_polarisa(alpha, nx * ny * nz))
        if case["kind"] == "solve":
            ff0 = inp[2]
            s.update(nrhs=case["nrhs"], spectrum=case["spectrum"], host=case["host"])
            if case["host"]:
                s.update(pol=s["pol"].cpu().numpy(), ff0=ff0.cpu().numpy(), tab=None if tab is None else tab.cpu().numpy())
                s.update(out=(np.empty_like(s["ff0"]), np.empty_like(s["ff0"])))
            else:
                s.update(ff0=ff0, ff=torch.empty_like(ff0), loc=torch.empty_like(ff0))
        if case["kind"] == "microscope":
            s.update(xs=x.cpu().numpy(), ys=y.cpu().numpy(), zs=z.cpu().numpy(), pol=s["pol"].cpu().numpy(),
                     nfft2d=case["nfft2d"])
    torch.cuda.synchronize()  # the context works on a stream of its own
    return s


# --------------------------------------------------------------------- run --
def run(s):
    if s["kind"] == "matvec":
        s["green"].matvec_device(s["nrhs"], s["nd"], s["x"].data_ptr(), s["b"].data_ptr(),
                                 None if s["tab"] is None else s["tab"].data_ptr(), s["prec"])
        return s["b"]
    if s["kind"] == "solve":
        g = s["green"]
        if s["spectrum"]:
            g.recompute(s["d"], K0)
        if s["host"]:
            r = g.inverserig(s["nd"], s["pol"], s["nmax"], s["ff0"], s["method"], s["tol"], tabdip=s["tab"],
                             precision=s["prec"], out=s["out"])
            return {"FF": r.FF, "FFloc": r.FFloc}
        g.inverserig_device(s["nrhs"], s["nd"], s["nmax"], None if s["tab"] is None else s["tab"].data_ptr(),
                            s["pol"].data_ptr(), s["ff0"].data_ptr(), s["ff"].data_ptr(), s["loc"].data_ptr(),
                            s["method"], s["tol"], precision=s["prec"])
        return {"FF": s["ff"], "FFloc": s["loc"]}
    if s["kind"] == "ragged":
        _context().inverserig_ragged_device(s["items"], s["method"], s["tol"], s["prec"])
        return [{"FF": o[3], "FFloc": o[4]} for o in s["objects"]]
    r = s["green"].microscope(s["xs"], s["ys"], s["zs"], s["pol"], s["method"], s["tol"], nfft2d=s["nfft2d"],
                              precision=s["prec"])
    return r.image


# -------------------------------------------------------------------- work --
def _matvec_work(nx, ny, nz, nrhs, size):
    """The product x -> b - G x: x and b read, b written, the six components of the spectrum's octant read; the
    transforms of the three components along each axis over the lines that are not zero, there and back."""
    n, m = nx * ny * nz, (nx + 1) * (ny + 1) * (nz + 1)
    lines = [(2 * nx, ny * nz), (2 * ny, 2 * nx * nz), (2 * nz, 4 * nx * ny)]
    fft = sum(2 * 3 * cnt * 5 * ln * math.log2(ln) for ln, cnt in lines)
    return {"bytes": size * (9 * n * nrhs + 6 * m), "flops": nrhs * (fft + 8 * n * 66)}


def work(case):
    size = 8 if case["prec"] == "f32" else 16
    if case["kind"] == "matvec":
        return _matvec_work(case["nx"], case["ny"], case["nz"], case["nrhs"], size)
    # a solve of these objects takes 12 iterations of two products each (mixed, to 1e-11: 40, in 32 bits)
    its, size = (40, 8) if case["prec"] == "mixed" else (12, 16)
    if case["kind"] == "ragged":
        nx = ny = nz = case["box"]
        nrhs = case["objects"] * case["nrhs"]
    else:
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        nrhs = 42 if case["kind"] == "microscope" else case["nrhs"]
    w = _matvec_work(nx, ny, nz, nrhs, size)
    return {k: 2 * its * v for k, v in w.items()}


# ------------------------------------------------------------------- exact --
def _spectrum64(nx, ny, nz, d):
    """The six FFTs of the free-space dyadic on the circulant grid, complex128."""
    ax = []
    for n in (nx, ny, nz):
        i = torch.arange(2 * n, device="cuda", dtype=torch.float64)
        ax.append((torch.where(i > n, i - 2 * n, i) * d, i != n))
    Z, Y, X = torch.meshgrid(ax[2][0], ax[1][0], ax[0][0], indexing="ij")
    on = ax[2][1][:, None, None] & ax[1][1][None, :, None] & ax[0][1][None, None, :]
    r2 = X * X + Y * Y + Z * Z
    on &= r2 > 0
    r2 = torch.where(on, r2, torch.ones_like(r2))
    r = torch.sqrt(r2)
    e = torch.exp(1j * K0 * r)
    near, far = (1 / r - 1j * K0) / r2 * e, K0 * K0 / r * e
    del e, r
    out = []
    pos = (X, Y, Z)
    for a in range(3):
        for b in range(a, 3):
            rr = pos[a] * pos[b] / r2
            one = 1.0 if a == b else 0.0
            g = torch.where(on, (3 * rr - one) * near + (one - rr) * far, torch.zeros_like(near))
            out.append(torch.fft.fftn(g))
    return out


def _apply64(G, x, nx, ny, nz, tab):
    """conv(x) of one vector of 3 complex128 components per dipole."""
    if tab is None:
        full = x.reshape(-1, 3)
    else:
        full = torch.zeros((nx * ny * nz, 3), dtype=x.dtype, device=x.device)
        full[tab > 0] = x.reshape(-1, 3)
    grid = full.reshape(nz, ny, nx, 3)
    f = [torch.fft.fftn(grid[..., a], s=(2 * nz, 2 * ny, 2 * nx)) for a in range(3)]
    ix = ((0, 1, 2), (1, 3, 4), (2, 4, 5))
    out = torch.empty_like(full)
    for a in range(3):
        v = torch.fft.ifftn(G[ix[a][0]] * f[0] + G[ix[a][1]] * f[1] + G[ix[a][2]] * f[2])
        out[:, a] = v[:nz, :ny, :nx].reshape(-1)
    return out.reshape(-1) if tab is None else out[tab > 0].reshape(-1)


def _solve64(G, alpha3, b, nx, ny, nz, tab):
    """(I - G alpha) x = b by BiCGSTAB, to rounding."""
    A = lambda v: v - _apply64(G, alpha3 * v, nx, ny, nz, tab)  # noqa: E731
    x = b.clone()
    best, nb = x, float(torch.linalg.vector_norm(b))
    res = math.inf
    for _ in range(3):  # restarted on the true residual
        r = b - A(x)
        if float(torch.linalg.vector_norm(r)) < res:
            best, res = x, float(torch.linalg.vector_norm(r))
        if res < 1e-14 * nb:
            break
        r0, p, rho = r.clone(), r.clone(), torch.vdot(r, r)
        for _ in range(200):
            v = A(p)
            a = rho / torch.vdot(r0, v)
            s = r - a * v
            t = A(s)
            w = torch.vdot(t, s) / torch.vdot(t, t)
            x = x + a * p + w * s
            r = s - w * t
            if float(torch.linalg.vector_norm(r)) < 1e-14 * nb:
                break
            new = torch.vdot(r0, r)
            p = r + (new / rho) * (a / w) * (p - w * v)
            rho = new
    return x if float(torch.linalg.vector_norm(b - A(x))) < res else best


def exact(case, seed):
    if case["kind"] == "microscope":
        return None
    inp = _inputs(case, seed)
    d = inp[0]
    if case["kind"] == "ragged":
        out = []
        for sides, (x, y, z, alpha, tab), ff0 in inp[1]:
            G, a3 = _spectrum64(*sides, d), alpha.repeat_interleave(3)
            loc = torch.stack([_solve64(G, a3, b, *sides, tab) for b in ff0])
            out.append({"FF": a3 * loc, "FFloc": loc})
        return out
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    alpha, tab = inp[1][3], inp[1][4]
    G = _spectrum64(nx, ny, nz, d)
    if case["kind"] == "matvec":
        return torch.stack([b.to(torch.complex128) - _apply64(G, x.to(torch.complex128), nx, ny, nz, tab)
                            for x, b in zip(inp[2], inp[3])])
    a3 = alpha.repeat_interleave(3)
    loc = torch.stack([_solve64(G, a3, b, nx, ny, nz, tab) for b in inp[2]])
    return {"FF": a3 * loc, "FFloc": loc}
