"""The workloads this library is timed on, and what each one has to return.

A case is a dict of plain values: ``kind`` names the work, the rest are its
sizes and options.  ``prepare`` builds the gauge field(s) a user's program
already holds (links exp(i eps H), H = sum_a c_a lambda_a / 2 with c_a ~ N(0,1),
rows orthonormalised; eps = 0 stands for Haar-random links), ``run`` makes one
pass through the public entry points, ``work`` counts the bytes and operations
such a pass cannot do without, and ``exact`` gives the same results from plain
64-bit torch arithmetic.

Lattices are written (NT, NX, NY, NZ); ``prec`` is the field format: "c128"
(FP64 arithmetic), "c64" (FP32, 18 reals a link) or "r12" (FP32, two stored
rows).
"""
from __future__ import annotations

import itertools
import math

import numpy as np
import torch

from FLUE.compiled import flue_c
from flue_gb300 import flow, forces, gluonCalc
from flue_gb300.ensemble import Ensemble
from flue_gb300.field import GaugeField

FLOW_EPS = 0.01
FLOP_PER_PRODUCT = 198  # 3x3 complex product: 27 multiplications (6) and 18 additions (2)


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _case(kind, prec, dims, eps=0.3, **more):
    c = {"kind": kind, "prec": prec, "nt": dims[0], "nx": dims[1], "ny": dims[2], "nz": dims[3], "eps": eps}
    c.update(more)
    return c


def listed():
    return [
        # B^2 and its gradient, the production form: reconstruct-12 links at
        # the lattice the library's benchmark is quoted on
        dict(_case("b2_force", "r12", (64, 32, 32, 32), form="lie"), name="b2_force r12 32^3x64"),
        # the same at the reference's own precision
        dict(_case("b2_force", "c128", (64, 32, 32, 32), form="lie"), name="b2_force c128 32^3x64"),
        # a small odd lattice with full complex64 links, gradient in the
        # convention of torch.autograd: a training loop over small lattices
        dict(_case("b2_force", "c64", (19, 11, 13, 9), form="euclid"), name="b2_force c64 9x13x11x19"),
        # `magnetic` of the plain-method lattice: the smallest measurement
        dict(_case("b2", "c128", (16, 8, 8, 8)), name="b2 c128 8^3x16"),
        # plaquettes of every range and the Polyakov loop, hot links, FP64
        dict(_case("loops", "c128", (64, 32, 32, 32), eps=0.0), name="loops c128 32^3x64"),
        # the same on the largest lattice of the precision report, FP32
        dict(_case("loops", "c64", (96, 48, 48, 48)), name="loops c64 48^3x96"),
        # static-potential table W(R,T), R,T = 1..8 in a space-time plane
        dict(_case("wtable", "c128", (64, 32, 32, 32), eps=0.5, mu=2, nu=1, rmax=8, tmax=8),
             name="wtable c128 32^3x64"),
        # field strength of one electric plane (clover and 5-loop), FP32
        dict(_case("fmunu", "c64", (48, 24, 24, 24), eps=0.1, mu=4, nu=1), name="fmunu c64 24^3x48"),
        # a stretch of Wilson flow with its measurements, both precisions
        dict(_case("flow", "c64", (64, 32, 32, 32), steps=5), name="flow c64 32^3x64"),
        dict(_case("flow", "c128", (48, 24, 24, 24), steps=5), name="flow c128 24^3x48"),
        # an ensemble of uneven volume, all observables in one launch
        dict({"kind": "ensemble", "prec": "c128", "eps": 0.4, "fields": 6, "lmin": 16, "lmax": 24, "tmin": 32, "tmax": 48},
             name="ensemble c128 6 fields"),
        # a field in the caller's host memory through the f2py-style module:
        # complex128 in, FP32 arithmetic, complex128 gradient out
        dict(_case("host_force", "r12", (48, 24, 24, 24), form="lie"), name="host_force r12 24^3x48"),
    ]


def draw(rng):
    kind = rng.choice(["b2_force", "b2_force", "b2", "loops", "wtable", "fmunu", "flow", "ensemble", "host_force"])
    eps = rng.choice([0.1, 0.3, 0.4, 0.5, 0.0])

    def ext(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def dims(lo, hi, tlo, thi):
        l = ext(lo, hi)
        if rng.random() < 0.5:
            return (ext(tlo, thi), l, l, l)
        return (ext(tlo, thi), l, ext(max(lo, l // 2), l), ext(max(lo, l // 2), l))

    if kind == "b2_force":
        return _case(kind, rng.choice(["r12", "c64", "c128"]), dims(5, 32, 5, 64), eps, form=rng.choice(["lie", "euclid"]))
    if kind == "b2":
        return _case(kind, rng.choice(["r12", "c64", "c128"]), dims(5, 32, 5, 64), eps)
    if kind == "loops":
        return _case(kind, rng.choice(["r12", "c64", "c128"]), dims(6, 40, 6, 80), eps)
    if kind == "wtable":
        mu, nu = rng.choice([(2, 1), (3, 1), (4, 1), (2, 3), (4, 3)])
        return _case(kind, rng.choice(["c64", "c128"]), dims(6, 30, 6, 60), eps, mu=mu, nu=nu, rmax=rng.randint(2, 8),
                     tmax=rng.randint(2, 8))
    if kind == "fmunu":
        mu, nu = rng.choice([(4, 1), (2, 1), (3, 2), (2, 4), (1, 3)])
        return _case(kind, rng.choice(["r12", "c64", "c128"]), dims(5, 28, 5, 56), eps, mu=mu, nu=nu)
    if kind == "flow":
        return _case(kind, rng.choice(["c64", "c128"]), dims(5, 26, 5, 52), rng.choice([0.1, 0.3, 0.4]),
                     steps=rng.randint(1, 5))
    if kind == "ensemble":
        lmin = ext(6, 16)
        tmin = ext(6, 32)
        return {"kind": kind, "prec": rng.choice(["r12", "c64", "c128"]), "eps": rng.choice([0.3, 0.4]),
                "fields": rng.randint(2, 6), "lmin": lmin, "lmax": lmin + rng.randint(2, 8), "tmin": tmin,
                "tmax": tmin + rng.randint(2, 16)}
    return _case(kind, rng.choice(["r12", "c128"]), dims(5, 24, 5, 48), eps, form="lie")


def _dims(case):
    return (case["nt"], case["nx"], case["ny"], case["nz"])


def _ensemble_dims(case):
    """The lattices of an ensemble case: extents spread evenly over its ranges."""
    n = case["fields"]
    out = []
    for i in range(n):
        l = case["lmin"] + (case["lmax"] - case["lmin"]) * i // max(1, n - 1)
        t = case["tmin"] + (case["tmax"] - case["tmin"]) * ((2 * i) % n) // max(1, n - 1)
        out.append((t, l, l, l))
    return out


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
# Working layout of this file: W[a, b, mu, z, y, x, t] (colour indices first,
# sites contiguous), products as broadcasts over (a, k, b).
def _mm(p, q):
    """Matrix product of two (3, 3, ...) arrays."""
    out = p[:, 0, None] * q[None, 0]
    out = out + p[:, 1, None] * q[None, 1]
    return out + p[:, 2, None] * q[None, 2]


def _dag(p):
    return p.transpose(0, 1).conj()


def _orthonormal(w):
    """Rows 0 and 1 orthonormalised, row 2 = conj(row0 x row1)."""
    r0 = w[0] / torch.sqrt((w[0].real ** 2 + w[0].imag ** 2).sum(0))
    d = (r0.conj() * w[1]).sum(0)
    r1 = w[1] - r0 * d
    r1 = r1 / torch.sqrt((r1.real ** 2 + r1.imag ** 2).sum(0))
    return torch.stack([r0, r1, _row2(r0, r1)])


def _row2(r0, r1):
    return torch.stack([r0[1] * r1[2] - r0[2] * r1[1], r0[2] * r1[0] - r0[0] * r1[2],
                        r0[0] * r1[1] - r0[1] * r1[0]]).conj()


def _expi(c, eps):
    """exp(i eps H) from the 8 Gell-Mann coefficients c[a, ...]."""
    s3 = 1.0 / math.sqrt(3.0)
    h = torch.stack([
        torch.stack([torch.complex(c[2] + s3 * c[7], torch.zeros_like(c[0])), torch.complex(c[0], -c[1]),
                     torch.complex(c[3], -c[4])]),
        torch.stack([torch.complex(c[0], c[1]), torch.complex(-c[2] + s3 * c[7], torch.zeros_like(c[0])),
                     torch.complex(c[5], -c[6])]),
        torch.stack([torch.complex(c[3], c[4]), torch.complex(c[5], c[6]),
                     torch.complex(-2.0 * s3 * c[7], torch.zeros_like(c[0]))])])
    a = h * (0.5j * eps / 8.0)
    eye = torch.eye(3, dtype=a.dtype, device=a.device).reshape((3, 3) + (1,) * (a.dim() - 2))
    e = eye + a / 12.0
    for k in range(11, 0, -1):
        e = eye + _mm(a, e) / k
    for _ in range(3):
        e = _mm(e, e)
    return e


def _links(dims, eps, seed):
    """W[a, b, mu, z, y, x, t] of a random field, complex128 on the GPU."""
    nt, nx, ny, nz = dims
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    w = torch.empty((3, 3, 4, nz, ny, nx, nt), dtype=torch.complex128, device="cuda")
    step = max(1, (1 << 21) // (ny * nx * nt))
    for mu, z in itertools.product(range(4), range(0, nz, step)):
        n = min(step, nz - z)
        if eps:
            c = torch.randn((8, n, ny, nx, nt), generator=g, device="cuda", dtype=torch.float64)
            m = _expi(c, eps)
        else:
            m = torch.randn((3, 3, n, ny, nx, nt), generator=g, device="cuda", dtype=torch.complex128)
        w[:, :, mu, z:z + n] = _orthonormal(m)
    return w


def _stored(w, prec):
    """The links as the field format holds them, in 64 bits."""
    if prec == "c128":
        return w
    w = w.to(torch.complex64).to(torch.complex128)
    if prec == "r12":
        w[2] = _row2(w[0], w[1])
    return w


def _tensor(w, dtype):
    """data[t, x, y, z, mu, a, b] in the reference's memory order."""
    return w.transpose(0, 1).to(dtype).contiguous().permute(6, 5, 4, 3, 2, 1, 0)


def _field(w, prec):
    return GaugeField.from_array(_tensor(w, torch.complex128 if prec == "c128" else torch.complex64), prec=prec)


def prepare(case, seed):
    kind, prec = case["kind"], case["prec"]
    if kind == "ensemble":
        fields = [_field(_links(d, case["eps"], seed * 64 + i), prec) for i, d in enumerate(_ensemble_dims(case))]
        return {"case": case, "ensemble": Ensemble(fields)}
    w = _links(_dims(case), case["eps"], seed)
    if kind == "host_force":
        return {"case": case, "data": np.asfortranarray(_tensor(w, torch.complex128).cpu().numpy())}
    return {"case": case, "field": _field(w, prec)}


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    c = state["case"]
    kind = c["kind"]
    f = state.get("field")
    if kind == "b2_force":
        b2, grad = forces.magnetic_force(f, form=c["form"])
        return {"b2": b2, "grad": grad}
    if kind == "b2":
        return {"b2": gluonCalc.magnetic(f)}
    if kind == "loops":
        out = {}
        for name, rng in (("total", (1, 4, 4)), ("spatial", (2, 4, 4)), ("temporal", (1, 1, 4))):
            out[name] = gluonCalc.plaquette(f, *rng)[0]
        re, _, _, im = gluonCalc.polyakov(f, return_imag=True)
        out["polyakov_re"], out["polyakov_im"] = re, im
        return out
    if kind == "wtable":
        return {"w": gluonCalc.wmunu_table(f, c["mu"], c["nu"], c["rmax"], c["tmax"])}
    if kind == "fmunu":
        return {"clover": gluonCalc.cloverloopmunucoord(f, c["mu"], c["nu"]),
                "loop5": gluonCalc.loop5munucoord(f, c["mu"], c["nu"])}
    if kind == "flow":
        t = c["steps"] * FLOW_EPS
        g, recs = flow.wilson_flow(f, eps=FLOW_EPS, tmax=t, measure_every=t)
        return {"links": g.to_tensor(), "b2": [r["b2"] for r in recs], "plaq": [r["plaq"] for r in recs]}
    if kind == "ensemble":
        return {"obs": state["ensemble"].run()}
    b2, grad = flue_c.magnetic_force(state["data"], prec=c["prec"], form=c["form"])
    return {"b2": b2, "grad": grad}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
LINK_BYTES = {"c128": 144, "c64": 72, "r12": 48}
GRAD_BYTES = {"c128": 576, "c64": 288, "r12": 288}
# products per site: B^2 = 6 for the lines and 3 x 68 for the leaves; its
# gradient = 506 for the line cotangents and 21 for the links'
B2_PRODUCTS = 210
GRAD_PRODUCTS = 527


def work(case):
    kind, prec = case["kind"], case["prec"]
    if kind == "ensemble":
        v = sum(math.prod(d) for d in _ensemble_dims(case))
        p = B2_PRODUCTS + 12 + 1
        return {"bytes": v * 4 * LINK_BYTES[prec], "flops": v * p * FLOP_PER_PRODUCT}
    v = math.prod(_dims(case))
    link = LINK_BYTES[prec]
    if kind == "b2":
        b, p = 3 * link, B2_PRODUCTS
    elif kind == "b2_force":
        b, p = 3 * link + GRAD_BYTES[prec], B2_PRODUCTS + GRAD_PRODUCTS
    elif kind == "host_force":
        b, p = 3 * 96 + 576, B2_PRODUCTS + GRAD_PRODUCTS
    elif kind == "loops":  # four calls: all links three times (once spatial only), then the time links
        b, p = (4 + 3 + 4 + 1) * link, 12 + 6 + 6 + 1
    elif kind == "wtable":
        b, p = 2 * link, case["rmax"] + case["tmax"] - 2 + 2 * case["rmax"] * case["tmax"]
    elif kind == "fmunu":  # two calls, one F each
        out = 144 if prec == "c128" else 72
        b, p = 2 * (2 * link + out), 12 + 4 + 68
    else:  # flow: three stages a step (staples, update), two measurements; links in and out
        b = (case["steps"] * 3 * 2 * 4 + 2 * (3 + 4)) * link
        p = case["steps"] * 3 * (4 * 6 * 2 + 4 * 3) + 2 * (B2_PRODUCTS + 12)
    return {"bytes": int(v * b), "flops": int(v * p * FLOP_PER_PRODUCT)}


# ---------------------------------------------------------------------------
# the same results from 64-bit torch
# ---------------------------------------------------------------------------
# dimension of direction mu = 1..4 (t, x, y, z) in W[a, b, z, y, x, t]
_DIM = {1: -1, 2: -2, 3: -3, 4: -4}
K5 = 1.0 / 180.0
K1 = 19.0 / 9.0 - 55.0 * K5
K2 = 1.0 / 36.0 - 16.0 * K5
K3 = 64.0 * K5 - 32.0 / 45.0
K4 = 1.0 / 15.0 - 6.0 * K5
SHAPES5 = ((1, 1, K1), (2, 2, K2), (3, 3, K5), (1, 2, 0.5 * K3), (2, 1, 0.5 * K3), (1, 3, 0.5 * K4), (3, 1, 0.5 * K4))
SHAPES1 = ((1, 1, 1.0),)
B2_PLANES = ((3, 2), (2, 4), (4, 3))


def _at(m, mu, k):
    """m at x + k mu."""
    return torch.roll(m, -k, _DIM[mu])


def _lines(u, mu, nmax):
    """[L^1, L^2, ...], L^n(x) = U(x) U(x+mu) ... U(x+(n-1) mu)."""
    out = [u]
    for n in range(1, nmax):
        out.append(_mm(out[-1], _at(u, mu, n)))
    return out


def _clover_sum(um, un, mu, nu, shapes):
    """Weighted sum of the counter-clockwise leaves at every site."""
    n = max(max(a, b) for a, b, _ in shapes)
    lm, ln = _lines(um, mu, n), _lines(un, nu, n)
    q = 0
    for a, b, cf in shapes:
        m, v = lm[a - 1], ln[b - 1]
        # the rectangle anchored at x, cut open at each of its corners
        s1, s2, s3, s4 = m, _at(v, mu, a), _dag(_at(m, nu, b)), _dag(v)
        s12, s34 = _mm(s1, s2), _mm(s3, s4)
        s23, s41 = _mm(s2, s3), _mm(s4, s1)
        q = q + cf * (_mm(s12, s34) + _at(_mm(s23, s41), mu, -a) + _at(_at(_mm(s34, s12), mu, -a), nu, -b)
                      + _at(_mm(s41, s23), nu, -b))
    return q


def _fmunu(q):
    return (q - _dag(q)) * 0.125


def _energy(u, planes):
    """sum over sites and planes of -Re Tr F F."""
    e = 0.0
    for mu, nu in planes:
        f = _fmunu(_clover_sum(u[mu], u[nu], mu, nu, SHAPES5))
        e = e + (f.real ** 2 + f.imag ** 2).sum()
    return e


def _project(m):
    a = (m - _dag(m)) * 0.5
    tr = (a[0, 0] + a[1, 1] + a[2, 2]) / 3.0
    a = a.clone()
    for k in range(3):
        a[k, k] = a[k, k] - tr
    return a


def _b2(w, form=None):
    """B^2 and (form given) its gradient [b, a, mu, z, y, x, t], time slices in turn."""
    nt = w.shape[-1]
    v = w[0, 0, 0].numel()
    grad = torch.zeros_like(w) if form else None
    step = max(1, min(nt, (1 << 16) // (v // nt)))
    total = 0.0
    for t in range(0, nt, step):
        u = {mu: w[:, :, mu - 1, ..., t:t + step].contiguous().requires_grad_(bool(form)) for mu in (2, 3, 4)}
        e = _energy(u, B2_PLANES) / v
        total += float(e)
        if form:
            for mu, g in zip(u, torch.autograd.grad(e, list(u.values()))):
                if form == "lie":
                    g = -0.5 * _project(_mm(u[mu].detach(), _dag(g)))
                grad[:, :, mu - 1, ..., t:t + step] = g
    return total, grad


def _view(g):
    """W[a, b, mu, z, y, x, t] as [t, x, y, z, mu, a, b]."""
    return g.permute(6, 5, 4, 3, 2, 0, 1)


def _plaquettes(w, mustart, muend, nuend):
    s = 0.0
    for mu in range(mustart, muend + 1):
        for nu in range(mu + 1, nuend + 1):
            um, un = w[:, :, mu - 1], w[:, :, nu - 1]
            p = (_mm(um, _at(un, mu, 1)) * _mm(un, _at(um, nu, 1)).conj()).real
            s += float(p.sum())
    return s


def _polyakov(w):
    u = w[:, :, 0]
    p = u[..., 0]
    for t in range(1, u.shape[-1]):
        p = _mm(p, u[..., t])
    tr = (p[0, 0] + p[1, 1] + p[2, 2]).sum()
    return float(tr.real), float(tr.imag)


def _staple_velocity(w):
    """2 G, G = -1/2 TA(U N) of the plaquette action."""
    z = torch.empty_like(w)
    for mu in range(1, 5):
        um = w[:, :, mu - 1]
        n = 0
        for nu in range(1, 5):
            if nu == mu:
                continue
            un = w[:, :, nu - 1]
            up = _mm(_mm(_at(un, mu, 1), _dag(_at(um, nu, 1))), _dag(un))
            dn = _at(_mm(_dag(_mm(um, _at(un, mu, 1))), un), nu, -1)
            n = n + up + dn
        z[:, :, mu - 1] = -_project(_mm(um, n))
    return z


def _rotate(x, w):
    """exp(x) w for small anti-Hermitian x."""
    term, out = w, w
    for k in range(1, 17):
        term = _mm(x, term) / k
        out = out + term
    return out


def _flow(w, steps, fp32):
    for _ in range(steps):
        z0 = FLOW_EPS * _staple_velocity(w)
        for stage in range(3):
            if stage == 0:
                x = b = z0
                x = x / 4.0
            elif stage == 1:
                x = (8.0 / 9.0 * FLOW_EPS) * _staple_velocity(w) - (17.0 / 36.0) * b
                b = x
            else:
                x = (0.75 * FLOW_EPS) * _staple_velocity(w) - b
            for mu in range(4):
                m = _rotate(x[:, :, mu], w[:, :, mu])
                w[:, :, mu] = _orthonormal(m) if fp32 else m
    return w


def exact(case, seed):
    kind, prec = case["kind"], case["prec"]
    if kind == "ensemble":
        rows = []
        for i, dims in enumerate(_ensemble_dims(case)):
            w = _stored(_links(dims, case["eps"], seed * 64 + i), prec)
            re, im = _polyakov(w)
            rows.append([_plaquettes(w, 2, 4, 4), _plaquettes(w, 1, 1, 4), re, im, _b2(w)[0], float(math.prod(dims))])
        return {"obs": np.array(rows)}
    w = _stored(_links(_dims(case), case["eps"], seed), prec)
    if kind == "b2":
        return {"b2": _b2(w)[0]}
    if kind in ("b2_force", "host_force"):
        b2, grad = _b2(w, case["form"])
        grad = _view(grad)
        return {"b2": b2, "grad": grad if kind == "b2_force" else grad.cpu().numpy()}
    if kind == "loops":
        re, im = _polyakov(w)
        return {"total": _plaquettes(w, 1, 4, 4), "spatial": _plaquettes(w, 2, 4, 4), "temporal": _plaquettes(w, 1, 1, 4),
                "polyakov_re": re, "polyakov_im": im}
    if kind == "wtable":
        mu, nu = case["mu"], case["nu"]
        lm, ln = _lines(w[:, :, mu - 1], mu, case["rmax"]), _lines(w[:, :, nu - 1], nu, case["tmax"])
        out = np.empty((case["rmax"], case["tmax"]))
        for r, t in itertools.product(range(case["rmax"]), range(case["tmax"])):
            p = (_mm(lm[r], _at(ln[t], mu, r + 1)) * _mm(ln[t], _at(lm[r], nu, t + 1)).conj()).real
            out[r, t] = float(p.sum()) / p[0, 0].numel()
        return {"w": out}
    if kind == "fmunu":
        mu, nu = case["mu"], case["nu"]
        out = {}
        for name, shapes in (("clover", SHAPES1), ("loop5", SHAPES5)):
            f = _fmunu(_clover_sum(w[:, :, mu - 1], w[:, :, nu - 1], mu, nu, shapes))
            out[name] = f.permute(5, 4, 3, 2, 1, 0)  # transposed: genericPath returns U^T
        return out
    b2, plaq = [], []
    for steps in (0, case["steps"]):  # before the flow and after it
        w = _flow(w, steps, prec != "c128")
        b2.append(_b2(w)[0])
        plaq.append(_plaquettes(w, 1, 4, 4) / (6 * math.prod(_dims(case))) / 3.0)
    return {"links": _view(w), "b2": b2, "plaq": plaq}
