"""Performance cases: what a lattice-QCD program has this library do.

A case names a call of the public Python interface (qphix_b200.api), the
operator, its storage precision and links, the lattice and the number of
right-hand sides.  `prepare` makes what such a program holds before the call
(resident fields and the operator, or the solver), `run` is one call,
`exact` the same result in FP64 from plain torch on full-lattice arrays.

Host arrays are in the QDP++ CB2 order (both checkerboards, even first),
sources are Gaussian, links are SU(3) matrices near the identity, as the
configurations of qphix_b200.workloads and the benchmark have them.  The
operators act on the odd checkerboard, t is antiperiodic.
"""
import math

import numpy as np
import torch

from qphix_b200 import api

EPS = 0.3  # links: exp(i EPS H) to second order, H traceless Hermitian Gaussian, made unitary
CSW = 1.0
MU = 0.01  # twisted mass
PHASES = ((math.cos(0.3), math.sin(0.3)), (1.0, 0.0), (math.cos(0.7), -math.sin(0.7)), (1.0, 0.0))


def _case(call, kind, prec, dims, nrhs=1, recon=12, dagger=False, twisted=False, kappa=0.125, inner="", rsd=0.0,
          shifts=0, name=None):
    c = dict(call=call, kind=kind, prec=prec, nx=dims[0], ny=dims[1], nz=dims[2], nt=dims[3], nrhs=nrhs,
             recon=recon, dagger=dagger, twisted=twisted, kappa=kappa, inner=inner, rsd=rsd, shifts=shifts)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: the operator on a lattice of a few sites per processor (coarse grids, tests, tuning runs)
        _case("operator", "wilson", "f64", (8, 8, 8, 8), recon=18, name="op_wilson_f64_8x8x8x8"),
        # the smallest solve, where launches and their order count for more than bytes
        _case("cg", "wilson", "f64", (8, 8, 8, 8), recon=18, kappa=0.12, rsd=1e-10, name="cg_wilson_f64_8x8x8x8"),
        # one hop in FP64 on a production lattice, the step every outer residual and plain solve is made of
        _case("dslash", "wilson", "f64", (32, 32, 32, 64), name="dslash_wilson_f64_32x32x32x64"),
        # the daggered operator in FP32, the other half of a normal-equation iteration
        _case("operator", "clover", "f32", (24, 24, 24, 48), dagger=True, kappa=0.136,
              name="op_clover_f32_dagger_24x24x24x48"),
        # a lattice that is no multiple of anything, three right-hand sides and twisted boundaries (moving frames)
        _case("operator", "clover", "f32", (20, 12, 28, 36), nrhs=3, twisted=True, kappa=0.136,
              name="op_clover_f32_twisted_20x12x28x36_3"),
        # the inner operator of a mixed-precision solve of eight spin-colour sources
        _case("operator", "clover", "f16", (16, 16, 16, 32), nrhs=8, kappa=0.136, name="op_clover_f16_16x16x16x32_8"),
        # the same for a block of point sources with twisted mass, in the other 16-bit format
        _case("operator", "tmclover", "bf16", (24, 24, 24, 48), nrhs=12, kappa=0.1373,
              name="op_tmclover_bf16_24x24x24x48_12"),
        # FP64 residuals of many right-hand sides at once (block solves, the refinement of shifted solutions)
        _case("operator", "wilson", "f64", (24, 24, 24, 48), nrhs=16, name="op_wilson_f64_24x24x24x48_16"),
        # the set-up of a clover solve: both checkerboards' terms and the even one's inverse, once per configuration
        _case("clover_term", "clover", "f64", (24, 24, 24, 48), kappa=0.136, name="clover_term_f64_24x24x24x48"),
        # a propagator's column block: FP64 defect correction over a 16-bit BiCGStab
        _case("richardson", "clover", "f64", (16, 16, 16, 32), nrhs=8, kappa=0.136, inner="f16", rsd=1e-10,
              name="richardson_clover_f16_16x16x16x32_8"),
        # the same with one source and FP32 inside, as a program does that solves one column at a time
        _case("richardson", "clover", "f64", (16, 16, 16, 32), nrhs=1, kappa=0.136, inner="f32", rsd=1e-10,
              name="richardson_clover_f32_16x16x16x32_1"),
        # rational approximations in molecular dynamics: every shifted system of one source
        _case("multishift", "wilson", "f64", (24, 24, 24, 48), rsd=1e-9, shifts=16,
              name="multishift_wilson_f64_24x24x24x48_16"),
    ]


# most of (sites of a checkerboard) x (right-hand sides, or shifts) per call, within the listed cases' cost
_MOST = {"dslash": 1 << 22, "operator": 1 << 22, "clover_term": 330000, "cg": 1 << 17, "richardson": 1 << 18,
         "multishift": 1 << 21}


def draw(rng):
    call = rng.choice(("dslash", "operator", "operator", "clover_term", "cg", "richardson", "multishift"))
    kind = {"clover_term": "clover", "richardson": "clover", "multishift": "wilson"}.get(call)
    if kind is None:
        kind = rng.choice(("wilson", "clover") if call == "cg" else ("wilson", "clover", "tm", "tmclover"))
    prec = rng.choice(("f64", "f32", "f16", "bf16")) if call in ("dslash", "operator") else "f64"
    nrhs = 1
    if call in ("dslash", "operator", "richardson"):
        nrhs = rng.choice((1, 1, 2, 3, 4, 7, 8, 12) if call == "richardson" else (1, 1, 2, 3, 5, 8, 12, 16, 24))
    shifts = rng.choice((1, 4, 7, 12, 16)) if call == "multishift" else 0
    most = _MOST[call] // max(nrhs, shifts)
    least = 8192 if call == "dslash" else 128  # one hop of fewer sites is a launch and nothing else
    volume = math.exp(rng.uniform(math.log(least), math.log(most)))  # sites of a checkerboard, aimed at
    while True:
        side = (2 * volume) ** 0.25
        dims = [max(4, 2 * round(side * math.exp(rng.uniform(-0.4, 0.4)) / 2)) for _ in range(4)]
        if math.prod(dims) // 2 <= most:
            break
    plain = call in ("dslash", "operator")
    kappa = round(rng.uniform(0.11, 0.125) if kind in ("wilson", "tm") else rng.uniform(0.12, 0.136), 4)
    return _case(call, kind, prec, dims, nrhs=nrhs, recon=rng.choice((12, 12, 18)),
                 dagger=plain and rng.random() < 0.4, twisted=plain and rng.random() < 0.25, kappa=kappa,
                 inner=rng.choice(("f16", "f32", "bf16")) if call == "richardson" else "",
                 rsd={"cg": 1e-10, "richardson": 1e-10, "multishift": 1e-9}.get(call, 0.0), shifts=shifts)


# ----------------------------------------------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------------------------------------------
def _dims(case):
    return case["nx"], case["ny"], case["nz"], case["nt"]


def _mass(case):
    return 0.5 / case["kappa"] - 4.0


def _shifts(case):
    return np.logspace(-4, 0, case["shifts"])


def _gaussian(gen, shape):
    return torch.view_as_complex(torch.randn(*shape, 2, generator=gen, device="cuda", dtype=torch.float64)) / math.sqrt(2)


def _inputs(case, seed):
    """links [4, V, 3, 3] and sources [nrhs, V, 4, 3], complex128 in CB2 order, on the GPU"""
    gen = torch.Generator("cuda").manual_seed(seed)
    v = math.prod(_dims(case))
    h = _gaussian(gen, (4, v, 3, 3))
    h = (h + h.mH) / math.sqrt(2)
    h.diagonal(dim1=-2, dim2=-1).sub_(h.diagonal(dim1=-2, dim2=-1).mean(-1, keepdim=True))
    m = 1j * EPS * h - EPS * EPS / 2 * (h @ h)
    m.diagonal(dim1=-2, dim2=-1).add_(1.0)
    a = m[..., 0, :] / torch.linalg.vector_norm(m[..., 0, :], dim=-1, keepdim=True)
    b = m[..., 1, :] - (a.conj() * m[..., 1, :]).sum(-1, keepdim=True) * a
    b = b / torch.linalg.vector_norm(b, dim=-1, keepdim=True)
    return torch.stack((a, b, torch.linalg.cross(a, b).conj()), -2), _gaussian(gen, (case["nrhs"], v, 4, 3))


class Outputs(dict):
    """Result fields by name; they stay on the device and are copied out when one is looked at."""

    def __getitem__(self, key):
        field, cb = super().__getitem__(key)
        if cb is None:
            return field.download()
        lat, wide = field.lat, field.prec == api.PREC["f64"]
        host = np.empty((field.nrhs, 2 * lat.vh, 4, 3), np.complex128 if wide else np.complex64)
        return field.download_qdp(host, cb)[:, cb * lat.vh:(cb + 1) * lat.vh]


def _clover_fields(lat, case, links, prec):
    """the odd term A and the even one's inverse(s), built in FP64 and stored in `prec`"""
    u = lat.gauge("f64", 18).upload_qdp(links)
    odd, even = (api.clover_build(lat.clover("f64"), u, cb, _mass(case), CSW) for cb in (1, 0))
    if case["kind"] == "tmclover":
        inverse = api.clover_invert_twisted(lat.full_clover("f64"), lat.full_clover("f64"), even, MU)
    else:
        inverse = (api.clover_invert(lat.clover("f64"), even),)
    if prec == "f64":
        return odd, inverse
    low = tuple(api.clover_convert(lat.full_clover(prec) if case["kind"] == "tmclover" else lat.clover(prec), f)
                for f in inverse)
    return api.clover_convert(lat.clover(prec), odd), low


def _operator(lat, case, links, prec):
    u = lat.gauge(prec, case["recon"]).upload_qdp(links)
    tbc = dict(use_tbc=[p != (1.0, 0.0) for p in PHASES], tbc_phases=PHASES) if case["twisted"] else {}
    if case["kind"] == "wilson":
        return api.EvenOddWilsonOperator(_mass(case), u, **tbc)
    if case["kind"] == "tm":
        return api.EvenOddTMWilsonOperator(_mass(case), MU, u, **tbc)
    odd, inverse = _clover_fields(lat, case, links, prec)
    if case["kind"] == "clover":
        return api.EvenOddCloverOperator(u, odd, inverse[0], **tbc)
    return api.EvenOddTMCloverOperator(u, odd, inverse, prec_mass_rho=MU, **tbc)


def _dslash(lat, case, links):
    """the first half of the operator: odd to even, with the inverse of the even diagonal"""
    prec, use = case["prec"], [p != (1.0, 0.0) for p in PHASES] if case["twisted"] else None
    u = lat.gauge(prec, case["recon"]).upload_qdp(links)
    geometry, tbc = (lat, -1.0, 1.0, 1.0), dict(use_tbc=use, tbc_phases=PHASES)
    if case["kind"] == "wilson":
        return api.Dslash(*geometry, **tbc), (u,)
    if case["kind"] == "tm":
        return api.TMDslash(*geometry, _mass(case), MU, **tbc), (u,)
    _, inverse = _clover_fields(lat, case, links, prec)
    if case["kind"] == "clover":
        return api.ClovDslash(*geometry, **tbc), (u, inverse[0])
    return api.TMClovDslash(*geometry, prec_mass_rho=MU, **tbc), (u, inverse)


def prepare(case, seed):
    links, source = (t.cpu().numpy() for t in _inputs(case, seed))
    lat = api.Lattice(_dims(case))
    s = dict(case=case, lat=lat, isign=-1 if case["dagger"] else 1)
    if case["call"] == "clover_term":
        s.update(u=lat.gauge("f64", 18).upload_qdp(links), terms=(lat.clover("f64"), lat.clover("f64")),
                 inverse=lat.clover("f64"))
        lat.sync()
        return s
    s["b"] = lat.spinor(case["prec"], case["nrhs"]).upload_qdp(source, 1)
    if case["call"] == "dslash":
        s["D"], s["args"] = _dslash(lat, case, links)
    else:
        s["M"] = _operator(lat, case, links, case["prec"])
    if case["call"] == "cg":
        s["solve"] = api.InvCG(s["M"], 5000)
    elif case["call"] == "richardson":
        s["solve"] = api.InvRichardsonMultiPrec(s["M"], _operator(lat, case, links, case["inner"]), "bicgstab",
                                                delta=0.005, max_iters=100, inner_max_iters=5000)
    elif case["call"] == "multishift":
        s["solve"] = api.MInvCG(s["M"], 5000)
        s["shifts"], s["rsd"] = _shifts(case), [case["rsd"]] * case["shifts"]
        s["xs"] = [lat.spinor(case["prec"]) for _ in range(case["shifts"])]
    if "xs" not in s:
        s["x"] = lat.spinor(case["prec"], case["nrhs"])
    lat.sync()
    return s


def run(state):
    call = state["case"]["call"]
    if call == "clover_term":
        case, (even, odd) = state["case"], state["terms"]
        api.clover_build(even, state["u"], 0, _mass(case), CSW)
        api.clover_build(odd, state["u"], 1, _mass(case), CSW)
        api.clover_invert(state["inverse"], even)
        return Outputs(even=(even, None), odd=(odd, None), inverse=(state["inverse"], None))
    if call == "multishift":
        state["solve"](state["xs"], state["b"], state["shifts"], state["rsd"])
        return Outputs({"x%02d" % i: (x, 1) for i, x in enumerate(state["xs"])})
    x, b = state["x"], state["b"]
    if call == "dslash":
        state["D"].dslash(x, b, *state["args"], state["isign"], 0)
        return Outputs(x=(x, 0))
    if call == "operator":
        state["M"](x, b, state["isign"])
    else:  # from a zero guess
        api.zero(x)
        state["solve"](x, b, state["case"]["rsd"])
    return Outputs(x=(x, 1))


# ----------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ----------------------------------------------------------------------------------------------------------------
_HOP, _CLOVER, _REAL = 1320, 504, {"f64": 8, "f32": 4, "f16": 2, "bf16": 2}
# operator applications (M or its dagger) that these solves take, about
_APPLICATIONS = {"cg": 80, "richardson": 230, "multishift": 110}


def _spinor_bytes(prec):
    return 24 * _REAL[prec] + (4 if _REAL[prec] == 2 else 0)


def _operator_work(case, prec, hops):
    """one application: links, terms and the source read once, the result written once"""
    vh, e = math.prod(_dims(case)) // 2, _REAL[prec]
    term = {"wilson": 0, "tm": 0, "clover": 72, "tmclover": 144}[case["kind"]] + (
        72 if hops == 2 and "clover" in case["kind"] else 0)
    terms = hops if "clover" in case["kind"] else 0
    return {"bytes": vh * (8 * case["recon"] * e + term * e + 2 * case["nrhs"] * _spinor_bytes(prec)),
            "flops": vh * case["nrhs"] * (hops * _HOP + terms * _CLOVER + (hops - 1) * 48)}


def work(case):
    vh, call = math.prod(_dims(case)) // 2, case["call"]
    if call == "clover_term":
        # six planes of four leaves (a product of four links) a site, both checkerboards; one inverse
        return {"bytes": vh * (8 * 18 * 8 + 3 * 72 * 8), "flops": 2 * vh * 6 * 4 * 3 * 198 + vh * 2 * 4 * 6 ** 3}
    if call in ("dslash", "operator"):
        return _operator_work(case, case["prec"], 1 if call == "dslash" else 2)
    n = _APPLICATIONS[call]
    w = _operator_work(case, case["inner"] or case["prec"], 2)
    # the operator's bytes each application, and the solver's vectors: a CG half-iteration passes over about 4
    # spinors, a BiCGStab half-iteration over about 9; a multishift solve also writes each solution once
    spinor = vh * case["nrhs"] * _spinor_bytes(case["inner"] or case["prec"])
    return {"bytes": n * (w["bytes"] + {"richardson": 9}.get(call, 4) * spinor) + case["shifts"] * spinor,
            "flops": n * w["flops"]}


def tolerance(case):
    if case["call"] in ("cg", "richardson", "multishift"):
        # every solution within the residual target is right: they lie 5 to 10 targets from the exact one
        return {"rel": 4e-8 if case["call"] == "multishift" else 1e-8, "max": 1e-6}
    # storage of the result, once or (operator) twice, and the sums in the arithmetic type: the results lie
    # 1 to 4e-16, 1 to 3e-7, 3 to 5e-4 and 3 to 5e-3 from the exact ones
    return {"f64": {"rel": 2e-15, "max": 1e-13}, "f32": {"rel": 1e-6, "max": 4e-5},
            "f16": {"rel": 1.5e-3, "max": 4e-2}, "bf16": {"rel": 1.2e-2, "max": 0.3}}[case["prec"]]


# ----------------------------------------------------------------------------------------------------------------
# the same in FP64: arrays over the whole lattice, [t, z, y, x] after the leading indices
# ----------------------------------------------------------------------------------------------------------------
# gamma_mu psi = coefficient[s] psi[permutation[s]] (DeGrand-Rossi)
_GAMMA = (((3, 2, 1, 0), (1j, 1j, -1j, -1j)), ((3, 2, 1, 0), (-1, 1, 1, -1)), ((2, 3, 0, 1), (1j, -1j, -1j, 1j)),
          ((2, 3, 0, 1), (1, 1, 1, 1)))


def _gamma(mu):
    perm, coef = _GAMMA[mu]
    g = torch.zeros(4, 4, dtype=torch.complex128)
    for s in range(4):
        g[s, perm[s]] = coef[s]
    return g.cuda()


class _Exact:
    def __init__(self, case, links):
        self.case, self.dims = case, _dims(case)
        nx, ny, nz, nt = self.dims
        t, z, y, x = torch.meshgrid(*(torch.arange(n, device="cuda") for n in (nt, nz, ny, nx)), indexing="ij")
        self.parity = (x + y + z + t) & 1
        site = ((t * nz + z) * ny + y) * (nx // 2) + x // 2
        self.index = (self.parity * (nx * ny * nz * nt // 2) + site).reshape(-1)  # CB2 place of every site
        self.u = [self.full(links[mu]) for mu in range(4)]
        self.even, self.odd = (self.parity == p for p in (0, 1))
        if "clover" in case["kind"]:
            self.term = self.clover_term()

    def full(self, a):
        nx, ny, nz, nt = self.dims
        return a[self.index].reshape(nt, nz, ny, nx, *a.shape[1:])

    def half(self, a, cb):
        """checkerboard cb of a full-lattice array, in the library's order"""
        out = torch.empty_like(a.reshape(-1, *a.shape[4:]))
        out[self.index] = a.reshape(-1, *a.shape[4:])
        n = out.shape[0] // 2
        return out[cb * n:(cb + 1) * n]

    def edge(self, a, axis, at):
        if axis == 0:  # antiperiodic in t
            a[at] = -a[at]
        return a

    def hop(self, psi, sign):
        out = torch.zeros_like(psi)
        for mu, axis in enumerate((3, 2, 1, 0)):
            perm, coef = _GAMMA[mu]
            gamma = torch.tensor(coef, dtype=torch.complex128, device="cuda")[:, None]
            phase = complex(*PHASES[mu]) if self.case["twisted"] else 1.0
            ahead = self.edge(torch.roll(psi, -1, axis), axis, -1)
            ahead = (ahead - sign * gamma * ahead[..., perm, :]) * phase
            behind = psi + sign * gamma * psi[..., perm, :]
            u = self.u[mu].unsqueeze(-3)
            out += (u * ahead.unsqueeze(-2)).sum(-1)
            behind = (u.conj() * behind.unsqueeze(-1)).sum(-2)
            out += self.edge(torch.roll(behind, 1, axis), axis, 0) * np.conj(phase)
        return out

    def clover_term(self):
        """A as two 6 x 6 blocks a site: 4 + m - csw / 2 sum_(mu < nu) gamma_mu gamma_nu F, F = (Q - Q^+) / 8"""
        axis, n = (3, 2, 1, 0), self.parity.shape
        a = torch.zeros(*n, 2, 6, 6, dtype=torch.complex128, device="cuda")
        a.diagonal(dim1=-2, dim2=-1).add_(4.0 + _mass(self.case))
        for mu in range(4):
            for nu in range(mu + 1, 4):
                um, un = self.u[mu], self.u[nu]
                plaquette = um @ torch.roll(un, -1, axis[mu]) @ torch.roll(um, -1, axis[nu]).mH @ un.mH
                # the four leaves at x, each from the plaquette of which x is another corner
                q = plaquette.clone()
                q += torch.roll(un.mH @ plaquette @ un, 1, axis[nu])
                q += torch.roll(um.mH @ plaquette @ um, 1, axis[mu])
                corner = torch.roll(un, 1, axis[nu])  # U_nu(x - nu)
                both = torch.roll(um, 1, axis[mu]).mH @ torch.roll(corner, 1, axis[mu]).mH
                q += both @ torch.roll(torch.roll(plaquette, 1, axis[nu]), 1, axis[mu]) @ both.mH
                f = (q - q.mH) / 8
                g = _gamma(mu) @ _gamma(nu)
                for b in range(2):
                    spin = g[2 * b:2 * b + 2, 2 * b:2 * b + 2]
                    a[..., b, :, :] -= CSW / 2 * torch.einsum("ij,...ab->...iajb", spin, f).reshape(*n, 6, 6)
        return a

    def blocks(self, a, psi):
        v = psi.reshape(*psi.shape[:-2], 2, 6)
        return (a * v.unsqueeze(-2)).sum(-1).reshape(psi.shape)

    def twist(self, psi, mu):
        """i mu gamma_5 psi"""
        out = psi * (1j * mu)
        out[..., 2:, :] *= -1
        return out

    def inverse_diagonal(self, psi, sign):
        kind, alpha = self.case["kind"], 4.0 + _mass(self.case)
        if kind == "wilson":
            return psi
        if kind == "tm":
            m = MU / alpha
            return (psi - self.twist(psi, sign * m)) / (alpha * (1 + m * m))
        if not hasattr(self, "inv"):
            self.inv = {}
        if sign not in self.inv:
            a = self.term.clone()
            if kind == "tmclover":
                for b in range(2):
                    a[..., b, :, :].diagonal(dim1=-2, dim2=-1).add_(1j * MU * sign * (1 - 2 * b))
            self.inv[sign] = torch.linalg.inv(a)
        return self.blocks(self.inv[sign], psi)

    def dslash(self, psi, sign):
        return self.inverse_diagonal(self.hop(psi, sign), sign)

    def operator(self, psi, sign=1):
        kind, alpha = self.case["kind"], 4.0 + _mass(self.case)
        back = self.hop(self.dslash(psi, sign), sign)
        if kind == "wilson":
            return alpha * psi - 0.25 / alpha * back
        if kind == "tm":
            return alpha * psi + self.twist(psi, sign * MU) - 0.25 * back
        first = self.blocks(self.term, psi) - 0.25 * back
        return first + self.twist(psi, sign * MU) if kind == "tmclover" else first


def _inner(a, b):
    return torch.vdot(a.reshape(-1), b.reshape(-1))


def _bicgstab(op, b, rsd):
    x, r = torch.zeros_like(b), b.clone()
    r0, p, v = r.clone(), torch.zeros_like(b), torch.zeros_like(b)
    rho = alpha = omega = 1.0
    stop = (rsd * torch.linalg.vector_norm(b)).item()
    for _ in range(2000):
        new = _inner(r0, r)
        p = r + (new / rho) * (alpha / omega) * (p - omega * v)
        rho, v = new, op(p)
        alpha = rho / _inner(r0, v)
        s = r - alpha * v
        t = op(s)
        omega = _inner(t, s) / _inner(t, t)
        x += alpha * p + omega * s
        r = s - omega * t
        if torch.linalg.vector_norm(r).item() < stop:
            break
    return x


def _multishift(op, b, shifts, rsd):
    """CG on op + shift for every shift (Jegerlehner's recurrences), until the slowest has met rsd"""
    xs, ps = [torch.zeros_like(b) for _ in shifts], [b.clone() for _ in shifts]
    base, r, p = min(shifts), b.clone(), b.clone()
    zeta, zeta_old = [1.0] * len(shifts), [1.0] * len(shifts)
    rr, alpha_old, beta = _inner(r, r).real.item(), 1.0, 0.0
    stop = rsd * rsd * rr
    for _ in range(2000):
        q = op(p) + base * p
        alpha = rr / _inner(p, q).real.item()
        r = r - alpha * q
        new = _inner(r, r).real.item()
        next_beta = new / rr
        for i, s in enumerate(shifts):
            z, z0 = zeta[i], zeta_old[i]
            z1 = z * z0 * alpha_old / (alpha * beta * (z0 - z) + z0 * alpha_old * (1 + alpha * (s - base)))
            xs[i] += alpha * z1 / z * ps[i]
            ps[i] = z1 * r + next_beta * (z1 / z) ** 2 * ps[i]
            zeta[i], zeta_old[i] = z1, z
        p = r + next_beta * p
        rr, alpha_old, beta = new, alpha, next_beta
        if rr < stop:
            break
    return xs


def exact(case, seed):
    links, source = _inputs(case, seed)
    ref = _Exact(case, links)
    call, sign = case["call"], -1 if case["dagger"] else 1
    if call == "clover_term":
        def packed(a):  # two blocks of 6 diagonal reals and 15 complex numbers below the diagonal
            rows, cols = np.tril_indices(6, -1)
            below = torch.view_as_real(a[..., rows, cols].contiguous()).reshape(*a.shape[:-2], 30)
            return torch.cat((a.diagonal(dim1=-2, dim2=-1).real, below), -1).reshape(*a.shape[:4], 72)
        a = packed(ref.term)
        return dict(even=ref.half(a, 0), odd=ref.half(a, 1),
                    inverse=ref.half(packed(torch.linalg.inv(ref.term)), 0))
    odd = ref.odd[..., None, None]

    def normal(v):
        return ref.operator(ref.operator(v, 1), -1) * odd

    found = []
    for b in source:
        b = ref.full(b) * odd
        if call == "dslash":
            found.append(ref.half(ref.dslash(b, sign), 0))
        elif call == "operator":
            found.append(ref.half(ref.operator(b, sign), 1))
        elif call == "cg":
            found.append(ref.half(_multishift(normal, b, [0.0], 1e-14)[0], 1))
        elif call == "richardson":
            found.append(ref.half(_bicgstab(lambda v: ref.operator(v) * odd, b, 1e-14), 1))
        else:
            return {"x%02d" % i: ref.half(x, 1)[None]
                    for i, x in enumerate(_multishift(normal, b, list(_shifts(case)), 1e-13))}
    return dict(x=torch.stack(found))
