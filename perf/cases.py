"""Performance cases of the SU(3) Wilson-fermion path: what a user's program calls, at the sizes it is used at.

Every case goes through the package's public entry points (``WilsonContext.apply / solve`` and the
``SU3WilsonNf2`` operators, forces and molecular-dynamics hooks) with seeded synthetic fields: links
exp(i a H) with H traceless Hermitian and Gaussian, Gaussian or point spinors.  ``exact`` restates each
result in plain torch at 64 bits (4x4 gamma matrices, rolls, FP64 CG).

Kinds of case
  apply     one Wilson operator on a batch of fields
  force     the pseudofermion force of given solutions (unpreconditioned or even-odd)
  gauge     the gauge part of a molecular-dynamics step: staple force and exponential drift
  solve     a conjugate-gradient solve of the normal equations for a batch of right-hand sides
  md        one molecular-dynamics update of the Nf=2 theory: drift of the links, then the whole force
"""

from __future__ import annotations

import math

import torch

from jaxqft_b200.lib import WilsonContext
from jaxqft_b200.su3_wilson_nf2 import SU3WilsonNf2

# boundary phases (x, y, z, t) by name
BCS = {
    "periodic": (1, 1, 1, 1),
    "antiperiodic": (1, 1, 1, -1),
    "complex": (1, 1, 1j, -1),
}
SOLVE_KAPPAS = (0.120, 0.125, 0.130, 0.135)
# true residual of every solve: that of the HMC chain tests, so that a solution has ten digits to compare
TOL = 1e-12


def listed():
    return [
        # the operator on the smallest lattice a propagator server holds: latency of one call
        _case("d_8x8x8x8", "apply", (8, 8, 8, 8), op="D"),
        # the operator on the production lattice, one field
        _case("d_24x24x24x48", "apply", (24, 24, 24, 48), op="D"),
        # D^dagger on the twelve spin-colour point sources of a propagator (the source of the normal equations)
        _case("ddag_12_sources_16x16x16x32", "apply", (16, 16, 16, 32), op="DDAG", nrhs=12, source="point"),
        # the even-odd normal operator on an anisotropic lattice with a complex phase, a few fields
        _case("schur_normal_6x10x14x18", "apply", (6, 10, 14, 18), op="SCHUR_E_NORMAL", nrhs=3, bc="complex"),
        # the force of the unpreconditioned monomial from its solutions, two configurations of a batched chain
        _case("force_2_12x12x12x24", "force", (12, 12, 12, 24), nconf=2),
        # the force of the even-odd preconditioned monomial on the HMC lattice
        _case("force_eo_16x16x16x32", "force", (16, 16, 16, 32), eo=True),
        # the gauge sector of one MD step on the HMC lattice
        _case("gauge_16x16x16x32", "gauge", (16, 16, 16, 32)),
        # the solve of one pseudofermion: one right-hand side, FP32 iteration, FP64 reliable updates
        _case("solve_eo_single_16x16x16x32", "solve", (16, 16, 16, 32), op="eo_normal", inner="single"),
        # plain FP64 CG on the unpreconditioned normal equations
        _case("solve_double_12x12x12x24", "solve", (12, 12, 12, 24), op="normal", inner="double"),
        # the smallest propagator of a server: twelve point sources on 8^4, FP16 iteration
        _case("solve_eo_half_12_8x8x8x8", "solve", (8, 8, 8, 8), op="eo_normal", inner="half", nrhs=12,
              source="point", kappa=0.130),
        # the batched production solve: 12 point sources and 4 Gaussian ones, FP16 iteration
        _case("solve_eo_half_16_24x24x24x48", "solve", (24, 24, 24, 48), op="eo_normal", inner="half", nrhs=16,
              source="point"),
        # a whole MD update at the couplings of the HMC runs: new links, gauge force, CG solve, pseudofermion force
        _case("md_16x16x16x32", "md", (16, 16, 16, 32), kappa=0.150, scale=0.1),
    ]


def _case(name, kind, shape, op="", nrhs=1, nconf=1, kappa=0.135, scale=0.2, bc="antiperiodic", source="gauss",
          inner="", eo=False):
    c = {"name": name, "kind": kind, "lx": shape[0], "ly": shape[1], "lz": shape[2], "lt": shape[3], "op": op,
         "nrhs": nrhs, "nconf": nconf, "kappa": kappa, "scale": scale, "bc": bc, "source": source, "inner": inner,
         "eo": eo}
    if not name:
        del c["name"]
    return c


def _even(rng, lo, hi):
    """An even extent in [lo, hi], its logarithm uniform."""
    return max(lo, min(hi, 2 * round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / 2)))


def _shape(rng, sites):
    while True:
        s = (_even(rng, 4, 24), _even(rng, 4, 24), _even(rng, 4, 24), _even(rng, 4, 64))
        if 256 <= math.prod(s) <= sites:
            return s


def draw(rng):
    kind = rng.choice(("apply", "apply", "apply", "force", "gauge", "solve", "solve", "solve", "md"))
    bc = rng.choice(tuple(BCS))
    if kind == "apply":
        nrhs = rng.choice((1, 1, 2, 3, 4, 5, 8, 12))
        op = rng.choice(("D", "DDAG", "DDAGD", "HOP", "K_OE", "K_EO", "KDAG_OE", "SCHUR_E", "SCHUR_E_DAG", "SCHUR_O",
                         "SCHUR_E_NORMAL"))
        # the point sources sit on an even site, so operators on odd fields take Gaussian ones
        source = "gauss" if _APPLY_PARITY.get(op) == 1 else rng.choice(("gauss", "point"))
        return _case("", kind, _shape(rng, 1_500_000 // nrhs), op=op, nrhs=nrhs, bc=bc,
                     kappa=rng.uniform(0.120, 0.135), source=source)
    if kind == "force":
        nconf = rng.choice((1, 1, 2, 3))
        return _case("", kind, _shape(rng, 150_000), nconf=nconf, bc=bc, eo=rng.random() < 0.5)
    if kind == "gauge":
        nconf = rng.choice((1, 1, 2, 3))
        return _case("", kind, _shape(rng, 150_000), nconf=nconf, bc=bc)
    if kind == "solve":
        inner = rng.choice(("half", "half", "single", "single", "double"))
        nrhs = rng.randint(1, 3) if inner == "double" else rng.randint(1, 16)
        sites = 140_000 if inner == "double" else 1_200_000 // nrhs
        return _case("", kind, _shape(rng, min(sites, 300_000)), op=rng.choice(("eo_normal", "eo_normal", "normal")),
                     nrhs=nrhs, inner=inner, kappa=rng.choice(SOLVE_KAPPAS), source=rng.choice(("gauss", "point")),
                     bc=rng.choice(("antiperiodic", "complex")))
    return _case("", kind, _shape(rng, 140_000), kappa=0.150, scale=0.1, eo=rng.random() < 0.5)


# --------------------------------------------------------------------------- inputs
def _dims(case):
    return case["lx"], case["ly"], case["lz"], case["lt"]


def _mass(case):
    return 1.0 / (2.0 * case["kappa"]) - 4.0


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _normal(gen, shape):
    return torch.complex(torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64),
                         torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64))


def _traceless_antihermitian(m):
    y = 0.5 * (m - m.conj().transpose(-1, -2))
    tr = torch.diagonal(y, dim1=-2, dim2=-1).sum(-1) / 3.0
    return y - tr[..., None, None] * torch.eye(3, device=m.device, dtype=m.dtype)


def _links(gen, case):
    shape = (case["nconf"], 4, *_dims(case), 3, 3)
    return torch.linalg.matrix_exp(_traceless_antihermitian(case["scale"] * _normal(gen, shape)))


def _fields(gen, case, n):
    """n spinors: Gaussian with unit variance per component, or (source "point") unit sources at site 0, one
    per spin and colour, followed by Gaussian ones."""
    shape = _dims(case)
    psi = _normal(gen, (n, *shape, 4, 3)) / math.sqrt(2.0)
    if case["source"] == "point":
        k = min(n, 12)
        psi[:k] = 0
        for i in range(k):
            psi[i, 0, 0, 0, 0, i // 3, i % 3] = 1.0
    return psi


def _parity(case):
    x = [torch.arange(n, device="cuda") for n in _dims(case)]
    p = x[0][:, None, None, None] + x[1][:, None, None] + x[2][:, None] + x[3]
    return (p % 2)[..., None, None]


def _theory(case, **kw):
    return SU3WilsonNf2(lattice_shape=_dims(case), beta=5.6, batch_size=case["nconf"], mass=_mass(case),
                        fermion_bc=BCS[case["bc"]], solver_precision="single", cg_tol=TOL, cg_maxiter=20000,
                        fermion_monomial_kind="eo_preconditioned" if case["eo"] else "unpreconditioned", **kw)


_APPLY_PARITY = {"K_OE": 0, "KDAG_OE": 0, "SCHUR_E": 0, "SCHUR_E_DAG": 0, "SCHUR_E_NORMAL": 0, "K_EO": 1,
                 "SCHUR_O": 1}
MD_DT = 0.05


def _inputs(case, seed):
    """The tensors of a case, from the seed alone (shared by prepare and exact)."""
    gen = _generator(seed)
    U = _links(gen, case)
    kind = case["kind"]
    if kind == "apply":
        psi = _fields(gen, case, case["nrhs"])
        if case["op"] in _APPLY_PARITY:
            psi = psi * (_parity(case) == _APPLY_PARITY[case["op"]])
        return {"U": U, "psi": psi}
    if kind == "force":
        X, Y = _fields(gen, case, case["nconf"]), _fields(gen, case, case["nconf"])
        if case["eo"]:
            even = _parity(case) == 0
            X, Y = X * even, Y * even
        return {"U": U, "X": X, "Y": Y}
    if kind == "gauge":
        return {"U": U, "P": _traceless_antihermitian(_normal(gen, U.shape))}
    if kind == "solve":
        psi = _fields(gen, case, case["nrhs"])
        if case["op"] == "eo_normal":
            psi = psi * (_parity(case) == 0)
        return {"U": U, "psi": psi}
    psi = _fields(gen, case, case["nconf"])
    if case["eo"]:
        psi = psi * (_parity(case) == 0)
    return {"U": U, "P": _traceless_antihermitian(_normal(gen, U.shape)), "phi": psi}


# --------------------------------------------------------------------------- the framework
def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = case
    kind = case["kind"]
    if kind in ("apply", "solve"):
        s["ctx"] = WilsonContext(_dims(case), bc=BCS[case["bc"]], device="cuda:0")
        s["gauge"] = s["ctx"].gauge(s["U"][0])
        s["mass"] = _mass(case)
    else:
        s["theory"] = _theory(case)
    if kind == "solve":
        # the sources of the normal equations, as propagator and pseudofermion code makes them
        if case["op"] == "eo_normal":
            s["b"] = s["ctx"].apply("SCHUR_E_DAG", s["gauge"], s["mass"], s["psi"], normalized=True)
        else:
            s["b"] = s["ctx"].apply("DDAG", s["gauge"], s["mass"], s["psi"])
        del s["psi"]
    if kind == "md":
        th = s["theory"]
        phi = (th.apply_eo_schur_even_dagger(s["U"], s["phi"], normalized=True) if case["eo"]
               else th.apply_Ddag(s["U"], s["phi"]))
        th.set_loaded_pseudofermion(phi)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "apply":
        normalized = case["op"].startswith("SCHUR")
        return s["ctx"].apply(case["op"], s["gauge"], s["mass"], s["psi"], normalized=normalized)
    if kind == "force":
        th = s["theory"]
        if case["eo"]:
            return th.eop_pseudofermion_force_from_solution(s["U"], s["X"], s["Y"])
        return th.pseudofermion_force_from_solution(s["U"], s["X"], s["Y"])
    if kind == "gauge":
        th = s["theory"]
        F = th.gauge_force(s["U"])
        return {"F": F, "U": th.evolve_q(MD_DT, s["P"], s["U"])}
    if kind == "solve":
        x, _ = s["ctx"].solve(s["gauge"], s["b"], s["mass"], op=case["op"], tol=TOL, maxiter=4000,
                              inner=case["inner"])
        return x
    th = s["theory"]
    U = th.evolve_q(MD_DT, s["P"], s["U"])
    return {"U": U, "F": th.force(U)}


# --------------------------------------------------------------------------- what a pass cannot do without
# CG iterations of the FP64 solve to TOL at SOLVE_KAPPAS (16^3x32, links exp(0.2 i H)), even-odd and full lattice
_ITERS = {"eo_normal": (77, 108, 182, 156), "normal": (221, 317, 500, 479)}
_D_FLOPS = 1368.0  # the rank-2 form: 8 hops of two 3x3 complex matrix-vector products, projections and sums


def work(case):
    V = float(math.prod(_dims(case)))
    link, spinor = 144.0, 192.0
    kind, n = case["kind"], case["nrhs"]
    if kind == "apply":
        op = case["op"]
        half = op in _APPLY_PARITY
        hops = {"DDAGD": 2.0, "SCHUR_E_NORMAL": 2.0, "SCHUR_E": 1.0, "SCHUR_E_DAG": 1.0, "SCHUR_O": 1.0}.get(
            op, 0.5 if half else 1.0)
        # half-lattice operators need the input of one parity; the whole output is written (zeros on the other)
        return {"bytes": V * 4 * link + n * V * spinor * (1.5 if half else 2.0), "flops": n * V * hops * _D_FLOPS}
    if kind == "force":
        # per link two half-spinor products U X, U Y and the outer products of spin
        return {"bytes": case["nconf"] * V * (8 * link + spinor * (1.0 if case["eo"] else 2.0)),
                "flops": case["nconf"] * V * 4 * (600.0 if case["eo"] else 1200.0)}
    if kind == "gauge":
        # 6 plaquettes per site: staples of 12 products per link, and a matrix exponential
        return {"bytes": case["nconf"] * V * 4 * 4 * link, "flops": case["nconf"] * V * 4 * (13 + 8) * 198.0}
    if kind == "solve":
        k = case["kappa"]
        i = min(range(len(SOLVE_KAPPAS)), key=lambda j: abs(SOLVE_KAPPAS[j] - k))
        iters = _ITERS[case["op"]][i]
        share = 0.5 if case["op"] == "eo_normal" else 1.0
        return {"bytes": V * 4 * link + n * V * spinor * (1.0 + share), "flops": n * iters * V * 2 * _D_FLOPS}
    iters = 250 if not case["eo"] else 110
    return {"bytes": case["nconf"] * V * (16 * link + spinor),
            "flops": case["nconf"] * V * (iters * 2 * _D_FLOPS + 4 * (13 + 8) * 198.0 + 4800.0)}


# --------------------------------------------------------------------------- the same in plain torch, 64 bits
def _gammas():
    s1 = torch.tensor([[0, 1], [1, 0]], dtype=torch.complex128)
    s2 = torch.tensor([[0, -1j], [1j, 0]], dtype=torch.complex128)
    s3 = torch.tensor([[1, 0], [0, -1]], dtype=torch.complex128)
    one = torch.eye(2, dtype=torch.complex128)
    return [torch.kron(a, b).cuda() for a, b in ((s1, s1), (s1, s2), (s2, one), (s3, one))]


class _Plain:
    """The Wilson operator of one configuration in plain torch."""

    def __init__(self, U, case):
        self.U = U.clone()  # [4, X, Y, Z, T, 3, 3], boundary phases folded in
        self.m0 = _mass(case) + 4.0
        for mu, phase in enumerate(BCS[case["bc"]]):
            if phase != 1:
                self.U[mu].select(mu, U.shape[1 + mu] - 1).mul_(phase)
        self.even = (_parity(case) == 0).to(torch.float64)
        self.gamma = []  # row s of gamma_mu: one entry `phase` in column `perm`
        for g in _gammas():
            perm = g.abs().argmax(dim=1)
            self.gamma.append((perm, g.gather(1, perm[:, None])))

    def g(self, mu, psi):
        perm, phase = self.gamma[mu]
        return psi[..., perm, :] * phase

    @staticmethod
    def color(u, psi, dagger=False):
        """u psi (or u^dagger psi) per site for psi [..., X, Y, Z, T, 4, 3]."""
        out = None
        for b in range(3):
            col = u[..., b, :].conj() if dagger else u[..., :, b]
            term = col[..., None, :] * psi[..., b:b + 1]
            out = term if out is None else out + term
        return out

    def hop(self, psi, dag=False):
        sign = -1.0 if dag else 1.0
        out = torch.zeros_like(psi)
        for mu in range(4):
            ax = psi.dim() - 6 + mu
            f = self.color(self.U[mu], torch.roll(psi, -1, ax))
            out = out + f - sign * self.g(mu, f)
            b = torch.roll(self.color(self.U[mu], psi, True), 1, ax)
            out = out + b + sign * self.g(mu, b)
        return -0.5 * out

    def D(self, psi, dag=False):
        return self.m0 * psi + self.hop(psi, dag)

    def schur(self, psi, parity, dag=False):
        """psi_p - K K psi_p / m0^2 on sites of `parity`."""
        p = self.even if parity == 0 else 1.0 - self.even
        t = self.hop(psi, dag) * (1.0 - p)
        return (psi - self.hop(t, dag) / self.m0 ** 2) * p

    def apply(self, op, psi):
        o = 1.0 - self.even
        table = {
            "D": lambda: self.D(psi), "DDAG": lambda: self.D(psi, True),
            "DDAGD": lambda: self.D(self.D(psi), True), "HOP": lambda: self.hop(psi),
            "K_OE": lambda: self.hop(psi) * o, "K_EO": lambda: self.hop(psi) * self.even,
            "KDAG_OE": lambda: self.hop(psi, True) * o,
            "SCHUR_E": lambda: self.schur(psi, 0), "SCHUR_E_DAG": lambda: self.schur(psi, 0, True),
            "SCHUR_O": lambda: self.schur(psi, 1),
            "SCHUR_E_NORMAL": lambda: self.schur(self.schur(psi, 0), 0, True),
        }
        return table[op]()

    def normal(self, op, psi):
        return self.apply("DDAGD" if op == "normal" else "SCHUR_E_NORMAL", psi)

    def cg(self, op, b, tol=1e-14, maxiter=3000):
        """CG for every field of b, stopped on the recursive residual."""
        x = torch.zeros_like(b)
        r = b.clone()
        p = b.clone()

        def norm2(v):
            return torch.linalg.vector_norm(v.flatten(1), dim=1) ** 2

        def wide(c):
            return c.reshape(-1, *([1] * (b.dim() - 1)))

        r2 = norm2(r)
        stop = tol ** 2 * r2
        for k in range(maxiter):
            if k % 10 == 0 and bool((r2 <= stop).all()):
                break
            ap = self.normal(op, p)
            pap = (p.conj() * ap).real.flatten(1).sum(1)
            alpha = torch.where(pap > 0, r2 / pap, torch.zeros_like(pap))
            x = x + wide(alpha) * p
            r = r - wide(alpha) * ap
            new = norm2(r)
            p = r + wide(torch.where(r2 > 0, new / r2, torch.zeros_like(r2))) * p
            r2 = new
        return x

    def force(self, X, Y):
        """The pseudofermion force of one configuration from fields X, Y [X, Y, Z, T, 4, 3]."""
        out = []
        for mu in range(4):
            u = self.U[mu]
            ux = self.color(u, torch.roll(X, -1, mu))
            w = ux - self.g(mu, ux)
            v = X + self.g(mu, X)
            z = self.color(u, torch.roll(Y, -1, mu))
            k = (torch.einsum("...sc,...sa->...ca", w, Y.conj()) - torch.einsum("...sc,...sa->...ca", v, z.conj()))
            out.append(_traceless_antihermitian(k))
        return torch.stack(out)

    def force_eo(self, X, Y):
        o = 1.0 - self.even
        kx, ky = self.hop(X) * o, self.hop(Y, True) * o
        return -(self.force(kx, Y) + self.force(X, ky)) / self.m0 ** 2


def _gauge_force(U, beta=5.6):
    """-(beta / 3) TA(U_mu V_mu^dagger) with the sum of the six staples V_mu, U [4, X, Y, Z, T, 3, 3]."""
    def dag(m):
        return m.conj().transpose(-1, -2)

    def mul(a, b):
        out = None
        for k in range(3):
            term = a[..., :, k, None] * b[..., None, k, :]
            out = term if out is None else out + term
        return out

    out = []
    for mu in range(4):
        V = torch.zeros_like(U[mu])
        for nu in range(4):
            if nu == mu:
                continue
            V = V + mul(mul(U[nu], torch.roll(U[mu], -1, nu)), dag(torch.roll(U[nu], -1, mu)))
            down = mul(mul(dag(U[nu]), U[mu]), torch.roll(U[nu], -1, mu))
            V = V + torch.roll(down, 1, nu)
        out.append(-(beta / 3.0) * _traceless_antihermitian(mul(U[mu], dag(V))))
    return torch.stack(out)


def exact(case, seed):
    kind = case["kind"]
    if kind == "solve" and case["nrhs"] * math.prod(_dims(case)) > 400_000:
        return None
    s = _inputs(case, seed)
    if kind == "apply":
        plain = _Plain(s["U"][0], case)
        return torch.cat([plain.apply(case["op"], f[None]) for f in s["psi"]])
    if kind == "force":
        plains = [_Plain(u, case) for u in s["U"]]
        return torch.stack([(p.force_eo if case["eo"] else p.force)(x, y)
                            for p, x, y in zip(plains, s["X"], s["Y"])])
    if kind == "gauge":
        return {"F": torch.stack([_gauge_force(u) for u in s["U"]]),
                "U": torch.linalg.matrix_exp(MD_DT * s["P"]) @ s["U"]}
    if kind == "solve":
        plain = _Plain(s["U"][0], case)
        b = plain.apply("SCHUR_E_DAG" if case["op"] == "eo_normal" else "DDAG", s["psi"])
        return plain.cg(case["op"], b)
    plain = _Plain(s["U"][0], case)
    phi = plain.schur(s["phi"], 0, True) if case["eo"] else plain.D(s["phi"], True)
    U = torch.linalg.matrix_exp(MD_DT * s["P"][0]) @ s["U"][0]
    plain = _Plain(U, case)
    if case["eo"]:
        x = plain.cg("eo_normal", phi)
        f = plain.force_eo(x[0], plain.schur(x, 0)[0])
    else:
        x = plain.cg("normal", phi)
        f = plain.force(x[0], plain.D(x)[0])
    return {"U": U[None], "F": (_gauge_force(U) + f)[None]}
