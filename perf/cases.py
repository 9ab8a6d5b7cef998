"""The work that a user of this library has it do, as cases to be timed.

A case names a lattice, a gauge group with a fermion representation and one call (or the
short sequence of calls that belong together) through `hirep_b200.hrgpu`.  `listed()` gives
the standing cases, `draw()` more of the same kinds over the same ranges, `prepare()` what a
program has in hand before the call (the lattice with its links, device fields, batches),
`run()` one pass, `exact()` the same results from plain torch in 64 bits.

The library drives one lattice with one gauge field per process, so the links belong to the
case (`links`, the seed they are made from) and the seed of `prepare()` makes the fields,
and for the molecular-dynamics cases the momenta.
"""
import math

import numpy as np
import torch

from hirep_b200 import hrgpu as G

REPR = {"fund": G.FUND, "adj": G.ADJ, "sym": G.SYM, "asym": G.ASYM}


def nf_of(c):
    n = c["ng"]
    return {"fund": n, "adj": n * n - 1, "sym": n * (n + 1) // 2, "asym": n * (n - 1) // 2}[c["repr"]]


def case(kind, dims, ng, repr_, eps, mass, csw=0.0, links=1, **more):
    t, x, y, z = dims
    return dict(kind=kind, t=t, x=x, y=y, z=z, ng=ng, repr=repr_, eps=eps, mass=mass, csw=csw, links=links, **more)


def listed():
    return [
        # config 1: a small hot lattice, where launches and latency count (tests, tuning runs, coarse levels)
        {"name": "eopre_su3_8x8", **case("op", (8, 8, 8, 8), 3, "fund", 0.0, 0.1, links=1234, call="Dphi_eopre", prec=64)},
        # config 2 and the benchmark's operator: the FP64 clover operator of a QCD-like run
        {"name": "clover_su3_32x16", **case("op", (32, 16, 16, 16), 3, "fund", 0.3, -0.2, 1.0, links=7, call="Cphi_eopre", prec=64)},
        # a ragged box, the full-lattice operator (measurements without even-odd preconditioning)
        {"name": "full_su4as_ragged", **case("op", (14, 6, 10, 12), 4, "asym", 0.25, -0.1, links=11, call="g5Dphi_sq", prec=64)},
        # config 4: the sextet clover operator at production size
        {"name": "clover_sextet_48x24", **case("op", (48, 24, 24, 24), 3, "sym", 0.3, -0.3, 1.0, links=21, call="Cphi_eopre", prec=64)},
        # config 5: the FP32 operator inside the mixed-precision force solves of the adjoint HMC
        {"name": "flt_su2adj_64x32", **case("op", (64, 32, 32, 32), 2, "adj", 0.2, -1.0, links=99, call="g5Dphi_eopre_sq_flt", prec=32)},
        # config 1's solve: CG on H^2 on a small lattice
        {"name": "cg_su3_8x8", **case("cg", (8, 8, 8, 8), 3, "fund", 0.0, 0.1, links=1234, err2=1e-24, flt=False, shifts=1, iters=60)},
        # config 2's solve: the mixed-precision CG of a force or propagator solve
        {"name": "cgmixed_clover_su3_32x16", **case("cg", (32, 16, 16, 16), 3, "fund", 0.3, -0.2, 1.0, links=7, err2=1e-24, flt=True, shifts=1, iters=115)},
        # an RHMC force solve: one source, ten shifts from 1e-4 to 10
        {"name": "rhmc_su4as_16x16", **case("cg", (16, 16, 16, 16), 4, "asym", 0.25, -0.1, links=11, err2=1e-20, flt=False, shifts=10, iters=60)},
        # a propagator solve with HiRep's own inverter for D
        {"name": "qmr_clover_su3_24x12", **case("qmr", (24, 12, 12, 12), 3, "fund", 0.3, -0.2, 1.0, links=5, err2=1e-20, iters=110)},
        # config 4's batched operator: twelve sources at once, FP32 (the inner operator of the batched solve)
        {"name": "batch12_sextet_48x24", **case("batch", (48, 24, 24, 24), 3, "sym", 0.3, -0.3, 1.0, links=21, nb=12, prec=32)},
        # config 3's force as one molecular-dynamics step: fermion force, gauge force, link update, first operator after it
        {"name": "md_su4as_16x16", **case("md", (16, 16, 16, 16), 4, "asym", 0.25, -0.1, links=11, beta=11.0)},
        # the same step with a clover term: clover force, log-det force, clover term and its inverse rebuilt
        {"name": "md_clover_sextet_24x12", **case("md", (24, 12, 12, 12), 3, "sym", 0.3, -0.3, 1.0, links=21, beta=6.0)},
    ]


GROUPS = [(2, "fund"), (3, "fund"), (4, "fund"), (2, "adj"), (3, "sym"), (4, "asym")]


def draw(rng):
    kind = rng.choice(["op", "op", "op", "cg", "cg", "qmr", "batch", "batch", "md", "md"])
    # lattice points times colour matrix size, at most (the largest listed case of the kind)
    most = {"op": 48 * 24**3 * 36, "cg": 16**4 * 36, "qmr": 24 * 12**3 * 9, "batch": 48 * 24**3 * 36, "md": 24 * 12**3 * 36}[kind]
    ng, r = rng.choice(GROUPS)
    c = {"ng": ng, "repr": r}
    nf = nf_of(c)
    while True:
        v = math.exp(rng.uniform(math.log(512), math.log(most / nf**2)))
        side = max(2, round(v**0.25 / 2)) * 2
        dims = [max(4, 2 * round(side * rng.uniform(0.55, 1.6) / 2)) for _ in range(4)]
        dims[0] = max(4, 2 * round(v / (dims[1] * dims[2] * dims[3]) / 2))
        if dims[0] <= 96 and math.prod(dims) * nf**2 <= most:
            break
    csw = rng.choice([0.0, 1.0])
    a = (kind, dims, ng, r, 0.25, rng.choice([-0.2, -0.1, 0.0, 0.1]), csw)
    more = {"links": rng.randrange(1 << 20)}
    if kind == "op":
        if csw:
            call = rng.choice(["Cphi_eopre", "g5Cphi_eopre_sq", "g5Cphi_eopre_flt", "g5Cphi"])
        else:
            call = rng.choice(["Dphi_eopre", "g5Dphi_eopre_sq", "Dphi_eopre_flt", "Dphi", "g5Dphi_flt"])
        more.update(call=call, prec=32 if call.endswith("flt") else 64)
    elif kind == "cg":
        n = rng.choice([1, 1, 3, 6, 10])
        more.update(err2=1e-20, flt=rng.random() < 0.5, shifts=n, iters=60)
    elif kind == "qmr":
        more.update(err2=1e-20, iters=70)
    elif kind == "batch":
        # as many (site, field) pairs as the largest listed case at most
        more.update(nb=rng.randint(1, 12), prec=rng.choice([32, 64]) if math.prod(dims) * nf**2 * 4 <= most else 32)
    else:
        more.update(beta=6.0)
    return case(*a, **more)


# ------------------------------------------------------------------ the lattice in hand

_live = {"key": None}


def generators(ng):
    """T_A of su(ng) in the library's order (Tr T_A T_B = delta/2)."""
    out = []
    for a in range(ng):
        for b in range(ng):
            m = np.zeros((ng, ng), complex)
            if a > b:
                m[a, b] = m[b, a] = 1
            elif a < b:
                m[a, b], m[b, a] = 1j, -1j
            elif a:
                q = math.sqrt(2.0 / (a * (a + 1)))
                m[np.arange(a), np.arange(a)] = q
                m[a, a] = -a * q
            else:
                continue
            out.append(m / 2)
    return torch.tensor(np.array(out), device="cuda")


def make_links(c):
    """Links U[t,x,y,z,mu] on the GPU: exp(i eps sum_A h_A T_A) with Gaussian h, or Haar-random for eps = 0."""
    ng, v4 = c["ng"], c["t"] * c["x"] * c["y"] * c["z"] * 4
    gen = torch.Generator("cuda").manual_seed(c["links"])
    out = torch.empty((v4, ng, ng), dtype=torch.complex128, device="cuda")
    step = 1 << 21
    for s in range(0, v4, step):
        n = min(step, v4 - s)
        if c["eps"]:
            h = torch.randn((n, ng * ng - 1), generator=gen, dtype=torch.float64, device="cuda")
            out[s : s + n] = torch.linalg.matrix_exp(1j * c["eps"] * torch.einsum("na,aij->nij", h + 0j, generators(ng)))
        else:
            q, r = torch.linalg.qr(torch.randn((n, ng, ng), generator=gen, dtype=torch.complex128, device="cuda"))
            d = torch.diagonal(r, dim1=1, dim2=2)
            q = q * (d / d.abs())[:, None, :]
            out[s : s + n] = q / torch.linalg.det(q)[:, None, None] ** (1.0 / ng)
    return out.reshape(c["t"], c["x"], c["y"], c["z"], 4, ng, ng)


def lattice(c):
    """The library's lattice for this case with its links set (kept while the case stays the same)."""
    key = tuple((k, c[k]) for k in ("t", "x", "y", "z", "ng", "repr", "eps", "csw", "links"))
    if _live["key"] != key:
        _live.update(key=None, lat=None, host=None)
        ipt = G.geometry(c["t"], c["x"], c["y"], c["z"])[0]
        lat = G.Lattice(c["t"], c["x"], c["y"], c["z"], c["ng"], REPR[c["repr"]], ipt=ipt)
        u = make_links(c).reshape(lat.V, 4, c["ng"], c["ng"])
        host = torch.empty_like(u)
        host[torch.from_numpy(ipt).long().cuda()] = u
        _live.update(lat=lat, host=host.cpu().numpy())
        del u, host
        lat.set_gauge(_live["host"])
        lat.represent_gauge_field(True)
        if c["csw"]:
            lat.clover_init(c["csw"])
        _live.update(key=key, moved=False)
    elif _live["moved"]:  # a molecular-dynamics step has moved the links: back to the case's own
        _live["lat"].set_gauge(_live["host"])
        _live["lat"].represent_gauge_field(True)
        _live["moved"] = False
    return _live["lat"]


def planes(f):
    """A field's buffer as [parity planes][4 NF][site][re, im]."""
    lat, real = f.lat, torch.float64 if f.prec == G.DOUBLE else torch.float32
    return f.buf.view(real).view(2 if f.par == G.FULL else 1, 4 * lat.nf, -1, 2)


def gaussian(lat, par, prec, gen):
    f = lat.field(par, prec)
    p = planes(f)
    shape = (p.shape[0], p.shape[1], lat.VH, 2)
    p[:, :, : lat.VH].copy_(torch.randn(shape, generator=gen, dtype=torch.float64, device="cuda"))
    return f


def rhmc_shifts(n):
    """The poles of a rational approximation: (M - shift)^-1 with shift = -sigma, sigma log-spaced from 1e-4 to 10."""
    return [0.0] if n == 1 else [-float(10.0 ** (-4 + 5 * k / (n - 1))) for k in range(n)]


MD_DT = 0.02


def prepare(c, seed):
    lat = lattice(c)
    gen = torch.Generator("cuda").manual_seed(seed)
    s = {"case": c, "lat": lat}
    if c["kind"] == "op":
        par = G.FULL if c["call"] in ("Dphi", "g5Dphi_sq", "g5Dphi_flt", "g5Cphi") else G.EVEN
        prec = G.DOUBLE if c["prec"] == 64 else G.FLOAT
        s.update(inp=gaussian(lat, par, prec, gen), out=lat.field(par, prec))
    elif c["kind"] == "cg":
        s.update(inp=gaussian(lat, G.EVEN, G.DOUBLE, gen), out=[lat.field(G.EVEN) for _ in range(c["shifts"])])
    elif c["kind"] == "qmr":
        s.update(inp=gaussian(lat, G.EVEN, G.DOUBLE, gen), out=lat.field(G.EVEN))
    elif c["kind"] == "batch":
        prec = G.DOUBLE if c["prec"] == 64 else G.FLOAT
        s["out"] = [gaussian(lat, G.EVEN, prec, gen) for _ in range(c["nb"])]
        s["inp"], s["res"] = lat.batch(c["nb"], prec, s["out"]), lat.batch(c["nb"], prec)
        for f in s["out"]:
            f.buf.zero_()
    else:
        lat.set_dirac_mass(c["mass"])
        s["seed"] = int(seed)
        s["x"], s["y"], s["eta"] = (gaussian(lat, G.EVEN, G.DOUBLE, gen) for _ in range(3))
        s["X"], s["Y"], s["out"] = lat.field(G.FULL), lat.field(G.FULL), lat.field(G.EVEN)
        for full, even in ((s["X"], s["x"]), (s["Y"], s["y"])):
            full.buf[: even.nbytes].copy_(even.buf)
    return s


def run(s):
    c, lat = s["case"], s["lat"]
    if c["kind"] == "op":
        getattr(lat, c["call"])(c["mass"], s["out"], s["inp"])
        return planes(s["out"])
    if c["kind"] == "cg":
        op = G.OP_G5CPHI_EOPRE_SQ if c["csw"] else G.OP_G5DPHI_EOPRE_SQ
        if c["shifts"] == 1:
            lat.la("zero", s["out"][0])  # the start vector
        _, ok = lat.cg_mshift(op, c["mass"], rhmc_shifts(c["shifts"]), c["err2"], s["inp"], s["out"], flt=c["flt"])
        if not ok:
            raise G.HRGPUError("cg_mshift did not converge")
        return [planes(f) for f in s["out"]]
    if c["kind"] == "qmr":
        lat.la("zero", s["out"])
        _, ok = lat.g5QMR_mshift(G.OP_CPHI_EOPRE if c["csw"] else G.OP_DPHI_EOPRE, c["mass"], [0.0], c["err2"], s["inp"], [s["out"]])
        if not ok:
            raise G.HRGPUError("g5QMR_mshift did not converge")
        return planes(s["out"])
    if c["kind"] == "batch":
        lat.apply_op_batch(G.OP_G5CPHI_EOPRE if c["csw"] else G.OP_G5DPHI_EOPRE, c["mass"], s["res"], s["inp"])
        s["res"].unpack(s["out"])
        return [planes(f) for f in s["out"]]
    # a molecular-dynamics step from fresh momenta, with the pair X, Y of a force solve
    _live["moved"] = True
    lat.random_seed(s["seed"])
    lat.gaussian_momenta()
    lat.fermion_force_begin()
    lat.force_fermion_core(s["X"], s["Y"], 1, MD_DT, 1.0)
    if c["csw"]:
        lat.force_clover_logdet(c["mass"], 2.0)
    lat.fermion_force_end_momenta(MD_DT)
    lat.force0(MD_DT, c["beta"])
    lat.update_gauge_field(MD_DT)
    (lat.g5Cphi_eopre if c["csw"] else lat.g5Dphi_eopre)(c["mass"], s["out"], s["eta"])
    return {"eta": planes(s["out"]), "X": planes(s["X"]), "Y": planes(s["Y"])}


# ------------------------------------------------------------------ bytes, operations, tolerances


def op_cost(c, v, full, size):
    """(bytes, flops) of one D application: fields in and out, the fundamental links and clover blocks once."""
    nf, ng = nf_of(c), c["ng"]
    field = 4 * nf * 2 * size * (v if full else v / 2)
    clov = (2 * (2 * nf + 2 * nf * (2 * nf - 1)) * size * v) if c["csw"] else 0
    mul = 8 * nf if c["repr"] != "adj" else 4 * nf
    flops = v * (8 * 2 * nf * mul + 8 * 24 * nf) + (v * 2 * (2 * nf) ** 2 * 8 if c["csw"] else 0)
    return 2 * field, 4 * ng * ng * 2 * size * v + clov, flops


def work(c):
    v, nf, ng = c["t"] * c["x"] * c["y"] * c["z"], nf_of(c), c["ng"]
    if c["kind"] == "op":
        full = c["call"] in ("Dphi", "g5Dphi_sq", "g5Dphi_flt", "g5Cphi")
        f, g, fl = op_cost(c, v, full, c["prec"] // 8)
        return {"bytes": f + g, "flops": fl * (2 if "_sq" in c["call"] else 1)}
    if c["kind"] in ("cg", "qmr"):
        # an iteration: the links once, the Krylov vectors and solutions read and written once
        size = 4 if c.get("flt") else 8
        f, g, fl = op_cost(c, v, False, size)
        n, twice = c.get("shifts", 1), 2 if c["kind"] == "cg" else 1
        return {"bytes": c["iters"] * (g + f * (2 + 2 * n)), "flops": c["iters"] * twice * fl}
    if c["kind"] == "batch":
        f, g, fl = op_cost(c, v, False, c["prec"] // 8)
        return {"bytes": f * c["nb"] + g, "flops": fl * c["nb"]}
    # links and momenta read and written, X and Y filled, the operator; products of links for staples and clover leaves
    f, g, fl = op_cost(c, v, False, 8)
    fields = 4 * nf * 2 * 8 * v * 2
    links = 4 * ng * ng * 16 * v * 2 + 4 * (ng * ng - 1) * 8 * v * 2
    force = 4 * v * (8 * nf * nf * 4 + 8 * nf * nf * 4) + 4 * v * 12 * 8 * ng**3
    if c["csw"]:
        force += v * 6 * 12 * 8 * ng**3 + 12 * v * 16 * 8 * nf**3
    return {"bytes": links + fields + f + g, "flops": 2 * fl + force}


def tolerance(c):
    if c["kind"] in ("cg", "qmr"):
        # converged to |r| <= sqrt(err2) |b|: solutions differ by that times the condition number (12 seen)
        return {"rel": 100 * math.sqrt(c["err2"])}
    if c["kind"] == "md":  # 3e-16 seen, the matrix exponential and the clover inverse in another order
        return {"rel": 1e-14}
    return {"rel": 2e-15} if c["prec"] == 64 else {"rel": 6e-7}  # 3e-16 and 1.3e-7 seen against 64 bits


# ------------------------------------------------------------------ the same in plain torch, 64 bits

GAMMA = []  # gamma_mu in the chiral basis of the operator, mu = t, x, y, z
for rows in (
    {(0, 2): -1, (1, 3): -1, (2, 0): -1, (3, 1): -1},
    {(0, 3): -1j, (1, 2): -1j, (2, 1): 1j, (3, 0): 1j},
    {(0, 3): -1, (1, 2): 1, (2, 1): 1, (3, 0): -1},
    {(0, 2): -1j, (1, 3): 1j, (2, 0): 1j, (3, 1): -1j},
):
    m = np.zeros((4, 4), complex)
    for k, v in rows.items():
        m[k] = v
    GAMMA.append(m)


def dag(m):
    return m.conj().transpose(-1, -2)


def rep_basis(c):
    """Orthonormal basis matrices of the representation space (symmetric, antisymmetric; T_A sqrt 2 for the adjoint)."""
    ng, e = c["ng"], []
    if c["repr"] == "adj":
        return generators(ng) * math.sqrt(2.0)
    for a in range(ng):
        for b in range(a + (c["repr"] == "sym")):
            m = np.zeros((ng, ng), complex)
            if a == b:
                m[a, a] = 1
            else:
                m[a, b] = math.sqrt(0.5)
                m[b, a] = math.sqrt(0.5) if c["repr"] == "sym" else -math.sqrt(0.5)
            e.append(m)
    return torch.tensor(np.array(e), device="cuda")


def represent(c, u):
    """Links in the representation, antiperiodic in time."""
    if c["repr"] == "fund":
        r = u
    else:
        e = rep_basis(c)
        right = u.conj() if c["repr"] == "adj" else u
        parts = []
        for a in range(e.shape[0]):  # U e_a U^+ (adjoint), U e_a U^T (two-index)
            w = (u @ e[a]) @ right.transpose(-1, -2)
            parts.append(torch.einsum("cij,...ij->...c", e.conj(), w))
        r = torch.stack(parts, -1)
        if c["repr"] == "adj":
            r = r.real + 0j
    sign = torch.ones(c["t"], dtype=torch.float64, device="cuda")
    sign[0] = -1
    head = r[:, :, :, :, :1] * sign.view(-1, 1, 1, 1, 1, 1, 1)
    return torch.cat([head, r[:, :, :, :, 1:]], 4)


class Exact:
    """The Dirac operator on fields [t, x, y, z, spin, colour] in plain torch."""

    def __init__(self, c, u=None):
        self.c, self.nf = c, nf_of(c)
        self.u = make_links(c) if u is None else u
        self.r = represent(c, self.u)
        dims = (c["t"], c["x"], c["y"], c["z"])
        g = torch.meshgrid(*[torch.arange(n, device="cuda") for n in dims], indexing="ij")
        self.par = (sum(g) % 2).view(*dims, 1, 1)
        self.g5 = torch.tensor([1.0, 1, -1, -1], device="cuda", dtype=torch.float64).view(4, 1)
        # device order: t, z, y, x, the sites of one parity in that order
        lex = (((g[0] * c["z"] + g[3]) * c["y"] + g[2]) * c["x"] + g[1]).reshape(-1)
        where = torch.argsort(lex)
        p = self.par.reshape(-1)[where]
        self.sites = [where[p == 0], where[p == 1]]
        self.d = self.di = None
        if c["csw"]:
            self.d = self.clover()

    def load(self, pl):
        """Device planes to a full-lattice field (zero where there is no parity)."""
        out = torch.zeros((self.par.numel(), 4 * self.nf), dtype=torch.complex128, device="cuda")
        z = torch.view_as_complex(pl.double().contiguous())
        for p in range(z.shape[0]):
            out[self.sites[p]] = z[p, :, : self.sites[p].numel()].T
        return out.view(*self.par.shape[:4], 4, self.nf)

    def store(self, psi, parities, ld):
        flat = psi.reshape(-1, 4 * self.nf)
        out = torch.zeros((len(parities), 4 * self.nf, ld), dtype=torch.complex128, device="cuda")
        for k, p in enumerate(parities):
            out[k, :, : self.sites[p].numel()] = flat[self.sites[p]].T
        return torch.view_as_real(out)

    def hop(self, psi):
        acc = torch.zeros_like(psi)
        one = torch.eye(4, dtype=torch.complex128, device="cuda")
        for mu in range(4):
            g = torch.tensor(GAMMA[mu], device="cuda")
            um = self.r[:, :, :, :, mu]
            acc += (one - g) @ (torch.roll(psi, -1, mu) @ um.transpose(-1, -2))
            acc += (one + g) @ torch.roll(psi @ um.conj(), 1, mu)
        return -0.5 * acc

    def plaquette_leaves(self, u, mu, nu):
        """The four leaves around each site in the plane (mu, nu), counter-clockwise, summed."""
        def s(m, a, b):
            return torch.roll(torch.roll(m, -a, mu), -b, nu) if a or b else m

        m, n = u[:, :, :, :, mu], u[:, :, :, :, nu]
        q = m @ s(n, 1, 0) @ dag(s(m, 0, 1)) @ dag(n)
        q = q + n @ dag(s(m, -1, 1)) @ dag(s(n, -1, 0)) @ s(m, -1, 0)
        q = q + dag(s(m, -1, 0)) @ dag(s(n, -1, -1)) @ s(m, -1, -1) @ s(n, 0, -1)
        return q + dag(s(n, 0, -1)) @ s(m, 0, -1) @ s(n, 1, -1) @ dag(m)

    def clover(self):
        """(4+m) + A as two chiral blocks [..., 2, 2NF, 2NF]."""
        k = []
        for mu, nu in ((0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3)):
            q = self.plaquette_leaves(self.r, mu, nu)
            k.append(dag(q) - q)
        w = -self.c["csw"] / 16
        a, b = 1j * k[2], 1j * k[3]
        e, d = 1j * k[0] + k[1], 1j * k[5] - k[4]
        s0, s1, s2, s3 = w * (a - b), w * (e - d), -w * (a + b), -w * (e + d)
        both = [torch.cat([torch.cat([p, q], -1), torch.cat([dag(q), -p], -1)], -2) for p, q in ((s0, s1), (s2, s3))]
        return torch.stack(both, 4) + (4 + self.c["mass"]) * torch.eye(2 * self.nf, dtype=torch.complex128, device="cuda")

    def diag(self, psi, inv=False):
        if self.d is None:
            return psi / (4 + self.c["mass"]) if inv else psi * (4 + self.c["mass"])
        if inv and self.di is None:
            self.di = torch.linalg.inv(self.d)
        v = psi.reshape(*psi.shape[:4], 2, 2 * self.nf, 1)
        return ((self.di if inv else self.d) @ v).reshape(psi.shape)

    def full(self, psi):
        return self.diag(psi) + self.hop(psi)

    def eopre(self, psi):
        """On even fields: D_ee - D_eo D_oo^-1 D_oe with clover, (4+m)^2 - D_eo D_oe without."""
        h = self.hop(psi) * self.par
        if self.d is None:
            return (4 + self.c["mass"]) ** 2 * psi - self.hop(h) * (1 - self.par)
        return (self.diag(psi) - self.hop(self.diag(h, True))) * (1 - self.par)

    def call(self, name, psi):
        d = self.full if name in ("Dphi", "g5Dphi_sq", "g5Dphi_flt", "g5Cphi") else self.eopre
        out = d(psi)
        if name.startswith("g5"):
            out = self.g5 * out
        if "_sq" in name:
            out = self.g5 * d(out)
        return out


def cg_exact(m, b, shifts):
    """Multi-shift CG (zero start) for (m - s) x = b, to the precision of 64 bits."""
    def dot(p, q):
        return torch.vdot(p.reshape(-1), q.reshape(-1)).real.item()

    n = len(shifts)
    x, p = [torch.zeros_like(b) for _ in shifts], [b.clone() for _ in shifts]
    r, k = b.clone(), b.clone()
    rr, bb = dot(b, b), dot(b, b)
    z0, z1, a_old, beta = [1.0] * n, [1.0] * n, 1.0, 0.0
    for _ in range(3000):
        mk = m(k)
        a = rr / dot(k, mk)
        z2 = []
        for i, s in enumerate(shifts):
            z2.append(z1[i] * z0[i] * a_old / (a * beta * (z0[i] - z1[i]) + z0[i] * a_old * (1 - s * a)))
            x[i] += (a * z2[i] / z1[i]) * p[i]
        r -= a * mk
        new = dot(r, r)
        beta = new / rr
        k = r + beta * k
        for i in range(n):
            p[i] = z2[i] * r + (beta * (z2[i] / z1[i]) ** 2) * p[i]
        z0, z1, a_old, rr = z1, z2, a, new
        if rr <= 1e-31 * bb:
            break
    return x


def philox_gauss(nq, stream, seed):
    """nq pairs of Gaussians from Philox4x32-10 blocks (counter q, stream; key seed), Box-Muller."""
    m32 = np.uint64(0xFFFFFFFF)
    q = np.arange(nq, dtype=np.uint64)
    ctr = [q & m32, q >> np.uint64(32), np.full(nq, stream & 0xFFFFFFFF, np.uint64), np.zeros(nq, np.uint64)]
    k = [seed & 0xFFFFFFFF, (seed >> 32) & 0xFFFFFFFF]
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * ctr[0], np.uint64(0xCD9E8D57) * ctr[2]
        ctr = [(p1 >> np.uint64(32)) ^ ctr[1] ^ np.uint64(k[0]), p1 & m32, (p0 >> np.uint64(32)) ^ ctr[3] ^ np.uint64(k[1]), p0 & m32]
        k = [(k[0] + 0x9E3779B9) & 0xFFFFFFFF, (k[1] + 0xBB67AE85) & 0xFFFFFFFF]
    u = [((((a << np.uint64(32)) | b) >> np.uint64(11)).astype(np.float64) + 0.5) * 2.0**-53 for a, b in ((ctr[0], ctr[1]), (ctr[2], ctr[3]))]
    rad = np.sqrt(-2.0 * np.log(u[0]))
    return torch.tensor(np.stack([rad * np.cos(2 * np.pi * u[1]), rad * np.sin(2 * np.pi * u[1])], 1), device="cuda")


def md_exact(c, s):
    """The molecular-dynamics step: forces as derivatives of the action along exp(i eps_A T_A) on each link."""
    lat, t = s["lat"], generators(c["ng"])
    e = Exact(c)
    ld = planes(s["eta"]).shape[2]
    dimg = t.shape[0]
    full = []
    for f in ("x", "y"):
        even = e.load(planes(s[f]))
        odd = e.hop(even) * e.par
        full.append(even + (e.diag(odd, True) if c["csw"] else odd))
    x, y = full
    dims = (c["t"], c["x"], c["y"], c["z"])
    # momenta drawn on the device: [mu][A][site in device order, both parities]
    g = philox_gauss(4 * dimg * ld, 0, s["seed"]).reshape(4, dimg, 2 * ld) * math.sqrt(2.0)
    mom = torch.zeros((e.par.numel(), 4, dimg), dtype=torch.float64, device="cuda")
    for p in range(2):
        n = e.sites[p].numel()
        mom[e.sites[p]] = g[:, :, p * ld : p * ld + n].permute(2, 0, 1)
    mom = mom.view(*dims, 4, dimg)

    def grad(fun):
        eps = torch.zeros((*dims, 4, dimg), dtype=torch.float64, device="cuda", requires_grad=True)
        v = fun(e.u + 1j * torch.einsum("...a,aij->...ij", eps + 0j, t) @ e.u)
        return torch.autograd.grad(v, eps)[0]

    def fermion(u):
        h = Exact.__new__(Exact)
        h.__dict__.update(e.__dict__)
        h.u, h.r = u, represent(c, u)
        w = -h.hop(x)
        if c["csw"]:
            h.d = h.clover()
            w = w + h.diag(x)
        return (y.conj() * (e.g5 * w)).sum().real

    def logdet(u):
        h = Exact.__new__(Exact)
        h.__dict__.update(e.__dict__)
        h.u, h.r = u, represent(c, u)
        return (torch.linalg.slogdet(h.clover())[1].sum(-1) * e.par[..., 0, 0]).sum()

    def plaq(u):
        v = 0
        for mu in range(4):
            for nu in range(mu):
                a, b = u[:, :, :, :, mu], u[:, :, :, :, nu]
                w1, w2 = a @ torch.roll(b, -1, mu), b @ torch.roll(a, -1, nu)
                v = v + (w1 * w2.conj()).sum().real
        return v

    mom = mom + 4 * MD_DT * grad(fermion) + 2 * MD_DT * c["beta"] / c["ng"] * grad(plaq)
    if c["csw"]:
        mom = mom + 4 * MD_DT * grad(logdet)  # two flavours
    unew = torch.linalg.matrix_exp(1j * MD_DT * torch.einsum("...a,aij->...ij", mom + 0j, t)) @ e.u
    h = Exact(c, unew)
    out = h.g5 * h.eopre(h.load(planes(s["eta"])))
    return {"eta": h.store(out, [0], ld), "X": e.store(x, [0, 1], ld), "Y": e.store(y, [0, 1], ld)}


def exact(c, seed):
    s = prepare(c, seed)
    if c["kind"] == "md":
        return md_exact(c, s)
    e = Exact(c)
    if c["kind"] == "op":
        pl = planes(s["inp"])
        out = e.call(c["call"], e.load(pl))
        return e.store(out, range(pl.shape[0]), pl.shape[2])
    if c["kind"] == "batch":
        s["inp"].unpack(s["out"])
        name = "g5Cphi_eopre" if c["csw"] else "g5Dphi_eopre"
        return [e.store(e.call(name, e.load(planes(f))), [0], planes(f).shape[2]) for f in s["out"]]
    pl = planes(s["inp"])
    b, ld = e.load(pl), pl.shape[2]

    def h2(psi):
        return e.call("g5Dphi_eopre_sq", psi)

    if c["kind"] == "cg":
        return [e.store(x, [0], ld) for x in cg_exact(h2, b, rhmc_shifts(c["shifts"]))]
    x = cg_exact(h2, e.g5 * b, [0.0])[0]  # D x = b with D = g5 H: H^2 (H^-1 x) = g5 b, x = H y
    return e.store(e.g5 * e.eopre(x), [0], ld)
