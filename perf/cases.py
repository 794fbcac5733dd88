"""What a user of this library has it do, as measured cases.

Each case is one call (or the short fixed sequence of calls a program makes
together) through the library's public entry points: the improved-staggered
D_eo, the CG solvers, the multi-shift solver, M^-1, the HISQ links with the
fermion force, and a whole RHMC trajectory.  Inputs are synthetic: thin links
exp(i a H) with H random, traceless and Hermitian, staggered phases and the
antiperiodic time boundary folded in, smeared here in torch where a solver
wants fat and long links; sources are Gaussian or points.

exact() restates each operation in torch on complex128 fields: D with rolled
lattices, plain CG to rounding, and the force as the autograd derivative of
the bilinear form through the smearing.
"""
import ctypes
import math
import os

import numpy as np
import torch

import milc_qcd_gb300 as m
from milc_qcd_gb300 import _lib
from milc_qcd_gb300.rhmc import load_rhmc_params, update

RATIONALS = os.path.join(os.path.dirname(m.__file__), "data", "rationals.hisq_2p1p1_ml0.0012_ms0.0363_mc0.432.txt")
PREC = {"double": m.PREC_DOUBLE, "single": m.PREC_SINGLE, "half": m.PREC_HALF}
PARITY = {"even": m.EVEN, "odd": m.ODD, "both": m.EVENANDODD}
CHARM_EPS = -0.117   # Naik epsilon of the charm group


def listed():
    return [
        # the smallest call: one D on the 8^4 lattice of the smallest runs and of every test; launches and latency
        _dslash("dslash_8c8_both", (8, 8, 8, 8), "both"),
        # D on a ragged lattice, odd sites (the odd reconstruction and the force input D_oe X)
        _dslash("dslash_ragged_odd", (14, 10, 18, 22), "odd"),
        # D in FP64 on the lattice of the benchmark
        _dslash("dslash_32c64_even", (32, 32, 32, 64), "even"),
        # the plain asqtad solve of a first run: FP64, one source, host arrays, 8^4, m = 0.05, 1e-8
        dict(_solve("cg_asqtad_8c8_double", (8, 8, 8, 8), 1, "double", 0.05, 1e-8), host=True, action="asqtad"),
        # one source in the cheapest precision (FP16 inner solve), a mid-size lattice, to 1e-12 (at 1e-10 the
        # solution is good to 1e-9, and which of its digits come out right is the 16-bit rounding's chance)
        _solve("cg_24c48_1src_half", (24, 24, 24, 48), 1, "half", 0.01, 1e-12),
        # the production solve: a block of 8 sources, FP32 inner solve, m = 0.01, 1e-10
        _solve("cg_32c64_8src_single", (32, 32, 32, 64), 8, "single", 0.01, 1e-10),
        # a propagator: M^-1 of the three colour point sources, host arrays, a ragged lattice
        dict(_base("propagator_ragged_3col", "propagator", (12, 16, 14, 30)), nsrc=3, prec="single", mass=0.03,
             resid=1e-10),
        # the rational-function solve: 11 offsets log-uniform in [1e-4, 1], to 1e-12 as a force or an action has it
        _shift("multishift_24c48_11off_single", (24, 24, 24, 48), 11, "single", 0.01, 1e-12),
        # one fermion-force evaluation in FP64 on new links: HISQ smearing, then 6 rational-function terms
        _force("links_force_16c32_double", (16, 16, 16, 32), 6, 1, "double"),
        # the same in the FP32 molecular-dynamics setting: ragged lattice, light, strange and charm terms, two Naik groups
        _force("links_force_ragged_single", (12, 14, 10, 20), 20, 2, "single"),
        # molecular dynamics, the production setting (FP32 solves and forces), 2+1+1 flavours
        _trajectory("rhmc_16c32_single", (16, 16, 16, 32), "single", 4),
        # the same all in FP64, what the production setting is checked against
        _trajectory("rhmc_12c24_double", (12, 12, 12, 24), "double", 2),
    ]


def draw(rng):
    kind = rng.choice(["dslash", "dslash", "solve", "solve", "multishift", "propagator", "force", "trajectory"])
    prec = rng.choice(["double", "single", "single"])
    mass = round(math.exp(rng.uniform(math.log(0.01), math.log(0.1))), 4)
    if kind == "dslash":
        c = _dslash("", _dims(rng, 4 ** 4, 2 ** 20), rng.choice(["even", "odd", "both"]))
    elif kind == "solve":
        nsrc = rng.choice([1, 1, 2, 3, 5, 8, 12, 16])
        if nsrc == 1:
            prec = rng.choice(["double", "single", "half"])
        top = 400000 if prec != "double" else 150000
        c = _solve("", _dims(rng, 4096, max(20000, top // nsrc)), nsrc, prec, mass,
                   1e-12 if prec == "half" else rng.choice([1e-8, 1e-9, 1e-10]))
    elif kind == "multishift":
        c = _shift("", _dims(rng, 4096, 300000 if prec != "double" else 100000), rng.randint(3, 16), prec, mass, 1e-12)
    elif kind == "propagator":
        c = dict(_base("", "propagator", _dims(rng, 4096, 60000)), nsrc=3, prec=prec, mass=max(mass, 0.02), resid=1e-10)
    elif kind == "force":
        c = _force("", _dims(rng, 4096, 100000), rng.randint(3, 24), rng.choice([1, 2]), rng.choice(["double", "single"]))
    else:
        prec = rng.choice(["double", "single"])
        c = _trajectory("", _dims(rng, 4096, 30000 if prec == "double" else 60000), prec, 2)
    del c["name"]
    return c


def _dims(rng, vmin, vmax):
    """Even extents of at least 4, ragged, the volume spread over its logarithm."""
    while True:
        v = math.exp(rng.uniform(math.log(vmin), math.log(vmax)))
        side = (v / 2) ** 0.25
        d = [2 * max(2, round(0.5 * side * rng.uniform(0.75, 1.3))) for _ in range(3)]
        d.append(2 * max(2, round(side * rng.uniform(0.75, 1.3))))
        if vmin <= math.prod(d) <= vmax:
            return tuple(d)


def _base(name, kind, dims):
    return dict(name=name, kind=kind, nx=dims[0], ny=dims[1], nz=dims[2], nt=dims[3])


def _dslash(name, dims, parity):
    return dict(_base(name, "dslash", dims), parity=parity)


def _solve(name, dims, nsrc, prec, mass, resid):
    return dict(_base(name, "solve", dims), nsrc=nsrc, prec=prec, mass=mass, resid=resid)


def _shift(name, dims, noff, prec, mass, resid):
    return dict(_base(name, "multishift", dims), noff=noff, prec=prec, mass=mass, resid=resid)


def _force(name, dims, terms, groups, prec):
    return dict(_base(name, "force", dims), terms=terms, groups=groups, prec=prec)


def _trajectory(name, dims, prec, steps):
    return dict(_base(name, "trajectory", dims), prec=prec, steps=steps)


def _geometry(case):
    return (case["nx"], case["ny"], case["nz"], case["nt"])


# ------------------------------------------------------------------ torch fields
# Lattice fields in torch: complex128, colour indices first, then (t, z, y, x).

def _grid(dims):
    return (dims[3], dims[2], dims[1], dims[0])


def _order(dims):
    """Lexicographic index of every site in MILC's order (even sites first)."""
    t, z, y, x = torch.meshgrid(*[torch.arange(n, device="cuda") for n in _grid(dims)], indexing="ij")
    odd = ((x + y + z + t) & 1).reshape(-1)
    return torch.cat([torch.nonzero(odd == 0)[:, 0], torch.nonzero(odd == 1)[:, 0]])


def _to_sites(field, dims):
    """(colour..., t, z, y, x) -> (site, colour...) in MILC's order."""
    k = field.dim() - 4
    flat = field.reshape(*field.shape[:k], -1)
    return flat.permute(k, *range(k))[_order(dims)].contiguous()


def _from_sites(sites, dims):
    out = torch.empty_like(sites)
    out[_order(dims)] = sites
    k = sites.dim() - 1
    return out.permute(*range(1, k + 1), 0).reshape(*sites.shape[1:], *_grid(dims)).contiguous()


def _links_out(links, dims):
    """Four (3, 3, t, z, y, x) fields -> MILC's su3_matrix[4 i + dir], float64 (V, 4, 18)."""
    return torch.view_as_real(torch.stack([_to_sites(u, dims) for u in links], 1)).reshape(-1, 4, 18).contiguous()


def _vector_out(v, dims):
    return torch.view_as_real(_to_sites(v, dims)).reshape(-1, 6).contiguous()


def _vector_in(sites, dims):
    return _from_sites(torch.view_as_complex(sites.reshape(-1, 3, 2).contiguous()), dims)


def _sh(a, mu, k):
    """a(x + k mu)"""
    return torch.roll(a, -k, -1 - mu)


def _adj(a):
    return a.transpose(0, 1).conj()


def _mm(a, b):
    return (a[:, :, None] * b[None]).sum(1)


def _mv(a, v):
    return (a * v[None]).sum(1)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)


def _normal(shape, gen):
    return torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64) * math.sqrt(0.5)


def _complex_normal(shape, gen):
    return torch.complex(_normal(shape, gen), _normal(shape, gen))


def _thin(dims, gen, a):
    """exp(i a H), H random, traceless and Hermitian, without phases."""
    one = torch.eye(3, dtype=torch.complex128, device="cuda").reshape(3, 3, 1, 1, 1, 1)
    links = []
    for _ in range(4):
        h = _complex_normal((3, 3) + _grid(dims), gen)
        h = 0.5 * (h + _adj(h))
        h = 1j * a * (h - one * (h[0, 0] + h[1, 1] + h[2, 2]) / 3)
        u = one + h / 16
        for k in range(15, 0, -1):
            u = one + _mm(h, u) / k
        links.append(u)
    return links


def _phased(links, dims):
    """MILC's staggered phases and the antiperiodic time boundary."""
    t, z, y, x = torch.meshgrid(*[torch.arange(n, device="cuda") for n in _grid(dims)], indexing="ij")
    signs = [1 - 2 * (t & 1), 1 - 2 * ((t + x) & 1), 1 - 2 * ((t + x + y) & 1), 1 - 2 * (t == dims[3] - 1).long()]
    return [u * s for u, s in zip(links, signs)]


def _staple(U, mu, nu, A):
    up = _mm(U[nu], _mm(_sh(A, nu, 1), _adj(_sh(U[nu], mu, 1))))
    return up + _sh(_mm(_mm(_adj(U[nu]), A), _sh(U[nu], mu, 1)), nu, -1)


def _fatten(U, one, c3, c5, c7, lepage):
    out = []
    for mu in range(4):
        f = (one - 6 * lepage) * U[mu]
        for nu in range(4):
            if nu == mu:
                continue
            s = _staple(U, mu, nu, U[mu])
            f = f + c3 * s
            if lepage:
                f = f + lepage * _staple(U, mu, nu, s)
            for rho in range(4):
                if rho in (mu, nu):
                    continue
                q = _staple(U, mu, rho, s)
                f = f + c5 * q
                sig = 6 - mu - nu - rho
                f = f + c7 * _staple(U, mu, sig, q)
        out.append(f)
    return out


def _naik(U, c):
    return [c * _mm(u, _mm(_sh(u, mu, 1), _sh(u, mu, 2))) for mu, u in enumerate(U)]


def _project(V):
    """V (V^dag V)^(-1/2) by Newton's iteration (the fat links' singular values are below sqrt 3)."""
    one = torch.eye(3, dtype=torch.complex128, device="cuda").reshape(3, 3, 1, 1, 1, 1)
    out = []
    for w in V:
        for _ in range(11):
            w = 0.5 * _mm(w, 3 * one - _mm(_adj(w), w))
        out.append(w)
    return out


def _hisq(U, eps=(0.0,)):
    """Fat and long links of every Naik group from phased thin links."""
    W = _project(_fatten(U, 1 / 8, -1 / 16, 1 / 64, -1 / 384, 0.0))
    fat = _fatten(W, 1.0, -1 / 16, 1 / 64, -1 / 384, -1 / 8)
    lng = _naik(W, -1 / 24)
    return [([f + e / 8 * w for f, w in zip(fat, W)], [(1 + e) * q for q in lng]) for e in eps]


def _asqtad(U):
    return _fatten(U, 5 / 8, -1 / 16, 1 / 64, -1 / 384, -1 / 16), _naik(U, -1 / 24)


def _apply_d(fat, lng, v):
    out = 0
    for mu in range(4):
        for U, k in ((fat[mu], 1), (lng[mu], 3)):
            out = out + _mv(U, _sh(v, mu, k)) - _sh(_mv(_adj(U), v), mu, -k)
    return out


def _smeared(case, seed):
    dims = _geometry(case)
    U = _phased(_thin(dims, _generator(seed), 0.3), dims)
    return _asqtad(U) if case.get("action") == "asqtad" else _hisq(U)[0]


def _gaussian_sources(case, seed, n):
    """n even-site sources (V, 6)."""
    dims, gen = _geometry(case), _generator(seed + 1000003)
    V = math.prod(dims)
    out = []
    for _ in range(n):
        b = torch.zeros((V, 6), dtype=torch.float64, device="cuda")
        b[:V // 2] = _normal((V // 2, 6), gen)
        out.append(b)
    return out


def _full_source(case, seed):
    return _normal((math.prod(_geometry(case)), 6), _generator(seed + 2000003))


def _point_sources(case, seed):
    """The three colour sources at one site of the source time slice."""
    V = math.prod(_geometry(case))
    site = int(np.random.default_rng(seed).integers(0, V))
    out = []
    for c in range(case["nsrc"]):
        b = np.zeros((V, 6))
        b[site, 2 * (c % 3)] = 1.0
        out.append(b)
    return out


def _offsets(case):
    return 4 * case["mass"] ** 2 + np.logspace(-4, 0, case["noff"])


# ------------------------------------------------------------------ states
class State:
    """Inputs in hand, and for the solvers a link slot of the library."""
    free = list(range(_lib.MKS_MAX_SLOTS))
    dims = None          # the lattice that the library is set to
    generation = 0       # counts the changes of lattice, which drop every slot

    def __init__(self, case):
        self.case, self.dims, self.slot = case, _geometry(case), None

    def use(self):
        """Set the lattice; load this state's links into its slot unless they are there."""
        if State.dims != self.dims:
            m.set_lattice(self.dims)
            State.dims = self.dims
            State.generation += 1
        if self.slot is not None and self.loaded != State.generation:
            m.check(m.init().mks_load_fn_links_dev(self.slot, self.fat.data_ptr(), self.lng.data_ptr(), 0.0),
                    "mks_load_fn_links_dev")
            self.loaded = State.generation

    def links(self, fat, lng):
        self.fat, self.lng = _links_out(fat, self.dims), _links_out(lng, self.dims)
        torch.cuda.synchronize()
        self.slot, self.loaded = State.free.pop(0), -1

    def __del__(self):
        if getattr(self, "slot", None) is not None:
            State.free.append(self.slot)


def _pinned(t):
    """Page-locked host copy, as MILC's arrays are when the library allocates them."""
    return torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t).numpy()


def _addresses(ts):
    return (ctypes.c_void_p * len(ts))(*[t.data_ptr() for t in ts])


def prepare(case, seed):
    m.init(0)
    kind, s = case["kind"], State(case)
    V = math.prod(s.dims)
    if kind in ("dslash", "solve", "multishift", "propagator"):
        s.links(*_smeared(case, seed))
    if kind == "dslash":
        s.src = _full_source(case, seed)
        s.out = torch.zeros_like(s.src)
    elif kind == "solve":
        s.src = _gaussian_sources(case, seed, case["nsrc"])
        if case.get("host"):
            s.src = [b.cpu().numpy() for b in s.src]
        else:
            s.out = [torch.zeros_like(b) for b in s.src]
    elif kind == "multishift":
        s.src = _gaussian_sources(case, seed, 1)[0]
        s.offsets = _offsets(case)
        s.out = [torch.zeros_like(s.src) for _ in s.offsets]
    elif kind == "propagator":
        s.src = _point_sources(case, seed)
    elif kind == "force":
        s.thin, s.xxx, s.residues, s.mom, s.orders, s.eps = _force_inputs(case, seed)
        s.thin = _pinned(_links_out(s.thin, s.dims))
        s.xxx = [_pinned(x) for x in s.xxx]
        s.mom = _pinned(s.mom)
    elif kind == "trajectory":
        s.thin = _pinned(_links_out(_thin(s.dims, _generator(seed), 0.2), s.dims))
        s.mom = np.zeros((V, 4, 10))
        s.pf = load_rhmc_params(RATIONALS)
        s.seed = int(seed) % 1000003 + 1
    s.use()
    torch.cuda.synchronize()
    return s


def _force_inputs(case, seed):
    dims, gen = _geometry(case), _generator(seed)
    V, n = math.prod(dims), case["terms"]
    U = _phased(_thin(dims, gen, 0.3), dims)
    xxx = [_normal((V, 6), gen) for _ in range(n)]
    mom = torch.zeros((V, 4, 10), dtype=torch.float64, device="cuda")
    mom[..., :6] = _normal((V, 4, 6), gen)
    d = _normal((V, 4, 2), gen)
    mom[..., 6], mom[..., 7] = d[..., 0] + d[..., 1] / math.sqrt(3), -d[..., 0] + d[..., 1] / math.sqrt(3)
    mom[..., 8] = -2 * d[..., 1] / math.sqrt(3)
    residues = np.sort(np.random.default_rng(seed).uniform(0.1, 1.0, n))
    orders = [n] if case["groups"] == 1 else [n - n // 4, n // 4]
    return U, xxx, residues, mom, orders, (0.0, CHARM_EPS)[:case["groups"]]


FORCE_EPS = 0.02


def run(s):
    case, kind, lib = s.case, s.case["kind"], m.init()
    s.use()
    if kind == "dslash":
        m.check(lib.mks_dslash_fn_field_dev(s.src.data_ptr(), s.out.data_ptr(), PARITY[case["parity"]], s.slot),
                "mks_dslash_fn_field_dev")
        return s.out
    if kind == "solve" and case.get("host"):
        qic = m.QuarkInvertControl(resid=case["resid"], max=1000, nrestart=5, parity=m.EVEN, prec=PREC[case["prec"]])
        out = [np.zeros_like(b) for b in s.src]
        for b, x in zip(s.src, out):
            m.ks_congrad_parity(b, x, qic, case["mass"], s.slot)
        return out
    if kind == "solve":
        n = len(s.src)
        with torch.cuda.stream(torch.cuda.ExternalStream(lib.mks_stream())):   # zero initial guesses
            for x in s.out:
                x.zero_()
        arg = _lib.InvertArg(1000, 10, m.EVEN, PREC[case["prec"]], case["resid"], 0.0, 0.1)
        res = (_lib.InvertResult * n)()
        m.check(lib.mks_ks_congrad_block_parity_dev(n, _addresses(s.src), _addresses(s.out), case["mass"], s.slot,
                                                    ctypes.byref(arg), res), "mks_ks_congrad_block_parity_dev")
        return s.out
    if kind == "multishift":
        arg = _lib.InvertArg(1000, 10, m.EVEN, PREC[case["prec"]], case["resid"], 0.0, 0.1)
        res = (_lib.InvertResult * len(s.out))()
        m.check(lib.mks_ks_multicg_offset_field_dev(s.src.data_ptr(), _addresses(s.out),
                                                    s.offsets.ctypes.data_as(_lib.DP), len(s.out), s.slot,
                                                    ctypes.byref(arg), res), "mks_ks_multicg_offset_field_dev")
        return s.out
    if kind == "propagator":
        qic = m.QuarkInvertControl(resid=case["resid"], max=1000, nrestart=5, prec=PREC[case["prec"]])
        out = [np.zeros_like(b) for b in s.src]
        m.mat_invert_block_uml(s.src, out, qic, case["mass"], s.slot)
        return out
    # The links of a force or a trajectory are the library's resident ones, which replace the solvers' slots
    # 0 and 1: a program that solves afterwards loads its own again.
    State.generation += 1
    single = case["prec"] == "single"
    if kind == "force":
        mom = s.mom.copy()
        m.md_precision(PREC[case["prec"]])
        m.load_hisq_links(s.thin, s.eps)
        m.eo_fermion_force_multi(FORCE_EPS, s.residues, s.xxx, mom, n_orders_naik=s.orders, n_naiks=len(s.eps))
        m.md_precision(m.PREC_DOUBLE)
        # a force of the FP32 setting is worth 32 bits (MILC's single-precision build keeps its momenta so)
        return mom.astype(np.float32) if single else mom
    m.gauge_load(s.thin)
    m.mom_load(s.mom)
    m.rng_seed(s.seed)
    p, n = PREC[case["prec"]], len(s.pf)
    r = update(s.pf, 6.3, 0.86, 4, 0.05, case["steps"], "leapfrog", [1e-6] * n, [1e-10] * n, [1e-10] * n, 5000, p, p, p,
               5, True, prec_force=p)
    links, mom = m.gauge_get(), m.mom_get()
    if single:   # MILC's configuration files hold 32-bit links
        return [links.astype(np.float32), mom.astype(np.float32)]
    return [links, mom, list(r["start"]) + list(r["end"])]


# ------------------------------------------------------------------ bytes and operations
def _iterations(case):
    """CG iterations that these links take (spectrum of M^dag M from about 4 m^2 + 0.04 to 22)."""
    return 0.5 * math.log(2 / case["resid"]) * math.sqrt(22 / (4 * case["mass"] ** 2 + 0.04))


def work(case):
    V = math.prod(_geometry(case))
    kind, size = case["kind"], {"double": 16, "single": 8, "half": 4}.get(case.get("prec"), 16)
    if kind == "dslash":
        half = 2 if case["parity"] == "both" else 1
        return {"bytes": V * 8 * 144 + half * V * 48.0, "flops": 1146.0 * V / 2 * half}
    if kind in ("solve", "propagator"):
        # each iteration: the links in either D, the vectors of D (2 in, 2 out) and of the update (4 in, 3 out)
        n = case["nsrc"] * (2 if kind == "propagator" else 1)
        it = _iterations(case) * (1.2 if kind == "propagator" else 1)
        links, vector = V / 2 * 16 * 9 * size, V / 2 * 3 * max(size, 8)
        return {"bytes": it * (2 * links + 11 * n * vector), "flops": it * n * 1187.0 * V}
    if kind == "multishift":
        it = _iterations(case)
        links, vector = V / 2 * 16 * 9 * size, V / 2 * 3 * size
        return {"bytes": it * (2 * links + (8 + 2 * case["noff"]) * vector), "flops": it * 1187.0 * V}
    if kind == "force":
        # thin links, the solutions and the momenta; two levels of smearing (60 staples each) and their reverse
        size = 8 if case["prec"] == "single" else 16
        return {"bytes": V * (4 * 144.0 + case["terms"] * 48 + 4 * 160), "flops": V * (2 * 60 * 4 + 2 * 60 * 12) * 198.0}
    # a trajectory: per step one force on new links, a gauge force (48 staple paths, about 180 products per link)
    # and the three fields' solves (about 100 iterations each)
    it = 300.0 * (case["steps"] + 2)
    links, vector = V / 2 * 16 * 9 * size, V / 2 * 3 * size
    return {"bytes": it * (2 * links + 20 * vector),
            "flops": case["steps"] * V * (960 + 960 + 720) * 198.0 + it * 1187.0 * V}


# ------------------------------------------------------------------ the same in 64 bits
def _even_mask(dims):
    t, z, y, x = torch.meshgrid(*[torch.arange(n, device="cuda") for n in _grid(dims)], indexing="ij")
    return ((x + y + z + t) & 1) == 0


def _cg(fat, lng, sigma, b):
    """(sigma - D D)^-1 b to rounding."""
    norm = float((b.abs() ** 2).sum())
    x, r = torch.zeros_like(b), b.clone()
    p, rr = r.clone(), norm
    for k in range(4000):
        if rr <= 1e-28 * norm:
            break
        ap = sigma * p - _apply_d(fat, lng, _apply_d(fat, lng, p))
        a = rr / float((p.conj() * ap).real.sum())
        x = x + a * p
        r = r - a * ap if k % 50 != 49 else b - (sigma * x - _apply_d(fat, lng, _apply_d(fat, lng, x)))
        new = float((r.abs() ** 2).sum())
        p, rr = r + (new / rr) * p, new
    return x


def exact(case, seed):
    kind, dims = case["kind"], _geometry(case)
    if kind == "trajectory":
        return None
    if kind == "force":
        return _exact_force(case, seed)
    fat, lng = _smeared(case, seed)
    if kind == "dslash":
        out = _vector_out(_apply_d(fat, lng, _vector_in(_full_source(case, seed), dims)), dims)
        V = out.shape[0]
        if case["parity"] == "even":
            out[V // 2:] = 0
        elif case["parity"] == "odd":
            out[:V // 2] = 0
        return out
    if kind == "solve":
        src = _gaussian_sources(case, seed, case["nsrc"])
        most = 2 if math.prod(dims) > 2 ** 20 else 8   # the others take as long again
        return [_vector_out(_cg(fat, lng, 4 * case["mass"] ** 2, _vector_in(b, dims)), dims) if k < most else None
                for k, b in enumerate(src)]
    if kind == "multishift":
        b = _vector_in(_gaussian_sources(case, seed, 1)[0], dims)
        return [_vector_out(_cg(fat, lng, float(sig), b), dims) for sig in _offsets(case)]
    out = []
    for b in _point_sources(case, seed):   # M^-1 = M^dag (M^dag M)^-1
        v = _vector_in(torch.from_numpy(b).cuda(), dims)
        y = _cg(fat, lng, 4 * case["mass"] ** 2, v)
        out.append(_vector_out(2 * case["mass"] * y - _apply_d(fat, lng, y), dims))
    return out


def _exact_force(case, seed):
    """mom + 2 eps TA(U K), K the derivative of 2 Re sum_j r_j X_j^dag D Y_j through the smearing."""
    dims = _geometry(case)
    U, xxx, residues, mom, orders, eps = _force_inputs(case, seed)
    U = [u.detach().requires_grad_(True) for u in U]
    even = _even_mask(dims)
    S, j = 0, 0
    for (fat, lng), order in zip(_hisq(U, eps), orders if len(eps) == len(orders) else [len(xxx)]):
        # X^dag D Y is linear in the links: the terms of a group share one contraction with each link
        for mu in range(4):
            for links, k in ((fat[mu], 1), (lng[mu], 3)):
                K = 0
                for i in range(j, j + order):
                    v = _vector_in(xxx[i], dims)
                    K = K + float(residues[i]) * _sh(v, mu, k)[:, None] * v.conj()[None]
                K = torch.where(even, K, -K)
                S = S + 2 * (links * K.transpose(0, 1)).sum().real
        j += order
    S.backward()
    out = mom.clone()
    for mu in range(4):
        A = 2 * FORCE_EPS * _mm(U[mu].detach(), _adj(U[mu].grad) / 2)
        A = _to_sites(0.5 * (A - _adj(A)), dims)
        tr = (A[:, 0, 0] + A[:, 1, 1] + A[:, 2, 2]).imag / 3
        for n, (a, b) in enumerate(((0, 1), (0, 2), (1, 2))):
            out[:, mu, 2 * n] += A[:, a, b].real
            out[:, mu, 2 * n + 1] += A[:, a, b].imag
        for a in range(3):
            out[:, mu, 6 + a] += A[:, a, a].imag - tr
    return out
