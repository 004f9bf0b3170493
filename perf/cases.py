"""Cases of the Car-Parrinello step by which its speed is measured.

Each case is work that a program using this package has it do: native CP
steps (``CPDriver.run_native``), the batching form (``run_batch``), the force
half of a step (``CPDriver.forces``), the constraint and orthonormalisation
half (the PairCalculator / Ortho entry points of ``CPContext``) and the
electronic minimiser (``CPMinimizer``).  Systems are liquid-density water
boxes of 2 to 128 molecules at 20 to 85 Ry on the smallest 2-3-5 grid that
holds the density sphere, four states per molecule (or a few fewer), in the
FP64 and the mixed form, with structure-factor or EES nonlocal forces,
PZ-LDA or BLYP, fixed or moving atoms.

Every pass restarts from the coefficients in hand (bond and lone-pair
Gaussians, Loewdin-orthonormalised), as a run does from a state file, so a
pass gives the same results however often it is repeated.
"""
import dataclasses
import functools
import math

import numpy as np
import torch

from openatom_b200 import ees as ees_mod
from openatom_b200.gpu import CPDriver, CPMinimizer, run_batch
from openatom_b200.system import atom_masses, make_system

TERMS = ("EKE", "EHART", "EEXT", "EEXC", "ENL", "EGGA", "EWALD_RECIP", "MUXC", "FICT_KE")
NORB_TOL = 0.003
NOISE = 0.1     # random part of the starting coefficients, over 1 + g^2


def _smooth(n):
    """Smallest 2^a 3^b 5^c >= n."""
    while True:
        m = n
        for p in (2, 3, 5):
            while m % p == 0:
                m //= p
        if m == 1:
            return n
        n += 1


def _box(nmol):
    """Cubic cell edge (bohr) of nmol waters at the density of 32 in 18.6 bohr."""
    return 18.6 * (nmol / 32.0) ** (1.0 / 3.0)


def _kmax(nmol, ecut):
    return int(math.floor(math.sqrt(ecut) * _box(nmol) / (2.0 * math.pi))) + 1


def _grid(nmol, ecut):
    return _smooth(4 * _kmax(nmol, ecut))


def _case(name, kind, nmol, ecut, precision, nstate=None, steps=1, nl="sf", order=6, xc="pz_lda", ions=False,
          eext=0, nsys=1, grid=None):
    c = dict(kind=kind, nmol=nmol, ecut=ecut, grid=grid or _grid(nmol, ecut), precision=precision,
             nstate=nstate or 4 * nmol, steps=steps, nl=nl, order=order, xc=xc, ions=ions, eext=eext, nsys=nsys)
    return dict(c, name=name) if name else c


def listed():
    return [
        # force half of a step on the smallest system of the tests: launch latency
        _case("force_w2_fp64", "force", 2, 20.0, "fp64", grid=24),
        # 20 CPMD steps of 8 waters, the precision-run system, mixed form
        _case("run_w8_mixed", "run", 8, 70.0, "mixed", steps=20, grid=64),
        # CG minimisation of the same system to prepare a ground state, FP64
        _case("minimize_w8_fp64", "minimize", 8, 70.0, "fp64", steps=5, grid=64),
        # replicas of uneven sizes advanced together (path-integral beads, tempering)
        _case("batch_6x_w8_w14_mixed", "batch", 8, 70.0, "mixed", steps=8, nsys=6),
        # an ordinary size off the tuned grids, odd state count: the force half
        _case("force_w13_odd_mixed", "force", 13, 70.0, "mixed", nstate=51),
        # moving atoms: EES local path and structure-factor nonlocal forces
        _case("run_w16_ions_mixed", "run", 16, 70.0, "mixed", steps=5, ions=True, eext=6),
        # gradient-corrected functional
        _case("run_w20_blyp_mixed", "run", 20, 80.0, "mixed", steps=5, xc="blyp"),
        # the headline system: 32 waters, 128 states, 108^3, both forms
        _case("run_w32_mixed", "run", 32, 80.0, "mixed", steps=10),
        _case("run_w32_fp64", "run", 32, 80.0, "fp64", steps=5),
        # constraint and orthonormalisation half at an odd count above the cluster kernel's
        _case("ortho_w50_odd_fp64", "ortho", 50, 70.0, "fp64", nstate=199),
        # FP64 forces of a larger box on a general 2-3-5 grid
        _case("force_w64_fp64", "force", 64, 60.0, "fp64"),
        # the large system: 128 waters, 512 states, 160^3, EES nonlocal forces
        _case("run_w128_ees_mixed", "run", 128, 70.0, "mixed", steps=2, nl="ees", order=4, grid=160),
    ]


def draw(rng):
    kind = rng.choice(["run", "run", "run", "force", "force", "ortho", "minimize", "batch"])
    precision = rng.choice(["mixed", "mixed", "fp64"])
    top = {"run": 72, "force": 96, "ortho": 110, "minimize": 40, "batch": 14}[kind]
    low = 6 if kind == "batch" else 2
    nmol = int(round(math.exp(rng.uniform(math.log(low), math.log(top)))))
    ecut = rng.uniform(60.0, 85.0) if nmol >= 8 else rng.uniform(25.0, 85.0)
    ecut = round(ecut * 2.0) / 2.0
    nstate = 4 * nmol
    if kind in ("force", "ortho", "minimize") and rng.random() < 0.5:
        nstate -= rng.randint(1, 3)
    nl, order = ("ees", rng.choice([4, 6])) if rng.random() < 0.35 else ("sf", 6)
    xc = "blyp" if kind in ("run", "force") and rng.random() < 0.25 else "pz_lda"
    ions = kind == "run" and nmol <= 48 and rng.random() < 0.25
    eext = 6 if ions and rng.random() < 0.5 else 0
    steps = {"run": 10 if nmol < 24 else 4 if nmol < 48 else 2, "minimize": 4, "batch": 6}.get(kind, 1)
    return _case(None, kind, nmol, ecut, precision, nstate, steps, nl, order, xc, ions, eext,
                 nsys=rng.randint(3, 6) if kind == "batch" else 1)


# ----------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------

@functools.lru_cache(maxsize=8)
def _base(nmol, ecut, grid, nstate, xc):
    """Cell, g-sphere and pseudopotential tables, which no seed changes."""
    s = make_system("w2", seed=1, nstate=1, nmol=1, box=_box(nmol), ecut_ry=ecut, nfft=(grid,) * 3, ecut_mass=2.0,
                    cmass0=400.0, dt=5.0, xc=xc)
    typ = np.tile(np.array([0, 1, 1], dtype=np.int32), nmol)
    return dataclasses.replace(s, name="water", nstate=nstate, atm_type=typ, q=np.where(typ == 0, 6.0, 1.0),
                               occ=np.ones(nstate), psi=None)


def _waters(nmol, box, rng):
    """Rigid waters of random orientation on a jittered lattice: positions
    [3 nmol, 3] (O H H ...) and the four bond / lone-pair centres of each."""
    m = int(math.ceil(nmol ** (1.0 / 3.0) - 1e-9))
    site = rng.permutation(m ** 3)[:nmol]
    o = (np.stack([site % m, site // m % m, site // (m * m)], 1) + 0.5) * (box / m)
    o = o + rng.uniform(-0.3, 0.3, o.shape)
    q, r = np.linalg.qr(rng.standard_normal((nmol, 3, 3)))
    ex, ey, ez = q[:, :, 0], q[:, :, 1], q[:, :, 2]
    ang = 1.0 / 0.529177210903
    a = math.radians(104.5) / 2.0
    h = [o + 0.96 * ang * (sg * math.sin(a) * ex + math.cos(a) * ez) for sg in (1.0, -1.0)]
    lone = [o + 0.55 * (sg * 0.82 * ey - 0.58 * ez) for sg in (1.0, -1.0)]
    pos = np.stack([o, h[0], h[1]], 1).reshape(-1, 3)
    centre = np.stack([o + 0.5 * (h[0] - o), o + 0.5 * (h[1] - o)] + lone, 1).reshape(-1, 3)
    return pos, centre


def _kx0_partner(s):
    key = {(int(s.ky[i]), int(s.kz[i])): i for i in range(s.nkx0)}
    return np.array([key[(-int(s.ky[i]), -int(s.kz[i]))] for i in range(s.nkx0_red)], dtype=np.int64)


def _start(s, centre, rng, dev):
    """Gaussians of slightly uneven width on the centres with a small random
    part (it gives the sharper components that the oxygen projector sees),
    Loewdin-orthonormalised to S = 2 I."""
    f = 2.0 * math.pi / s.box
    t = functools.partial(torch.as_tensor, device=dev, dtype=torch.float64)
    k = f * torch.stack([t(s.kx), t(s.ky), t(s.kz)])
    g2 = (k * k).sum(0)
    sig = t(rng.uniform(0.8, 1.0, s.nstate))
    c = torch.polar(torch.exp(-0.5 * sig[:, None] ** 2 * g2), t(centre[:s.nstate]) @ k)
    gen = torch.Generator(device=dev).manual_seed(int(rng.integers(1 << 40)))
    c += torch.randn(c.shape, generator=gen, dtype=c.dtype, device=dev) * (NOISE / (1.0 + g2))
    c[:, g2 == 0] = c[:, g2 == 0].real.to(c.dtype)
    c[:, :s.nkx0_red] = c[:, torch.as_tensor(_kx0_partner(s), device=dev)].conj()
    w = torch.where(t(s.kx) == 0, 1.0, 2.0).repeat_interleave(2)
    rv = torch.view_as_real(c).reshape(s.nstate, -1)
    e, u = torch.linalg.eigh((rv * w) @ rv.T / 2.0)
    rv = ((u / e.sqrt()) @ u.T) @ rv
    return torch.view_as_complex(rv.reshape(s.nstate, -1, 2).contiguous())


def _inputs(case, seed, dev):
    """System and starting coefficients of one case from the seed alone."""
    rng = np.random.default_rng([seed, 77])
    base = _base(case["nmol"], case["ecut"], case["grid"], case["nstate"], case["xc"])
    pos, centre = _waters(case["nmol"], base.box, rng)
    s = dataclasses.replace(base, seed=seed, pos=pos)
    if case["eext"]:
        s.eext_ees = ees_mod.local_grid(s, 1.2, case["eext"]) + (case["eext"],)
    return s, _start(s, centre, rng, dev), rng


def _members(case, seed):
    """The systems of a batch: uneven sizes up to twice the first one's."""
    rng = np.random.default_rng([seed, 5])
    top = max(case["nmol"] + 1, case["nmol"] * 7 // 4)
    out = []
    # sizes from the case alone, inputs from the seed
    sizes = np.linspace(case["nmol"], top, case["nsys"]).round().astype(int)
    for i, n in enumerate(sizes):
        e = case["ecut"] - 5.0 * (i % 3)
        out.append((dict(case, nmol=int(n), ecut=e, nstate=4 * int(n), grid=_grid(int(n), e)),
                    int(rng.integers(1 << 30))))
    return out


def _driver(case, seed):
    s, psi, rng = _inputs(case, seed, "cuda")
    d = CPDriver(s, case["precision"], psi0=psi.cpu().numpy(), norb_tol=NORB_TOL, nl_method=case["nl"],
                 ees_order=case["order"])
    return s, d, psi, rng


def _thermal(s, rng):
    m = atom_masses(s)
    return m, rng.standard_normal(s.pos.shape) * np.sqrt(300.0 * 3.1668115634556e-6 / m)[:, None]


def prepare(case, seed):
    if case["kind"] == "batch":
        parts = [_driver(c, sd) for c, sd in _members(case, seed)]
        ds = [p[1] for p in parts]
        return dict(case=case, drivers=ds, psi0=[p[2] for p in parts], states=[d.native_state() for d in ds])
    s, d, psi, rng = _driver(case, seed)
    st = dict(case=case, sys=s, driver=d, psi0=psi)
    if case["kind"] == "run":
        if case["ions"]:
            st["masses"], st["vel"] = _thermal(s, rng)
            d.ctx.set_ions(st["masses"], st["vel"])
        st["state"] = d.native_state()
    elif case["kind"] == "minimize":
        st["minimizer"] = CPMinimizer(d, "cg")
    elif case["kind"] == "ortho":
        st.update(_ortho_inputs(s, psi, rng))
        st["v"], st["psi_t"] = st["v0"].clone(), st["psi_t0"].clone()
        st["mats"] = [torch.empty(s.nstate, s.nstate, dtype=torch.float64, device=psi.device) for _ in range(4)]
        st["F2"], st["psi"] = torch.empty_like(psi), torch.empty_like(psi)
    return st


def _ortho_inputs(s, psi, rng):
    """A force, a velocity, a drifted non-orthogonal set and its T, of the
    sizes that they have between two steps of a run."""
    g2 = torch.as_tensor(s.g2(), device=psi.device)
    w = torch.as_tensor(s.kx_weight(), device=psi.device)
    force = -psi * (w * g2) + 0.3 * psi.roll(1, 0) * w + 0.05 * psi.roll(3, 0)
    v = 2e-4 * psi.roll(2, 0) / (1.0 + g2)
    psi_t = psi + 3e-4 * psi.roll(1, 0) / (1.0 + 0.1 * g2)
    e = rng.standard_normal((s.nstate, s.nstate)) * 1e-4
    T = torch.as_tensor(np.eye(s.nstate) + e + e.T, device=psi.device)
    return dict(force=force.contiguous(), v0=v.contiguous(), psi_t0=psi_t.contiguous(), T0=T)


# ----------------------------------------------------------------------------
# one pass
# ----------------------------------------------------------------------------

def _restart(d, psi0, state=None):
    d.psi.copy_(psi0)
    d.psi_t.copy_(psi0)
    d.v.zero_()
    d.T.zero_()
    d.T.fill_diagonal_(1.0)
    d.iteration, d.half_step = 0, True
    if state is not None:
        state.iteration, state.psiv_pending = 0, 0


def _terms(records):
    return np.array([[r[k] for k in TERMS] for r in records])


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "batch":
        with torch.cuda.stream(st["drivers"][0].stream):
            for d, p, s in zip(st["drivers"], st["psi0"], st["states"]):
                _restart(d, p, s)
        recs = run_batch(st["drivers"], st["states"], case["steps"])
        return [dict(e=_terms(r), psi=d.psi, v=d.v, psi_t=d.psi_t) for r, d in zip(recs, st["drivers"])]
    d = st["driver"]
    if kind == "run":
        with torch.cuda.stream(d.stream):
            _restart(d, st["psi0"], st["state"])
            if case["ions"]:
                d.ctx.set_atoms(st["sys"].pos)
                d.ctx.set_ions(st["masses"], st["vel"])
        recs = d.run_native(st["state"], case["steps"])
        out = dict(e=_terms(recs), psi=d.psi, v=d.v, psi_t=d.psi_t)
        if case["ions"]:
            out["pos"], out["vel"] = d.ctx.get_ions()
        return out
    if kind == "force":
        d.forces()
        e = d.ctx.energies()
        return dict(force=d.F, e=np.array([e[k] for k in TERMS[:8]]))
    if kind == "minimize":
        _restart(d, st["psi0"])
        m = st["minimizer"]
        m.conj.zero_()
        m.iteration, m.num_reset, m.fovlap, m.fmag = 0, 0, 0.0, 0.0
        recs = m.run(case["steps"])
        return dict(e=np.array([[r[k] for k in TERMS[:6]] + [r["FMAG"]] for r in recs]), psi=d.psi, conj=m.conj)
    c, s = d.ctx, st["sys"]
    lam, gam, S, T = st["mats"]
    st["v"].copy_(st["v0"])
    st["psi_t"].copy_(st["psi_t0"])
    fwd, bwd = (c.pc_forward_mixed, c.pc_backward_mixed) if d.mixed else (c.pc_forward, c.pc_backward)
    fwd(st["psi0"], st["force"], 1.0, 1.0, lam)
    c.small_gemm(st["T0"], lam, 1.0, gam)
    bwd(gam, st["psi0"], -0.5, -1.0, st["F2"], M2=st["T0"], X2=st["force"], a2=1.0)
    c.integrate(st["F2"], st["v"], st["psi_t"], s.dt, True)
    c.pc_forward(st["psi_t"], st["psi_t"], 2.0, 0.5, S)
    c.ortho_invsqrt(S, T)
    c.pc_backward(T, st["psi_t"], 1.0, 1.0, st["psi"])
    return dict(lam=lam, F2=st["F2"], v=st["v"], psi_t=st["psi_t"], S=S, T=T, psi=st["psi"])


# ----------------------------------------------------------------------------
# what a pass cannot do without
# ----------------------------------------------------------------------------

def work(case):
    if case["kind"] == "batch":
        parts = [work(dict(c, kind="run", nsys=1)) for c, _ in _members(case, 0)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n, grid = case["nstate"], case["grid"]
    ng = _base(case["nmol"], case["ecut"], grid, n, case["xc"]).ng
    coef = 16.0 * n * ng
    npts = float(grid) ** 3
    prod = 2.0 * n * n * 2.0 * ng                       # one states x states product
    nl = 2.0 * 2.0 * n * case["nmol"] * 2.0 * ng        # Z and its force (structure factor)
    # psi(g) -> psi(r) -> V psi -> force: two real transforms per state; the
    # density side: 8 transforms with the gradient correction, else 2
    fft = 2.5 * npts * math.log2(npts)
    force = (2 * n + (8 if case["xc"] == "blyp" else 2)) * fft + 3.0 * n * npts + (nl if case["nl"] == "sf" else 0.0)
    half = 4.0 * prod + 0.5 * prod                      # Lambda, two-term F', Psi T, symmetric S
    if case["kind"] == "force":
        return {"bytes": 2 * coef, "flops": force}
    if case["kind"] == "ortho":
        return {"bytes": 9 * coef, "flops": half}       # psi, F, T in; F', v, psi_t in and out; psi out
    if case["kind"] == "minimize":
        return {"bytes": case["steps"] * 4 * coef, "flops": case["steps"] * (force + half)}
    # a step reads and writes psi, psi_t and v
    return {"bytes": case["steps"] * 6 * coef, "flops": case["steps"] * (force + half)}


def tolerance(case):
    """About four times the distance from exact() seen over the ranges: FP64
    1e-13 (velocities after several steps), mixed 6e-6 at 32 molecules and
    7e-5 at 128, where FP32 sums run over more states."""
    if case["precision"] == "fp64":
        return {"rel": 1e-11, "max": 1e-8}
    rel = 3e-5 * max(1.0, case["nmol"] / 32.0) ** 1.7
    return {"rel": rel, "max": min(0.5, 200.0 * rel)}


# ----------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ----------------------------------------------------------------------------

class _Ref:
    """FP64 restatement of the step's pieces on torch tensors."""

    def __init__(self, s, case, dev):
        self.s, self.case, self.dev = s, case, dev
        t = functools.partial(torch.as_tensor, device=dev)
        self.t = t
        self.n, self.N = s.nstate, s.nfft[0]
        self.npts, self.vol = float(self.N) ** 3, s.box ** 3
        self.f = 2.0 * math.pi / s.box
        self.kx, self.ky, self.kz = (t(k, dtype=torch.int64) for k in (s.kx, s.ky, s.kz))
        self.g2 = self.f ** 2 * (self.kx ** 2 + self.ky ** 2 + self.kz ** 2).double()
        self.w = torch.where(self.kx == 0, 1.0, 2.0).double()
        self.k0 = s.nkx0
        self.red, self.partner = s.nkx0_red, t(_kx0_partner(s))
        self.cmass = t(s.cmass)
        N = self.N
        a = torch.arange(N // 2 + 1, device=dev)
        b = torch.arange(-(N // 2), N - N // 2, device=dev)
        K = torch.meshgrid(a, b, b, indexing="ij")
        g2 = self.f ** 2 * (K[0] ** 2 + K[1] ** 2 + K[2] ** 2).double()
        m = g2 <= 4.0 * s.ecut_ry
        self.dk = [k[m] for k in K]
        self.dg2 = g2[m]
        self.dw = torch.where(self.dk[0] == 0, 1.0, 2.0).double()
        self.at = (self.dk[2] % N, self.dk[1] % N, self.dk[0])
        pos = t(s.pos)
        self.sums = []
        for ty in range(2):
            p = pos[t(s.atm_type) == ty]
            e = [torch.polar(torch.ones((), dtype=torch.float64, device=dev), self.f * p[:, d, None] * x.double())
                 for d, x in ((0, a), (1, b), (2, b))]
            full = torch.einsum("ax,ay,az->xyz", *e) if len(p) < 4 else torch.stack(
                [(e[0][:, i, None] * e[1]).T @ e[2] for i in range(len(a))])
            self.sums.append(full[m])
        if case["nl"] == "ees":
            self._ees(pos[t(s.atm_type) == 0])
        else:
            p = pos[t(s.atm_type) == 0]
            k = self.f * torch.stack([self.kx, self.ky, self.kz]).double()
            self.sf = torch.polar((self.w * self._proj())[None].expand(len(p), -1).contiguous(), -(p @ k))

    def _spline(self, coef, g):
        s = self.s.vloc
        i = ((g - s.gmin) / s.dg + 1.0).long().clamp(1, coef.shape[0])
        h = g - ((i - 1).double() * s.dg + s.gmin)
        c = coef[i - 1]
        return ((c[:, 3] * h + c[:, 2]) * h + c[:, 1]) * h + c[:, 0]

    def _proj(self):
        s = self.s
        g = self.g2.sqrt()
        p = self._spline(self.t(s.nl_proj.coef[0]), torch.where(g == 0, 1.0, g))
        return torch.where(g == 0, float(s.nl_gz0[0]), p) / math.sqrt(4.0 * math.pi)

    def _spline_grid(self):
        n = int(2.0 * 1.2 * (int(np.abs(self.s.kx).max()) + 1))
        return _smooth(max(n, 2 * (int(np.abs(self.s.kx).max()) + 1)))

    def _ees(self, p):
        """Cardinal B-spline stencils of the atoms and the projector factor dyp."""
        o, n = self.case["order"], self._spline_grid()
        self.en = n

        def spline(u):          # M_o(u)
            if len(u.shape) == 0:
                u = u[None]
            def M(k, x):
                if k == 2:
                    return torch.clamp(1.0 - (x - 1.0).abs(), min=0.0)
                return (x * M(k - 1, x) + (k - x) * M(k - 1, x - 1.0)) / (k - 1)
            return M(o, u)
        x = (p / self.s.box) % 1.0 * n
        i0 = x.floor()
        j = torch.arange(o, device=self.dev)
        self.ei = ((i0[:, :, None] - j).long()) % n                  # grid points u = x - i in (0, o)
        self.em = spline((x - i0)[:, :, None] + j)
        k = torch.arange(1, o, device=self.dev).double()
        mk = spline(k)
        m = torch.arange(n, device=self.dev).double()
        unit = torch.ones((), dtype=torch.float64, device=self.dev)
        den = (torch.polar(unit, 2 * math.pi / n * m[:, None] * (k - 1)) * mk).sum(1)
        b = torch.polar(unit, 2 * math.pi * (o - 1) / n * m) / den
        self.dyp = b[self.kx % n] * b[self.ky % n] * b[self.kz % n] * self._proj()
        z = self.g2 == 0
        self.dyp[z] = self.dyp[z].real.to(self.dyp.dtype)

    def chunks(self, N):
        step = max(1, int(6e8 / (16.0 * N ** 3)))
        return [slice(a, min(self.n, a + step)) for a in range(0, self.n, step)]

    def to_r(self, c, N):
        h = torch.zeros(c.shape[0], N, N, N // 2 + 1, dtype=torch.complex128, device=self.dev)
        h[:, self.kz % N, self.ky % N, self.kx] = c.conj()
        return torch.fft.irfftn(h, s=(N, N, N), dim=(1, 2, 3)) * float(N) ** 3

    def to_g(self, r, N):
        return torch.fft.rfftn(r, dim=(1, 2, 3))[:, self.kz % N, self.ky % N, self.kx].conj()

    def field(self, vals):
        N = self.N
        h = torch.zeros(N, N, N // 2 + 1, dtype=torch.complex128, device=self.dev)
        h[self.at] = vals
        return torch.fft.irfftn(h, s=(N, N, N), dim=(0, 1, 2)) * self.npts

    def xc(self, rho, blyp):
        rs = (3.0 / (4.0 * math.pi * rho)) ** (1.0 / 3.0)
        sq, ln = rs.sqrt(), rs.log()
        x = -(3.0 * rho / math.pi) ** (1.0 / 3.0)
        c1 = 1.0 + 1.0529 * sq + 0.3334 * rs
        c2 = 1.0 + 7.0 / 6.0 * 1.0529 * sq + 4.0 / 3.0 * 0.3334 * rs
        hi, hm = -0.1423 / c1, -0.1423 * c2 / (c1 * c1)
        lo = 0.0311 * ln - 0.048 + 0.002 * rs * ln - 0.0116 * rs
        lm = 0.0311 * ln + (-0.048 - 0.0311 / 3) + 2 * 0.002 / 3 * rs * ln + (2 * -0.0116 - 0.002) / 3 * rs
        c, m = torch.where(rs >= 1, hi, lo), torch.where(rs >= 1, hm, lm)
        if blyp:
            c, m = 0 * c, 0 * m
        dv = self.vol / self.npts
        return x + m, float((0.75 * x * rho + c * rho).sum()) * dv, float(((x + m) * rho).sum()) * dv

    def gga(self, rho):
        """Becke 88 + LYP with the switching function, by automatic differentiation."""
        cut = self.s.gga_cut
        gv = [self.f * k.double() for k in self.dk]
        rg = torch.fft.rfftn(rho / self.npts)[self.at]
        grad = torch.stack([self.field(1j * k * rg) for k in gv])
        on = rho > 0.1 * cut
        r = torch.where(on, rho, 1.0).requires_grad_(True)
        g = (grad * grad).sum(0).sqrt().requires_grad_(True)
        with torch.enable_grad():
            t = ((r - 0.1 * cut) / (3.9 * cut)).clamp(0.0, 1.0)
            sw = t * t * (3.0 - 2.0 * t)
            rs = 0.5 * r
            x = 0.5 * g / rs ** (4.0 / 3.0)
            fx = -2 * 0.0042 * rs ** (4.0 / 3.0) * x * x / (1.0 + 6 * 0.0042 * x * torch.asinh(x))
            a, b, c, d = 0.04918, 0.132, 0.2533, 0.349
            cf = 0.3 * (3.0 * math.pi ** 2) ** (2.0 / 3.0)
            u = r ** (-1.0 / 3.0)
            den = 1.0 + d * u
            om = torch.exp(-c * u) * u ** 11 / den
            dl = c * u + d * u / den
            A = cf * r ** (8.0 / 3.0) + (5.0 / 12 - 7.0 * dl / 72 - 11.0 / 24) * g * g
            fc = -a * r / den - a * b * om * A * r * r
            e = torch.where(on, (fx + fc) * sw, 0.0)
            dr, dg = torch.autograd.grad(e.sum(), (r, g))
        g = g.detach()
        h = grad * torch.where(on & (g > 0), dg / g, 0.0)
        hg = [torch.fft.rfftn(h[i] / self.npts)[self.at] for i in range(3)]
        v = torch.where(on, dr, 0.0) - self.field(sum(1j * k * q for k, q in zip(gv, hg)))
        return v, float(e.detach().sum()) * self.vol / self.npts

    def vks(self, rho):
        s, en = self.s, {}
        blyp = self.case["xc"] == "blyp"
        v, en["EEXC"], en["MUXC"] = self.xc(rho, blyp)
        en["EGGA"] = 0.0
        if blyp:
            vg, en["EGGA"] = self.gga(rho)
            v = v + vg
        rg = torch.fft.rfftn(rho * (self.vol / self.npts))[self.at]
        z = self.dg2 == 0
        g2 = torch.where(z, 1.0, self.dg2)
        hf = torch.where(z, 0.0, 4 * math.pi / (g2 * self.vol))
        en["EHART"] = float((hf * rg.abs() ** 2 * self.dw).sum()) / 2
        ext = sum(self._spline(self.t(s.vloc.coef[ty]), g2.sqrt()) / self.vol * self.sums[ty] for ty in range(2))
        ext = torch.where(z, 0.0, ext)
        ewd = hf * torch.exp(-g2 / (4 * s.alp_ewd ** 2))
        q = 6.0 * self.sums[0] + self.sums[1]
        en["EWALD_RECIP"] = float((ewd * q.abs() ** 2 * self.dw).sum()) / 2
        v0 = float(np.sum(s.gzvps[s.atm_type])) / self.vol
        en["EEXT"] = float(((rg * ext).real * self.dw).sum()) + v0 * float(rg[z].real)
        vg = rg * hf + ext.conj()
        vg[z] = v0
        return v + self.field(vg), en

    def rv(self, a):
        return torch.view_as_real(a).reshape(a.shape[0], -1)

    def cv(self, a):
        return torch.view_as_complex(a.reshape(a.shape[0], -1, 2).contiguous())

    def nonlocal_(self, psi):
        vn = float(self.s.nl_vnorm[0]) / self.vol
        if self.case["nl"] != "ees":
            Z = self.rv(psi) @ self.rv(self.sf).T
            return -self.cv((2 * vn * Z) @ self.rv(self.sf)), float((Z * Z).sum()) * vn
        n, o = self.en, self.case["order"]
        ia, ib, ic = (self.ei[:, d] for d in range(3))
        wt = torch.einsum("ai,aj,ak->akji", self.em[:, 0], self.em[:, 1], self.em[:, 2]).reshape(len(ia), -1)
        at = ((ic[:, :, None, None] * n + ib[:, None, :, None]) * n + ia[:, None, None, :]).reshape(len(ia), -1)
        out, enl = torch.empty_like(psi), 0.0
        for c in self.chunks(n):
            pr = self.to_r((self.dyp * psi[c]).conj(), n).reshape(-1, n ** 3)
            Z = (pr[:, at] * wt).sum(2)
            enl += float((Z * Z).sum()) * vn
            scr = torch.zeros_like(pr)
            scr.index_add_(1, at.reshape(-1), ((2 * vn * Z)[:, :, None] * wt).reshape(len(Z), -1))
            P = self.to_g(scr.reshape(-1, n, n, n), n)
            P = torch.where(self.g2 == 0, P.real.to(P.dtype), P)
            out[c] = -self.w * (self.dyp * P).conj()
        return out, enl

    def forces(self, psi):
        rho = 0.0
        for c in self.chunks(self.N):
            rho = rho + (self.to_r(psi[c], self.N) ** 2).sum(0) / self.vol
        v, en = self.vks(rho)
        F, en["ENL"] = self.nonlocal_(psi)
        for c in self.chunks(self.N):
            F[c] += self.w * (-2.0 / self.npts) * self.to_g(self.to_r(psi[c], self.N) * v, self.N)
        F -= psi * (self.w * self.g2)
        F[:, self.g2 > self.s.ecut_ry] = 0.0
        en["EKE"] = float((self.w * self.g2 * psi.abs() ** 2).sum()) / 2
        return F, en

    def constrain(self, psi, F, T):
        lam = self.rv(psi) @ self.rv(F).T
        p = psi.clone()
        p[:, :self.k0] *= 0.5
        return self.cv(T.T @ self.rv(F) - (T @ lam).T @ self.rv(p)), lam

    def sync(self, a):
        a[:, :self.red] = a[:, self.partner].conj()
        return a

    def integrate(self, F, v, p, dt, complete):
        r0, zero, r1 = self.red, self.red, self.red + self.s.nkx0_zero
        f = F.clone()
        f[:, zero:r1] = f[:, zero:r1].real.to(f.dtype)
        v = v.clone()
        v[:, zero:r1] = v[:, zero:r1].real.to(v.dtype)
        kick = torch.zeros_like(v)
        kick[:, r0:] = f[:, r0:] * (0.5 * dt / self.cmass[r0:])
        if complete:
            v = v + kick
        m = self.cmass.clone()
        m[r1:self.red + self.s.nkx0_uni] *= 2.0
        fict = 0.5 * float((m[r0:] * v[:, r0:].abs() ** 2).sum())
        v = v + kick
        p = p.clone()
        p[:, r0:] += dt * v[:, r0:]
        return self.sync(v), self.sync(p), fict

    def ortho(self, p):
        r = self.rv(p)
        wt = self.w.repeat_interleave(2)
        S = (r * wt) @ r.T
        e, u = torch.linalg.eigh(S / 2.0)
        T = (u / e.sqrt()) @ u.T
        return self.cv(T.T @ r), S, T


def _exact_run(s, case, psi, dev):
    r = _Ref(s, case, dev)
    p, v, T = psi.clone(), torch.zeros_like(psi), torch.eye(s.nstate, dtype=torch.float64, device=dev)
    recs, half = [], True
    for it in range(case["steps"]):
        F, en = r.forces(psi)
        F, _ = r.constrain(psi, F, T)
        v, p, en["FICT_KE"] = r.integrate(F, v, p, s.dt, it > 0 and half)
        old, half = psi, True
        psi, S, T = r.ortho(p)
        if float((S - 2.0 * torch.eye(s.nstate, device=dev)).abs().max()) > NORB_TOL:
            v, p, half = (psi - old) / s.dt, psi.clone(), False
            T = torch.eye(s.nstate, dtype=torch.float64, device=dev)
        recs.append(en)
    return dict(e=_terms(recs), psi=psi, v=v, psi_t=p)


def _exact_minimize(s, case, psi, dev):
    r = _Ref(s, case, dev)
    eye = torch.eye(s.nstate, dtype=torch.float64, device=dev)
    conj, fov, rows = torch.zeros_like(psi), 0.0, []
    count, fmag = 0, 0.0
    for it in range(case["steps"]):
        F, en = r.forces(psi)
        F, _ = r.constrain(psi, F, eye)
        old, fov = fov, float((F.abs() ** 2).sum())
        last, fmag = fmag, math.sqrt(fov)
        gamma = 0.0
        if it == 0 or (fmag > 1.05 * last and count >= 5) or fmag > 2.0 * last:
            count = 0
        else:
            gamma = fov / old
        count += 1
        inside = r.g2 <= s.ecut_ry
        conj = torch.where(inside, conj * gamma + F, conj)
        psi, _, _ = r.ortho(r.sync(psi + conj * (s.dt / r.cmass)))
        rows.append([en[k] for k in TERMS[:6]] + [fmag])
    return dict(e=np.array(rows), psi=psi, conj=conj)


def exact(case, seed):
    if case["ions"]:
        return None     # the atoms' EES and Ewald forces have no short restatement here
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "batch":
        out = []
        for c, sd in _members(case, seed):
            s, psi, _ = _inputs(c, sd, dev)
            out.append(_exact_run(s, c, psi, dev))
        return out
    s, psi, rng = _inputs(case, seed, dev)
    if case["kind"] == "run":
        return _exact_run(s, case, psi, dev)
    if case["kind"] == "minimize":
        return _exact_minimize(s, case, psi, dev)
    r = _Ref(s, case, dev)
    if case["kind"] == "force":
        F, en = r.forces(psi)
        en["FICT_KE"] = 0.0
        return dict(force=F, e=np.array([en[k] for k in TERMS[:8]]))
    i = _ortho_inputs(s, psi, rng)
    F2, lam = r.constrain(psi, i["force"], i["T0"])
    v, p, _ = r.integrate(F2, i["v0"], i["psi_t0"], s.dt, True)
    new, S, T = r.ortho(p)
    return dict(lam=lam, F2=F2, v=v, psi_t=p, S=S, T=T, psi=new)
