"""The work that programs have this package do, as cases that can be timed.

A case is one call pattern of the package's public interface (Context, Batch)
at one size.  `listed` holds the fixed ones, `draw` makes more of the same
ranges, `prepare` builds what a program holds before the call (a context with
its state on the GPU), `run` is one pass, `work` what one pass cannot do
without, and `exact` the same answers from plain torch in 64 bits.

Sizes come from the workloads of tcp_allpair_gb300/system.py and bench.py
(N = 1,024 plain Ewald; N = 16,384 with a 64^3 mesh; N = 65,536 with a 128^3
mesh of order 5; 64 replicas of 512 to 8,192 particles; N = 4,096 derivatives)
and odd ones in between.

The FP32C precisions compute pairs and meshes in 32 bits: their arrays are
handed on as float32, those of the FP64 precision as they are.
"""
import math

import numpy as np
import torch

import tcp_allpair_gb300 as T
from tcp_allpair_gb300.system import NDIST

EPS = 14.399644154020082     # e^2/(4 pi eps0) in eV A


def listed():
    """The fixed cases."""
    return [
        # a small plasma, hundreds of steps a second of wall time wanted: launches and latency
        {"name": "md_n512", "kind": "md", "n": 512, "gamma": 1.0, "lam": 0.5, "K": 32, "order": 4, "precision": "fp32c",
         "thermo": "notemp", "period": 1, "steps": 50},
        # the plain method at its usual size: FP64 pairs and the direct k-sum, NVE
        {"name": "md_n1024_ewald_fp64", "kind": "md", "n": 1024, "gamma": 1.0, "lam": 0.5, "K": 0, "order": 4,
         "precision": "fp64", "thermo": "notemp", "period": 1, "steps": 20},
        # what the Fortran main program does with its defaults (FP64, Deutsch, order 4): the routines one by
        # one, the thermostat, RDF and VDF every step and the records refreshed; uneven species, odd size
        {"name": "routines_n3001_fp64", "kind": "routines", "n": 3001, "gamma": 0.7, "lam": 0.4, "K": 32, "order": 4,
         "precision": "fp64", "thermo": "isokin", "period": 1, "steps": 4},
        # the production size with a velocity rescale every ten steps
        {"name": "md_n16384_isokin", "kind": "md", "n": 16384, "gamma": 2.0, "lam": 0.4, "K": 64, "order": 4,
         "precision": "fp32c", "thermo": "isokin", "period": 10, "steps": 20},
        # the headline system, ten steps between two looks at the state
        {"name": "md_n65536", "kind": "md", "n": 65536, "gamma": 1.0, "lam": 0.5, "K": 128, "order": 5,
         "precision": "fp32c", "thermo": "notemp", "period": 1, "steps": 10},
        # the headline system stepped on the caller's own records, as the main loop updates them
        {"name": "records_n65536", "kind": "records", "n": 65536, "gamma": 1.0, "lam": 0.5, "K": 128, "order": 5,
         "precision": "fp32c", "thermo": "notemp", "period": 1, "steps": 2},
        # pair-correlation sampling on every step, an odd size
        {"name": "md_rdf_n24001", "kind": "rdf", "n": 24001, "gamma": 3.0, "lam": 0.3, "K": 64, "order": 5,
         "precision": "fp32c", "thermo": "berend", "period": 1, "steps": 8},
        # FP32C pairs with the reciprocal sum in FP64, a mesh that is no power of two and a higher order
        {"name": "md_r64_n9000", "kind": "md", "n": 9000, "gamma": 1.5, "lam": 0.6, "K": 48, "order": 6,
         "precision": "fp32c_r64", "thermo": "notemp", "period": 1, "steps": 10},
        # one force evaluation of the headline system in FP64, as a check or a restart makes it
        {"name": "force_n65536_fp64", "kind": "force", "n": 65536, "gamma": 1.0, "lam": 0.5, "K": 128, "order": 5,
         "precision": "fp64", "thermo": "notemp", "period": 1, "steps": 1},
        # a parameter scan: 64 replicas of uneven size stepped together
        {"name": "batch64", "kind": "batch", "nrep": 64, "nmin": 512, "nmax": 8192, "steps": 20},
        # a Hessian-vector product and the energy derivatives in FP64
        {"name": "hvp_n4096_fp64", "kind": "hvp", "n": 4096, "gamma": 1.0, "lam": 0.5, "K": 32, "order": 4,
         "precision": "fp64", "thermo": "notemp", "period": 1, "steps": 1},
        # the gradient of the mean kinetic temperature through 200 steps, checkpoints every 20
        {"name": "reverse_n4096", "kind": "reverse", "n": 4096, "gamma": 1.0, "lam": 0.5, "K": 32, "order": 4,
         "precision": "fp32c", "thermo": "notemp", "period": 1, "steps": 200, "every": 20},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mesh(n):
    """The mesh that a program takes for n particles: about two points per mean distance."""
    return 32 if n < 3000 else 48 if n < 10000 else 64 if n < 30000 else 96 if n < 50000 else 128


def draw(rng):
    """One more case of the ranges that the listed ones stand for."""
    kind = rng.choice(["md", "md", "md", "ewald", "routines", "records", "rdf", "force", "batch", "hvp", "reverse"])
    c = {"kind": "md" if kind == "ewald" else kind, "gamma": round(math.exp(rng.uniform(math.log(0.1), math.log(10.0))), 3),
         "lam": round(rng.uniform(0.2, 0.8), 3), "order": rng.choice([4, 4, 5, 6]), "precision": "fp32c",
         "thermo": rng.choice(["notemp", "isokin", "berend"]), "period": rng.choice([1, 10]), "steps": 1}
    if kind == "md":
        c["n"] = _log_int(rng, 512, 65536)
        c["precision"] = rng.choice(["fp32c", "fp32c", "fp32c_r64", "fp64"])
        c["steps"] = 50 if c["n"] < 4096 else 10
        if c["precision"] == "fp64":
            c["n"] = min(c["n"], 20000)
            c["steps"] = 10 if c["n"] < 8000 else 3
    elif kind == "ewald":
        c.update(n=_log_int(rng, 512, 3000), precision=rng.choice(["fp64", "fp64", "fp32c"]), steps=20)
    elif kind == "routines":
        c.update(n=_log_int(rng, 1000, 12000), precision=rng.choice(["fp64", "fp64", "fp32c"]), steps=4)
    elif kind == "records":
        c.update(n=_log_int(rng, 4096, 65536), steps=2)
    elif kind == "rdf":
        c.update(n=_log_int(rng, 2000, 65536), precision=rng.choice(["fp32c", "fp32c", "fp64"]), steps=4)
        if c["precision"] == "fp64":
            c["n"] = min(c["n"], 20000)
    elif kind == "force":
        c.update(n=_log_int(rng, 2048, 60000), precision=rng.choice(["fp32c", "fp64", "fp64"]))
    elif kind == "batch":
        return {"kind": "batch", "nrep": _log_int(rng, 6, 64), "nmin": _log_int(rng, 512, 1500), "nmax": _log_int(rng, 3000, 8192),
                "steps": 20}
    elif kind == "hvp":
        c.update(n=_log_int(rng, 1024, 8192), precision=rng.choice(["fp64", "fp32c"]), thermo="notemp")
    else:
        c.update(n=_log_int(rng, 512, 4096), steps=rng.choice([40, 100]), every=rng.choice([10, 20]), thermo="notemp")
    c["K"] = 0 if kind == "ewald" else _mesh(c["n"])
    return c


# ---- inputs -----------------------------------------------------------------------
def _system(case, seed):
    """Seeded particles in reference units.  The plain Ewald sum takes its usual alpha = 5.6/L; the systems
    of order 5 the alpha of a 1e-6 Ewald error, the others 3.1/rc."""
    kw = {"alpha_rc": 2.8} if case["K"] == 0 else {"ewald_rel_err": 1e-6} if case["order"] == 5 else {"alpha_rc": 3.1}
    return T.make_system(case["n"], gamma=case["gamma"], lam=case["lam"], seed=seed, K=case["K"], order=case["order"], **kw)


def _params(case, s):
    return T.params_for(s, precision=case["precision"], ei="deutsch" if case["kind"] == "routines" else "kelbg",
                        recip="ewald" if case["K"] == 0 else "spme", thermo=case["thermo"], thermo_period=case["period"],
                        tau=20.0 * s.dt)


def _vector(case, seed):
    """The direction of a Hessian-vector product: a Gaussian vector of length 1."""
    w = np.random.default_rng(seed + 1000).normal(size=(case["n"], 3))
    return w / np.linalg.norm(w)


def _batch_layout(case):
    """(n, gamma, lambda) of every replica, by the rules of make_batch_systems: the layout of a scan, the same for
    every seed of the particles."""
    rng = np.random.default_rng(case["nrep"])
    lo, hi = math.log(case["nmin"]), math.log(case["nmax"])
    return [(2 * int(round(math.exp(rng.uniform(lo, hi)) / 2)), math.exp(rng.uniform(math.log(0.1), math.log(10.0))),
             rng.uniform(0.2, 0.8)) for _ in range(case["nrep"])]


def _batch_mesh(n):
    return 32 if n < 2048 else 48 if n < 4096 else 64


def _batch(case, seed):
    return [T.make_system(n, gamma=g, lam=lam, seed=1000 * seed + r, alpha_rc=3.1, K=_batch_mesh(n), order=4)
            for r, (n, g, lam) in enumerate(_batch_layout(case))]


def prepare(case, seed):
    """A context (or batch) with its particles on the GPU and the forces of the start, where steps follow."""
    if case["kind"] == "batch":
        ss = _batch(case, seed)
        b = T.Batch([T.params_for(s) for s in ss], [s.nel for s in ss], [s.nion for s in ss])
        b.EWALD_SELF()
        for r, s in enumerate(ss):
            b.upload(r, x=s.x, v=s.v)
        b.force()
        return {"case": case, "batch": b, "dt": ss[0].dt}
    s = _system(case, seed)
    ctx = T.Context(_params(case, s), s.nel, s.nion)
    if case["kind"] in ("rdf", "routines"):
        ctx.set_flags(T.FLAG_ENERGY | T.FLAG_RDF | T.FLAG_VDF)
    ctx.EWALD_SELF()
    state = {"case": case, "ctx": ctx, "dt": s.dt, "x": s.x, "v": s.v}
    if case["kind"] in ("records", "routines"):
        state["qel"], state["qion"] = s.to_pt()
        ctx.upload_pt(state["qel"], state["qion"])
    else:
        ctx.upload(x=s.x, v=s.v)
    ctx.force()
    if case["kind"] in ("rdf", "routines"):
        ctx.histograms(reset=True)
    if case["kind"] == "records":
        ctx.download_pt(state["qel"], state["qion"])
    if case["kind"] == "hvp":
        state["w"] = _vector(case, seed)
    return state


# ---- one pass ---------------------------------------------------------------------
def _arrays(case, *arrays):
    """Result arrays: float32 for the 32-bit precisions."""
    return [a if case["precision"] == "fp64" else a.astype(np.float32) for a in arrays]


def _scalars(e):
    """What the energy files of a run hold."""
    return {k: e[k] for k in ("Epot", "Um", "mv2el", "mv2ion")}


def run(state):
    case = state["case"]
    return _RUN[case["kind"]](case, state)


def _run_md(case, st):
    e = st["ctx"].md_steps(st["dt"], case["steps"])
    x, v, f, _ = st["ctx"].download()
    return {"energy": _scalars(e), "xvf": _arrays(case, x, v, f)}


def _run_rdf(case, st):
    e = st["ctx"].md_steps(st["dt"], case["steps"])
    rdf, vdf = st["ctx"].histograms(reset=True)
    x, v, f, _ = st["ctx"].download()
    return {"energy": _scalars(e), "xvf": _arrays(case, x, v, f), "hist": _arrays(case, rdf, vdf)}


def _run_records(case, st):
    qel, qion = st["qel"], st["qion"]
    e = st["ctx"].md_steps_pt(st["dt"], case["steps"], qel, qion)
    return {"energy": _scalars(e), "rec": [_arrays(case, q["xx"], q["xv"], q["ff"]) for q in (qel, qion)]}


def _run_routines(case, st):
    """main.f90's loop body with the records and the histograms refreshed on every step."""
    ctx, dt = st["ctx"], st["dt"]
    rdf, vdf = 0.0, 0.0
    for _ in range(case["steps"]):
        ctx.VVerlet1(dt)
        um = ctx.Force_SPME4()
        ur = ctx.Force_direct_self()
        ctx.SPME_SUM()
        ctx.REMOVE_RIGIDMTN()
        mv2el, mv2ion = ctx.VVerlet2(dt)
        ctx.download_pt(st["qel"], st["qion"])
        a, b = ctx.histograms(reset=True)
        rdf, vdf = rdf + a, vdf + b
    return {"energy": {"ur": ur, "um": um, "mv2el": mv2el, "mv2ion": mv2ion}, "hist": _arrays(case, rdf, vdf),
            "rec": [_arrays(case, q["xx"], q["xv"], q["ff"]) for q in (st["qel"], st["qion"])]}


def _run_force(case, st):
    e = st["ctx"].force()
    _, _, f, frec = st["ctx"].download(x=False, v=False, f=True, frec=True)
    return {"energy": {"Epot": e["Epot"], "Um": e["Um"]}, "f": _arrays(case, f, frec)}


def _run_batch(case, st):
    b = st["batch"]
    e = b.md_steps(st["dt"], case["steps"])
    parts = [b.download(r) for r in range(b.nrep)]
    xvf = [np.concatenate([p[k] for p in parts]).astype(np.float32) for k in range(3)]
    return {"energy": np.array([list(_scalars(q).values()) for q in e], dtype=np.float32), "xvf": xvf}


def _run_hvp(case, st):
    hw, dfdl_w = st["ctx"].hvp(st["w"])
    e, dedl, deds = st["ctx"].adjoint_energy()
    return {"hw": _arrays(case, hw), "dfdl_w": dfdl_w, "e": e, "dedl": dedl, "deds": deds}


def _run_reverse(case, st):
    """An initial-value problem: the start is given with every call, as an optimiser does."""
    ctx = st["ctx"]
    ctx.upload(x=st["x"], v=st["v"])
    j, dj = ctx.reverse_md(st["dt"], case["steps"], case["every"])
    return {"j": j, "djdl": dj}


_RUN = {"md": _run_md, "rdf": _run_rdf, "records": _run_records, "routines": _run_routines, "force": _run_force,
        "batch": _run_batch, "hvp": _run_hvp, "reverse": _run_reverse}


# ---- what a pass cannot do without ----------------------------------------------------
def _recip_flops(n, K, order):
    if K == 0:
        return 2109 * n * 2 * 8.0
    return 2 * 2.5 * K ** 3 * math.log2(K ** 3) + 4.0 * n * order ** 3 + 8.0 * K ** 3


def work(case):
    """Every unique pair once (about 33 operations: separation, distance, erfc and exponential, energy, both
    forces), the reciprocal sum, and the state read and written once."""
    if case["kind"] == "batch":
        ss = [n for n, _, _ in _batch_layout(case)]
        flops = sum(33.0 * n * (n - 1) / 2 + _recip_flops(n, _batch_mesh(n), 4) for n in ss) * case["steps"]
        return {"bytes": 18.0 * 8 * sum(ss), "flops": flops}
    n = case["n"]
    step = 33.0 * n * (n - 1) / 2 + _recip_flops(n, case["K"], case["order"])
    if case["kind"] == "hvp":
        step = 3.0 * step
    elif case["kind"] == "reverse":
        step = 4.0 * step
    return {"bytes": 18.0 * 8 * n, "flops": step * case["steps"]}


# ---- the same in 64 bits with plain torch ---------------------------------------------
class _Exact:
    """The system of one case in FP64: forces of every term, the step and the thermostats."""

    def __init__(self, s, ei, thermo, period, tau):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.s, self.ei, self.thermo, self.period, self.tau = s, ei, thermo, period, tau
        t = lambda a: torch.tensor(a, dtype=torch.float64, device=self.dev)  # noqa: E731
        self.x, self.v = t(s.x), t(s.v)
        self.q = t([s.q[0]] * s.nel + [s.q[1]] * s.nion)
        self.m = t([s.xm[0]] * s.nel + [s.xm[1]] * s.nion)
        self.L, self.rc2, self.al, self.n = s.box, s.rc * s.rc, s.alpha, s.n
        self.lam = t(s.lambda_ei)
        self.hist = self.vdf = None
        if s.K:
            self.infl = self._influence()
        else:
            k = torch.arange(-8, 9, dtype=torch.float64, device=self.dev)
            k = torch.stack(torch.meshgrid(k, k, k, indexing="ij"), -1).reshape(-1, 3)
            k2 = (k * k).sum(-1)
            self.kvec = k[(k2 > 0) & (k2 <= 64)] / self.L
        qsum = s.nel * s.q[0] + s.nion * s.q[1]
        self.uo = (-(s.nel * s.q[0] ** 2 + s.nion * s.q[1] ** 2) * self.al / math.sqrt(math.pi)
                   - math.pi * qsum ** 2 / (2 * self.L ** 3 * self.al ** 2))

    # real space: (force, Ur); with dedl also the lambda derivative of the pair energy
    def direct(self, x, lam, count=False):
        n, L, al, q = self.n, self.L, self.al, self.q
        rows = max(1, int(3.0e7) // n)
        fs, ur, dedl = [], torch.zeros((), dtype=torch.float64, device=self.dev), torch.zeros((), dtype=torch.float64, device=self.dev)
        el = torch.arange(n, device=self.dev) < self.s.nel
        dx = self.s.rc / NDIST
        for a in range(0, n, rows):
            b = min(n, a + rows)
            d = x[a:b, None, :] - x[None, :, :]
            d = d - L * torch.round(d.detach() / L)
            r2 = (d * d).sum(-1)
            ok = (r2 < self.rc2) & (torch.arange(a, b, device=self.dev)[:, None] != torch.arange(n, device=self.dev)[None, :])
            r2 = torch.where(ok, r2, torch.ones_like(r2))
            r = torch.sqrt(r2)
            e = torch.erfc(al * r) / r
            w = (e + 2 * al / math.sqrt(math.pi) * torch.exp(-al * al * r2)) / r2
            ei = ok & (el[a:b, None] != el[None, :])
            if self.ei == "kelbg":
                g = torch.exp(-r2 / lam ** 2)
                ek = torch.erfc(r / lam) * math.sqrt(math.pi) / lam
                e = e + torch.where(ei, ek - g / r, torch.zeros_like(r))
                w = w - torch.where(ei, g / (r2 * r), torch.zeros_like(r))
                dl = -math.sqrt(math.pi) * torch.erfc(r / lam) / lam ** 2
            else:
                y = torch.exp(-r / lam)
                e = e - torch.where(ei, y / r, torch.zeros_like(r))
                w = w - torch.where(ei, y * (1 / r + 1 / lam) / r2, torch.zeros_like(r))
                dl = -y / lam ** 2
            qq = torch.where(ok, q[a:b, None] * q[None, :], torch.zeros_like(r))
            fs.append(EPS * ((qq * w)[:, :, None] * d).sum(1))
            ur = ur + 0.5 * (qq * e).sum()
            dedl = dedl + 0.5 * EPS * (qq * torch.where(ei, dl, torch.zeros_like(r))).sum()
            if count and self.hist is not None:
                kind = (~el[a:b]).long()[:, None] + (~el).long()[None, :]
                bins = torch.floor(torch.sqrt(r2) / dx).long()
                keep = ok & (bins <= NDIST)
                self.hist += torch.bincount((kind * (NDIST + 1) + bins)[keep], minlength=3 * (NDIST + 1))
        return torch.cat(fs), ur, dedl

    def _moduli(self):
        K, p = self.s.K, self.s.order
        w, _ = self._weights(torch.zeros(1, dtype=torch.float64, device=self.dev))
        ph = torch.exp(2j * math.pi * torch.arange(K, device=self.dev, dtype=torch.float64)[:, None]
                       * torch.arange(p, device=self.dev, dtype=torch.float64)[None, :] / K)
        den = (ph * w[0][None, :]).sum(-1).abs() ** 2
        near = 0.5 * (torch.roll(den, 1) + torch.roll(den, -1))
        return 1.0 / torch.where(den < 1e-7, near, den)

    def _influence(self):
        K = self.s.K
        m = torch.fft.fftfreq(K, 1.0 / K, dtype=torch.float64, device=self.dev) / self.L
        m2 = m[:, None, None] ** 2 + m[None, :, None] ** 2 + m[None, None, :] ** 2
        b = self._moduli()
        m2[0, 0, 0] = 1.0
        th = torch.exp(-math.pi ** 2 * m2 / self.al ** 2) / m2 * b[:, None, None] * b[None, :, None] * b[None, None, :]
        th[0, 0, 0] = 0.0
        return th

    def _weights(self, w):
        """Cardinal B-spline weights and derivatives at fraction w, grid points INT(u) - (p - 3) + j."""
        p = self.s.order
        a = [torch.ones_like(w)]
        for n in range(2, p + 1):
            if n == p:
                d = [(a[j - 1] if j > 0 else 0.0) - (a[j] if j < p - 1 else 0.0) for j in range(p)]
            a = [((w + (n - 1 - j)) * (a[j - 1] if j > 0 else 0.0) + (1.0 - w + j) * (a[j] if j < n - 1 else 0.0)) / (n - 1)
                 for j in range(n)]
        return torch.stack(a, -1), torch.stack([x * torch.ones_like(w) for x in d], -1)

    def spme(self, x):
        K, p, L = self.s.K, self.s.order, self.L
        u = (x + 0.5 * L) * (K / L)
        i0 = torch.trunc(u.detach())
        W, D = self._weights(u - i0)
        idx = (i0.long()[:, :, None] - (p - 3) + torch.arange(p, device=self.dev)) % K
        flat = ((idx[:, 0, :, None, None] * K + idx[:, 1, None, :, None]) * K + idx[:, 2, None, None, :]).reshape(-1)
        cub = lambda a, b, c: a[:, :, None, None] * b[:, None, :, None] * c[:, None, None, :]  # noqa: E731
        Q = torch.zeros(K ** 3, dtype=torch.float64, device=self.dev).index_add(
            0, flat, (self.q[:, None, None, None] * cub(W[:, 0], W[:, 1], W[:, 2])).reshape(-1)).reshape(K, K, K)
        F = torch.fft.fftn(Q)
        V = L ** 3
        um = EPS / (2 * math.pi * V) * (self.infl * (F.real ** 2 + F.imag ** 2)).sum()
        phi = (torch.fft.ifftn(F * self.infl).real * K ** 3).reshape(-1)[flat].reshape(-1, p, p, p)
        g = [(cub(D[:, 0], W[:, 1], W[:, 2]) * phi).sum((1, 2, 3)), (cub(W[:, 0], D[:, 1], W[:, 2]) * phi).sum((1, 2, 3)),
             (cub(W[:, 0], W[:, 1], D[:, 2]) * phi).sum((1, 2, 3))]
        return -EPS / (math.pi * V) * (K / L) * self.q[:, None] * torch.stack(g, -1), um

    def ewald(self, x):
        V = self.L ** 3
        k2 = (self.kvec ** 2).sum(-1)
        th = torch.exp(-math.pi ** 2 * k2 / self.al ** 2) / k2
        ph = 2 * math.pi * x @ self.kvec.T
        c, s = torch.cos(ph), torch.sin(ph)
        sr, si = (self.q[:, None] * c).sum(0), (self.q[:, None] * s).sum(0)
        f = (2 * EPS / V) * self.q[:, None] * (((s * sr - c * si) * th) @ self.kvec)
        return f, EPS / (2 * math.pi * V) * (th * (sr ** 2 + si ** 2)).sum()

    def force(self, x, lam=None, count=False):
        """(total force without its mean, Ur, Um, reciprocal force, dE/dlambda)"""
        f, ur, dedl = self.direct(x, self.lam if lam is None else lam, count)
        frec, um = self.spme(x) if self.s.K else self.ewald(x)
        f = f + frec
        return f - f.mean(0), ur, um, frec, dedl

    def step(self, k, dt, f, count=False, lam=None):
        """Step k (from 0): the new force and energies; x and v move on."""
        s, m = self.s, self.m[:, None]
        self.v = self.v + 0.5 * dt * f / m
        x = self.x + dt * self.v
        self.x = x - self.L * torch.round(x.detach() / self.L)
        f, ur, um, _, _ = self.force(self.x, lam, count)
        self.v = self.v + 0.5 * dt * f / m
        if self.thermo != "notemp" and (k + 1) % self.period == 0:
            for sl, T0 in ((slice(0, s.nel), s.Te), (slice(s.nel, None), s.Ti)):
                t = (self.m[sl, None] * self.v[sl] ** 2).sum() / (3 * self.v[sl].shape[0])
                self.v[sl] *= torch.sqrt(T0 / t) if self.thermo == "isokin" else torch.sqrt(1 + dt * (T0 / t - 1) / self.tau)
        mv2 = (self.m[:, None] * self.v ** 2).sum(-1)
        if count and self.vdf is not None:
            for j, (sl, T0) in enumerate(((slice(0, s.nel), s.Te), (slice(s.nel, None), s.Ti))):
                b = torch.floor(mv2[sl] / 3 / (T0 * 4.0 / NDIST)).long()
                self.vdf[j] += torch.bincount(b[b <= NDIST], minlength=NDIST + 1)
        return f, ur, um, mv2[:s.nel].sum(), mv2[s.nel:].sum()


def _cpu(t):
    return t.detach().cpu().numpy()


def exact(case, seed):
    """What run() returns for a new state, in 64 bits; None where that would take long."""
    if case["kind"] == "batch":
        return None
    passes = case["steps"] + 1 if case["kind"] != "force" else 1
    cost = passes * float(case["n"]) ** 2 * (4.0 if case["kind"] in ("reverse", "hvp") else 1.0)
    if cost > 2.0e10:
        return None
    s = _system(case, seed)
    X = _Exact(s, "deutsch" if case["kind"] == "routines" else "kelbg", case["thermo"], case["period"], 20.0 * s.dt)
    if case["kind"] == "hvp":
        return _exact_hvp(case, X, _vector(case, seed))
    if case["kind"] == "reverse":
        return _exact_reverse(case, X, s.dt)
    with torch.no_grad():
        f, ur, um, frec, _ = X.force(X.x)
        epot = lambda: float((ur + X.uo) * EPS)  # noqa: E731
        if case["kind"] == "force":
            return {"energy": {"Epot": epot(), "Um": float(um)}, "f": [_cpu(f), _cpu(frec)]}
        count = case["kind"] in ("rdf", "routines")
        if count:
            X.hist = torch.zeros(3 * (NDIST + 1), dtype=torch.int64, device=X.dev)
            X.vdf = torch.zeros(2, NDIST + 1, dtype=torch.int64, device=X.dev)
        for k in range(case["steps"]):
            f, ur, um, mel, mion = X.step(k, s.dt, f, count)
        x, v, f = _cpu(X.x), _cpu(X.v), _cpu(f)
        out = {"energy": {"Epot": epot(), "Um": float(um), "mv2el": float(mel), "mv2ion": float(mion)}}
        if case["kind"] == "routines":
            out["energy"] = {"ur": float(ur), "um": float(um), "mv2el": float(mel), "mv2ion": float(mion)}
        if count:
            out["hist"] = [_cpu(X.hist).reshape(3, -1).astype(float), _cpu(X.vdf).astype(float)]
        if case["kind"] in ("records", "routines"):
            out["rec"] = [[a[:s.nel] for a in (x, v, f)], [a[s.nel:] for a in (x, v, f)]]
        else:
            out["xvf"] = [x, v, f]
        return out


def _exact_hvp(case, X, w):
    import torch.autograd.forward_ad as fwd
    wt = torch.tensor(w, dtype=torch.float64, device=X.dev)
    with torch.no_grad(), fwd.dual_level():
        # the mean force is not removed: H w = -dF(x + t w)/dt
        f, _, _ = X.direct(fwd.make_dual(X.x, wt), X.lam)
        hw = -fwd.unpack_dual(f).tangent
        g, _ = X.spme(fwd.make_dual(X.x, wt)) if X.s.K else X.ewald(fwd.make_dual(X.x, wt))
        hw = hw - fwd.unpack_dual(g).tangent
        f, _, _ = X.direct(X.x, fwd.make_dual(X.lam, torch.ones_like(X.lam)))
        dfdl = (fwd.unpack_dual(f).tangent * wt).sum()
    with torch.no_grad():
        _, ur, um, _, dedl = X.force(X.x)
    e = float((ur + X.uo) * EPS + um)
    return {"hw": [_cpu(hw)], "dfdl_w": float(dfdl), "e": e, "dedl": float(dedl), "deds": 2 * e}


def _exact_reverse(case, X, dt):
    import torch.autograd.forward_ad as fwd
    with torch.no_grad(), fwd.dual_level():
        lam = fwd.make_dual(X.lam, torch.ones_like(X.lam))
        f = X.force(X.x, lam)[0]
        j = torch.zeros((), dtype=torch.float64, device=X.dev)
        for k in range(case["steps"]):
            f, _, _, mel, mion = X.step(k, dt, f, lam=lam)
            j = j + (mel + mion) / (3 * X.n * case["steps"])
        p, t = fwd.unpack_dual(j)
    return {"j": float(p), "djdl": float(t)}
