"""Timed cases: what a user of magic_b200 has it do, over the range it is used on.

Four kinds of work, through the package's public entry points:

* ``sht``    the drop-in transforms of a Plan: scalar and toroidal/poloidal round trip;
* ``stage``  the fused nonlinear stage of a radial loop (Plan.nl_bouss, Plan.nl_anel);
* ``lm``     the implicit updates of a time step (BoussinesqStep.lm_loop, AnelasticStep.lm_loop);
* ``step``   a whole CNAB2 time step (BoussinesqStep.step, AnelasticStep.step).

Fields are smooth along the radius (a few sine modes) and fall off like
(l + 1)^-2 over the degrees.  ``exact`` restates each kind in plain FP64 torch.
"""

import math

import numpy as np
import torch

CD, RD = torch.complex128, torch.float64
COURFAC, ALFFAC = 2.5, 1.0   # what a time step passes to its stage
RADRATIO = 0.35

# Plans and per-shape operators, which a program keeps for all its runs of one shape
_plans = {}
_shared = {}


# ---------------------------------------------------------------- the cases

def listed():
    return [
        # one scalar of the smallest grid there and back: launches and host time
        dict(name="sht_fp64_l16_b1", kind="sht", precision="fp64", l_max=16, minc=1, cols=1),
        # odd sizes: five prime factors in n_phi, a column count that fills no tile
        dict(name="sht_fp64_l213_b37", kind="sht", precision="fp64", l_max=213, minc=1, cols=37),
        # the transform benchmark: 65 levels, FP32-accurate transforms
        dict(name="sht_split_l127_b65", kind="sht", precision="split", l_max=127, minc=1, cols=65),
        # a dynamo's stage in the default precision of a plan
        dict(name="stage_fp64_l170_n65", kind="stage", precision="fp64", l_max=170, minc=1,
             n_r=65, anel=False, mag=True, chem=False),
        # the stage of the headline step
        dict(name="stage_ozaki_l255_n97", kind="stage", precision="ozaki", l_max=255, minc=1,
             n_r=97, anel=False, mag=True, chem=False),
        # a served run's stage
        dict(name="stage_split_l85_n49", kind="stage", precision="split", l_max=85, minc=1,
             n_r=49, anel=False, mag=True, chem=False),
        # anelastic convection in the default precision of AnelasticStep
        dict(name="anel_fp64_l127_n65", kind="stage", precision="fp64", l_max=127, minc=1,
             n_r=65, anel=True, mag=False, chem=False),
        # the largest stage that the benchmark runs
        dict(name="anel_ozaki_l383_n129", kind="stage", precision="ozaki", l_max=383, minc=1,
             n_r=129, anel=True, mag=False, chem=False),
        # implicit updates on finite differences: banded solves
        dict(name="lm_fd_l255_n97", kind="lm", precision="ozaki", l_max=255, minc=1, n_r=97,
             scheme="FD", anel=False),
        # implicit updates on Chebyshev levels: dense operators, coupled (w, p)
        dict(name="lm_anel_l383_n129", kind="lm", precision="split", l_max=383, minc=1, n_r=129,
             scheme="chebyshev", anel=True),
        # the headline step
        dict(name="step_ozaki_l255_n97", kind="step", precision="ozaki", l_max=255, minc=1,
             n_r=97, scheme="FD", anel=False),
        # a small served run, whole
        dict(name="step_split_l64_n33", kind="step", precision="split", l_max=64, minc=1,
             n_r=33, scheme="chebyshev", anel=False),
    ]


def _smooth_size(n):
    """The smallest 2^i 3^j 5^k that is at least n."""
    return min(2 ** i * 3 ** j * 5 ** k for i in range(13) for j in range(7) for k in range(7)
               if 2 ** i * 3 ** j * 5 ** k >= n)


def _sizes(l_max, minc):
    """(n_theta, n_phi of one sector, n_m) of a resolution."""
    tot = _smooth_size(2 * ((30 * l_max) // 20))
    return tot // 2, tot // minc, l_max // minc + 1


def _lm_max(l_max, minc):
    return sum(l_max - m + 1 for m in range(0, l_max + 1, minc))


def draw(rng):
    """A case of the same ranges, at most as large as the largest listed ones."""
    log = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))
    while True:
        kind = rng.choice(("sht", "sht", "stage", "stage", "stage", "lm", "step"))
        anel = kind != "sht" and rng.random() < 0.4
        precision = rng.choice(("fp64", "ozaki", "split"))
        if kind == "sht" and precision == "ozaki":
            precision = "fp64"  # the same transforms
        l_max = log(16, 383 if anel or kind == "sht" else 255)
        minc = rng.choice((1, 1, 1, 2, 4))
        tot = _sizes(l_max, 1)[1]
        if tot % (2 * minc) or tot % 4 or l_max < 4 * minc:
            continue  # an even number of points in a sector and of colatitudes
        c = dict(kind=kind, precision=precision, l_max=l_max, minc=minc)
        size = _lm_max(l_max, minc) * tot
        if kind == "sht":
            c["cols"] = log(1, 130)
            if size * c["cols"] > _lm_max(213, 1) * 640 * 60:
                continue
            return c
        c["n_r"] = log(17, 129)
        most = 300 if anel and kind != "lm" and precision != "fp64" else 97
        if size * c["n_r"] > _lm_max(255, 1) * 768 * most:
            continue
        c["anel"] = anel
        if kind == "stage":
            c["mag"] = not anel or rng.random() < 0.3
            c["chem"] = rng.random() < 0.25
        else:
            # finite differences and Chebyshev levels; the anelastic steps are Chebyshev ones
            c["scheme"] = "chebyshev" if anel else rng.choice(("FD", "chebyshev"))
            if c["scheme"] == "chebyshev" and l_max * c["n_r"] ** 2 > 383 * 129 ** 2:
                continue
        return c


# --------------------------------------------------------------- the inputs

def _device():
    return torch.device("cuda", torch.cuda.current_device())


class _Shell:
    """Sizes, radii and radial profiles of a case."""

    def __init__(self, case):
        self.l_max, self.minc = case["l_max"], case["minc"]
        self.n_theta, self.n_phi, self.n_m = _sizes(self.l_max, self.minc)
        self.lm_max = _lm_max(self.l_max, self.minc)
        self.dev = _device()
        l, m = [], []
        for k in range(0, self.l_max + 1, self.minc):
            l += range(k, self.l_max + 1)
            m += [k] * (self.l_max - k + 1)
        self.l = torch.tensor(l, device=self.dev)
        self.m = torch.tensor(m, device=self.dev)
        self.dL = (self.l * (self.l + 1)).to(RD)[:, None]
        self.m0 = self.m == 0
        n = self.n_r = case.get("n_r", 0)
        if not n:
            return
        self.anel = case["anel"]
        self.cheb = case.get("scheme", "chebyshev") != "FD"
        r_cmb = 1.0 / (1.0 - RADRATIO)
        k = np.arange(n)
        self.r = (0.5 * np.cos(math.pi * k / (n - 1)) + r_cmb - 0.5) if self.cheb else _fd_radii(n)
        r = self.r
        dr = np.abs(np.diff(r))
        edge = np.concatenate((dr[:1], np.minimum(dr[:-1], dr[1:]), dr[-1:]))
        one, nil = np.ones(n), np.zeros(n)
        p = dict(r=r, or1=1 / r, or2=1 / r ** 2, or4=1 / r ** 4, delxr2=edge ** 2,
                 delxh2=r ** 2 / (self.l_max * (self.l_max + 1.0)), orho1=one, orho2=one, rho0=one,
                 beta=nil, dbeta=nil, dLtemp0=nil, temp0=one, otemp1=one, visc=one, lambda_=one,
                 rgrav=r / r_cmb)
        # the physics of the steps: Boussinesq dynamo, anelastic convection
        if self.anel:
            self.phys = dict(ek=1e-4, ra=3e6, pr=1.0, prmag=5.0, dt=1e-6)
            strat, polind = 5.0, 2.0
            diss = (math.exp(strat / polind) - 1.0) * RADRATIO
            g = r_cmb ** 2 / r ** 2
            temp = diss * r_cmb ** 2 / r + 1.0 - diss * r_cmb
            dg = -2.0 * g / r
            p.update(rgrav=g, temp0=temp, otemp1=1 / temp, rho0=temp ** polind,
                     orho1=temp ** -polind, orho2=temp ** (-2 * polind),
                     beta=-polind * diss * g / temp, dLtemp0=-diss * g / temp,
                     dbeta=-polind * diss / temp ** 2 * (dg * temp + diss * g ** 2))
            self.polind, self.visc_heat = polind, diss * self.phys["pr"] / self.phys["ra"]
        else:
            self.phys = dict(ek=1e-5, ra=3e8, pr=1.0, prmag=1.0, dt=2e-7 if self.l_max > 100 else 1e-6)
            self.visc_heat = 0.0
        self.mag = case.get("mag", not self.anel)
        self.ohm = self.visc_heat / (self.phys["ek"] * self.phys["prmag"] ** 2) if self.mag else 0.0
        self.np = p
        self.prof = {k: torch.as_tensor(v, device=self.dev) for k, v in p.items()}
        f = self.phys
        self.LFfac, self.opm, self.opr = 1 / (f["ek"] * f["prmag"]), 1 / f["prmag"], 1 / f["pr"]
        self.CorFac, self.BuoFac = 1 / f["ek"], f["ra"] / f["pr"]

    def row(self, name):
        return self.prof[name][None, :]


def _fd_radii(n, stretch=0.3, ratio=0.1):
    """Finite-difference radii: geometric boundary layers around a uniform bulk."""
    nb = int((n - 1) / (2.0 * (1.0 + stretch)))
    g = math.exp(math.log(ratio) / nb)
    bulk = n - 1 - 2 * nb
    h = 1.0 / (bulk + 2.0 * g * (1.0 - ratio) / (1.0 - g))
    steps = [h * ratio / g ** i for i in range(nb)]
    r_cmb = 1.0 / (1.0 - RADRATIO)
    r = r_cmb - np.concatenate(([0.0], np.cumsum(steps + [h] * bulk + [x for x in steps[::-1]])))
    r[-1] = r_cmb - 1.0
    return r


def _spectrum(sh, gen, cols, amp=1.0):
    c = torch.randn(sh.lm_max, cols, dtype=CD, generator=gen, device=sh.dev)
    c = c * (amp * (sh.l + 1.0) ** -2)[:, None]
    c[sh.m0] = c[sh.m0].real.to(CD)
    return c


def _field(sh, gen, amp, orders=3, modes=6):
    """A field that is zero on both boundaries, and its r-derivatives up to `orders`."""
    k = torch.arange(1, modes + 1, dtype=RD, device=sh.dev)[:, None]
    c = _spectrum(sh, gen, modes, amp) * (k[:, 0] ** -1.5)[None, :]
    x = (sh.prof["r"] - (1.0 / (1.0 - RADRATIO) - 1.0))[None, :]
    s, t, w = torch.sin(math.pi * k * x), torch.cos(math.pi * k * x), math.pi * k
    s[:, 0] = s[:, -1] = 0.0
    return [c @ b.to(CD) for b in (s, w * t, -w ** 2 * s, -w ** 3 * t)[:orders + 1]]


def _fields(sh, gen, chem=False):
    f = {}
    f["w"], f["dw"], f["ddw"], f["dddw"] = _field(sh, gen, 0.1)
    f["z"], f["dz"], f["ddz"], _ = _field(sh, gen, 3.0)
    f["s"], f["ds"], f["dds"], _ = _field(sh, gen, 1e-3)
    # the conducting shell between s = 1 inside and s = 0 outside, as the l = m = 0 mode
    r, r_cmb = sh.prof["r"], 1.0 / (1.0 - RADRATIO)
    c = math.sqrt(4.0 * math.pi) * (r_cmb - 1.0)
    f["s"][0] += c * (r_cmb / r - 1.0)
    f["ds"][0] -= c * r_cmb / r ** 2
    f["dds"][0] += 2.0 * c * r_cmb / r ** 3
    if sh.mag:
        f["b"], f["db"], f["ddb"], _ = _field(sh, gen, 1e-3)
        f["aj"], f["dj"], f["ddj"], _ = _field(sh, gen, 3e-3)
    if chem:
        f["xi"], f["dxi"], _, _ = _field(sh, gen, 1e-3)
    return f


STAGE_IN = ("w", "dw", "ddw", "z", "dz", "s")
STAGE_IN_MAG = ("b", "db", "ddb", "aj", "dj")


def _equations(sh):
    return (("s", "z", "w") + (("b", "j") if sh.mag else ()) + (("p",) if sh.cheb else ()))


def _step_inputs(sh, seed):
    """Fields and time arrays of a running step: the terms that the last step left."""
    gen = torch.Generator(device=sh.dev).manual_seed(int(seed))
    f = _fields(sh, gen)
    p, dp, _, _ = _field(sh, gen, 1e3)
    if sh.cheb:
        f["p"], f["dp"] = p, dp
    ta = {}
    for e, x, dx, d2x in (("s", "s", "ds", "dds"), ("z", "z", "dz", "ddz"),
                          ("b", "b", "db", "ddb"), ("j", "aj", "dj", "ddj")):
        if x in f:
            ta[e] = _generic_terms(sh, e, f[x], f[dx], f[d2x])
    if sh.cheb:
        ta["w"], ta["p"] = _wp_terms(sh, f)
        if not sh.anel:
            for e in ("w", "p"):
                x = ta[e]["impl"]
                x[0] = 0.0
                x[:, 0] = x[:, -1] = 0.0
    else:
        k = _matrices(sh)
        ta["w"] = _w_terms(sh, f, f["dddw"], f["ddw"] @ k["D2"].T.to(CD))
    for e in _equations(sh):
        size = float(ta[e]["impl"].abs().max()) + 1e-30
        for k in ("expl0", "expl1"):
            ta[e][k] = _field(sh, gen, size, orders=0)[0]
    return f, ta


def prepare(case, seed):
    from magic_b200 import Plan
    from magic_b200.step import AnelasticStep, BoussinesqStep

    sh = _Shell(case)
    if case["kind"] in ("sht", "stage"):
        key = (case["l_max"], case["minc"], case["precision"], str(sh.dev))
        if key not in _plans:
            _plans[key] = Plan(case["l_max"], case["minc"], precision=case["precision"])
        plan = _plans[key]
    gen = torch.Generator(device=sh.dev).manual_seed(int(seed))
    if case["kind"] == "sht":
        return dict(kind="sht", plan=plan, spec=_sht_inputs(sh, gen, case["cols"]))
    if case["kind"] == "stage":
        f = _fields(sh, gen, case["chem"])
        names = STAGE_IN + (STAGE_IN_MAG if sh.mag else ()) + (("xi",) if case["chem"] else ())
        size = plan.nl_anel_workspace if sh.anel else plan.nl_bouss_workspace
        own = sh.anel and case["precision"] == "fp64"  # composed: the stage makes its own
        work = None if own else torch.empty(max(1, size(sh.n_r, sh.mag, case["chem"])),
                                            dtype=torch.uint8, device=sh.dev)
        zero = lambda: torch.zeros(sh.lm_max, sh.n_r, dtype=CD, device=sh.dev)
        return dict(kind="stage", plan=plan, sh=sh, fields={k: f[k] for k in names},
                    chem=case["chem"], work=work,
                    out={k: zero() for k in _stage_names(sh, case["chem"])})
    f = sh.phys
    make = AnelasticStep if sh.anel else BoussinesqStep
    step = make(case["l_max"], sh.n_r, minc=case["minc"], ek=f["ek"], ra=f["ra"], pr=f["pr"],
                prmag=f["prmag"], dt=f["dt"], precision=case["precision"],
                radial_scheme=case["scheme"], cache=_shared)
    fields, ta = _step_inputs(sh, seed)
    for k, x in step.f.items():
        if k in fields:
            x.copy_(fields[k])
    for e in step.ta:
        for k, x in step.ta[e].items():
            x.copy_(ta[e][k])
    return dict(kind=case["kind"], step=step)


def _sht_inputs(sh, gen, cols):
    s = [_spectrum(sh, gen, cols) for _ in range(4)]
    for x in s[2:]:
        x[0] = 0.0  # no l = 0 in the horizontal potentials
    return [x[:, 0].contiguous() if cols == 1 else x for x in s]


def _stage_names(sh, chem):
    return (("Advr", "Advt", "Advp", "VSr", "VSt") + (("VxBr", "VxBt", "VxBp") if sh.mag else ())
            + (("VXir", "VXit") if chem else ()) + (("heat",) if sh.anel else ()))


def run(state):
    if state["kind"] == "sht":
        plan, (x, q, s, t) = state["plan"], state["spec"]
        grid = plan.scal_to_spat(x)
        if x.dim() == 1:
            return dict(grid=grid, back=plan.scal_to_SH(grid))
        br, bt, bp = plan.torpol_to_spat(q, s, t)
        bs, bj = plan.spat_to_sphertor(bt, bp)
        return dict(grid=grid, back=plan.scal_to_SH(grid), br=br, bt=bt, bp=bp, bs=bs, bj=bj)
    if state["kind"] == "stage":
        sh, plan = state["sh"], state["plan"]
        common = dict(l_mag=sh.mag, l_chem=state["chem"], out=state["out"], work=state["work"])
        if sh.anel:
            out, dtr, dth = plan.nl_anel(state["fields"], sh.prof, sh.LFfac, sh.visc_heat, sh.ohm,
                                         COURFAC, ALFFAC, sh.opm, **common)
        else:
            out, dtr, dth = plan.nl_bouss(state["fields"], sh.prof, sh.LFfac, COURFAC, ALFFAC,
                                          sh.opm, **common)
        return dict(out, dtr=dtr, dth=dth)
    step = state["step"]
    res = {}
    if state["kind"] == "lm":
        step.lm_loop()
    else:
        res["dtr"], res["dth"] = step.step()
    res.update(step.f)
    for e in step.ta:
        for k in ("old", "impl", "expl1"):
            res[e + "_" + k] = step.ta[e][k]
    return res


# ------------------------------------------------------------------ the work

def work(case):
    l_max, minc = case["l_max"], case["minc"]
    n_theta, n_phi, _ = _sizes(l_max, minc)
    lm = _lm_max(l_max, minc)
    leg = 4.0 * (n_theta // 2) * lm              # one complex column through one table, folded
    fft = 2.5 * n_theta * n_phi * math.log2(n_phi)
    spec, grid = 16.0 * lm, 8.0 * n_theta * n_phi
    if case["kind"] == "sht":
        n = case["cols"]
        if n == 1:
            return dict(bytes=2 * spec + grid, flops=2 * (leg + fft))
        return dict(bytes=n * (7 * spec + 4 * grid), flops=n * ((2 + 5 + 4) * leg + 7 * fft))
    n = case["n_r"]
    anel = case["anel"]
    mag = case.get("mag", not anel)
    chem = bool(case.get("chem"))
    n_in = 6 + 5 * mag + chem
    n_out = 5 + 3 * mag + 2 * chem + anel
    synth, fields = (21, 12) if anel else (11, 7)  # contractions and grids without b and xi
    ana, prods = (9, 7) if anel else (8, 6)
    synth, fields, ana, prods = (synth + 10 * mag + chem, fields + 6 * mag + chem,
                                 ana + 5 * mag + 3 * chem, prods + 3 * mag + 3 * chem)
    stage = dict(bytes=n * spec * (n_in + n_out),
                 flops=n * (leg * (synth + ana) + fft * (fields + prods)))
    if case["kind"] == "stage":
        return stage
    cheb = case["scheme"] != "FD"
    eqs = 2 + 2 * mag                            # equations of one field each
    lm_bytes = n * spec * (9 * eqs + 2 * mag + (17 if cheb else 10))
    if cheb:  # one dense n x n solve per field, one 2n x 2n solve, dense derivatives
        lm_bytes += 8.0 * (l_max + 1) * n * n * (eqs + 4)
        lm_flops = 4.0 * lm * n * n * (3 * eqs + 4 + 4)
    else:
        lm_flops = 4.0 * lm * n * (eqs * 20 + 50)
    if case["kind"] == "lm":
        return dict(bytes=lm_bytes, flops=lm_flops)
    # the explicit terms read the stage's outputs and six fields, and write one array an equation
    td = n * spec * (n_out + 5 + eqs + (2 if cheb else 1))
    return dict(bytes=stage["bytes"] + td + lm_bytes, flops=stage["flops"] + lm_flops)


# ------------------------------------------------- the same in plain FP64 torch

def exact(case, seed):
    sh = _Shell(case)
    gen = torch.Generator(device=sh.dev).manual_seed(int(seed))
    if case["kind"] == "sht":
        return _exact_sht(sh, _sht_inputs(sh, gen, case["cols"]))
    if case["kind"] == "stage":
        out, dtr, dth = _exact_stage(sh, _fields(sh, gen, case["chem"]), case["chem"])
        return dict(out, dtr=dtr, dth=dth)
    f, ta = _step_inputs(sh, seed)
    res = {}
    if case["kind"] == "step":
        nl, res["dtr"], res["dth"] = _exact_stage(sh, f, False)
        for e, x in _exact_td(sh, f, nl).items():
            ta[e]["expl0"] = x
        del nl
    res.update(_exact_lm(sh, f, ta))
    return res


class _Horizontal:
    """Gauss-Legendre points and the tables P, sin dP/dtheta as (n_m, l_max + 1, n_theta / 2)."""

    def __init__(self, sh):
        self.sh = sh
        x, w = np.polynomial.legendre.leggauss(sh.n_theta)
        for _ in range(2):  # Newton on P_n, and the weights of the polished nodes
            p0, p1 = np.ones_like(x), x.copy()
            for j in range(2, sh.n_theta + 1):
                p0, p1 = p1, ((2 * j - 1) * x * p1 - (j - 1) * p0) / j
            dp = sh.n_theta * (x * p1 - p0) / (x * x - 1.0)
            x = x - p1 / dp
        w = 2.0 / ((1.0 - x * x) * dp * dp)
        nh = sh.n_theta // 2
        x, w = x[::-1][:nh].copy(), w[::-1][:nh].copy()
        dev = sh.dev
        c = torch.as_tensor(x, device=dev)[None, :]
        s = torch.sqrt((1.0 - c) * (1.0 + c))
        self.cos, self.sin, self.w = c[0], s[0], torch.as_tensor(2.0 * math.pi * w, device=dev)
        m = torch.arange(0, sh.l_max + 1, sh.minc, dtype=RD, device=dev)[:, None]
        # sqrt(prod_{k <= m} (2k + 1) / (2k)) / sqrt(4 pi)
        k = torch.arange(1, sh.l_max + 1, dtype=RD, device=dev)
        nrm = torch.cat((torch.zeros(1, dtype=RD, device=dev),
                         torch.cumsum(torch.log1p(0.5 / k), 0)))
        start = torch.exp(0.5 * nrm[m[:, 0].long()])[:, None] / math.sqrt(4 * math.pi) * s ** m
        P = torch.zeros(m.shape[0], sh.l_max + 2, nh, dtype=RD, device=dev)
        root = lambda v: torch.sqrt(torch.clamp(v, min=0.0))
        for l in range(sh.l_max + 2):
            p1 = P[:, l - 1] if l else torch.zeros_like(start)
            p2 = P[:, l - 2] if l > 1 else torch.zeros_like(start)
            d = torch.clamp((l - m) * (l + m), min=1.0)
            a = root((2.0 * l - 1) * (2.0 * l + 1) / d)
            b = root((2.0 * l + 1) * (l + m - 1) * (l - m - 1) / d / max(2.0 * l - 3, 1.0))
            P[:, l] = torch.where(m == l, start, torch.where(m < l, a * c * p1 - b * p2, 0.0))
        l = torch.arange(sh.l_max + 2, dtype=RD, device=dev)[None, :]
        cl = torch.where(l > m, root((l + m) * (l - m)) / root((2 * l - 1) * (2 * l + 1)), 0.0)
        up = (l[:, :-1] * cl[:, 1:])[..., None] * P[:, 1:]
        up[:, 1:] -= ((l[:, 1:-1] + 1) * cl[:, 1:-1])[..., None] * P[:, :-2]
        self.dP = torch.where((l >= m)[:, :-1, None], up, 0.0)
        self.P = P[:, :-1].contiguous()
        self.odd = ((l - m)[:, :-1].long() % 2 == 1)[..., None]
        self.im = 1j * m[:, :, None].to(CD)
        at = torch.zeros(m.shape[0], sh.l_max + 1, dtype=torch.long, device=dev)
        at[sh.m // sh.minc, sh.l] = torch.arange(sh.lm_max, device=dev)
        self.at, self.valid = at, (l >= m)[:, :-1, None]
        self.ost2 = torch.repeat_interleave(1.0 / self.sin ** 2, 2)[None, :, None]
        both = torch.stack((self.cos, -self.cos), 1).reshape(-1)
        self.cosn = both[None, :, None] * self.ost2

    def _mul(self, T, X):
        return torch.view_as_complex(torch.bmm(T, torch.view_as_real(X).reshape(
            X.shape[0], X.shape[1], -1)).reshape(X.shape[0], T.shape[1], -1, 2))

    def synth(self, terms):
        """Rows (n_m, n_theta, B), interleaved north and south, of the sum of c T X."""
        F = 0.0
        for T, c, X in terms:
            X = torch.where(self.valid, X[self.at], 0.0)
            tab = (self.P if T == "P" else self.dP).transpose(1, 2)
            E = self._mul(tab, torch.where(self.odd, 0.0, X))
            O = self._mul(tab, torch.where(self.odd, X, 0.0))
            S = E - O if T == "P" else O - E
            F = F + c * torch.stack((E + O, S), 2).reshape(E.shape[0], -1, E.shape[2])
        return F

    def grid(self, *terms):
        n = self.sh.n_phi
        F = self.synth(terms).permute(2, 1, 0)
        F = torch.nn.functional.pad(torch.view_as_real(F).contiguous(),
                                    (0, 0, 0, n // 2 + 1 - F.shape[2]))
        return torch.fft.irfft(torch.view_as_complex(F), n=n, dim=2, norm="forward")

    def modes(self, g):
        F = torch.fft.rfft(g, dim=2, norm="forward")[:, :, :self.sh.n_m]
        return F.permute(2, 1, 0)                 # (n_m, n_theta, B)

    def analyse(self, *terms):
        """(lm_max, B) of the sum over theta of c (weight T) F."""
        out = 0.0
        for T, c, F in terms:
            N, S = F[:, 0::2] * self.w[None, :, None], F[:, 1::2] * self.w[None, :, None]
            if T == "P":
                even, odd, tab = N + S, N - S, self.P
            else:
                even, odd, tab = N - S, N + S, self.dP
            out = out + c * torch.where(self.odd, self._mul(tab, odd), self._mul(tab, even))
        return out[self.sh.m // self.sh.minc, self.sh.l]

    def scalar(self, X):
        return self.grid(("P", 1.0, X))

    def vector(self, Q, S, T):
        S, T = S.clone(), T.clone()
        S[0] = T[0] = 0.0
        return (self.scalar(Q), self.grid(("dP", 1.0, S), ("P", self.im, T)),
                self.grid(("P", self.im, S), ("dP", -1.0, T)))

    def scalar_back(self, g):
        return self.analyse(("P", 1.0, self.modes(g)))

    def vector_back(self, vt, vp):
        t, p = self.modes(vt * self.ost2), self.modes(vp * self.ost2)
        inv = torch.where(self.sh.dL > 0, 1.0 / torch.clamp(self.sh.dL, min=1.0), 0.0)
        return (inv * self.analyse(("dP", 1.0, t), ("P", -self.im, p)),
                inv * self.analyse(("dP", -1.0, p), ("P", -self.im, t)))


def _exact_sht(sh, spec):
    H = _Horizontal(sh)
    if spec[0].dim() == 1:
        g = H.scalar(spec[0][:, None])
        return dict(grid=g[0], back=H.scalar_back(g)[:, 0])
    x, q, s, t = spec
    g = H.scalar(x)
    br, bt, bp = H.vector(q, s, t)
    bs, bj = H.vector_back(bt, bp)
    return dict(grid=g, back=H.scalar_back(g), br=br, bt=bt, bp=bp, bs=bs, bj=bj)


def _exact_stage(sh, f, chem):
    """The nonlinear stage in blocks of levels (the levels are independent)."""
    H = _Horizontal(sh)
    n = sh.n_r
    out = {k: torch.zeros(sh.lm_max, n, dtype=CD, device=sh.dev) for k in _stage_names(sh, chem)}
    lim = [torch.empty(n, dtype=RD, device=sh.dev) for _ in range(2)]
    per = max(1, int(4e8 / (8.0 * sh.n_theta * sh.n_phi)))
    for a in range(0, n, per):
        lev = slice(a, min(n, a + per))
        res, vr2, vh2 = _exact_levels(sh, H, {k: x[:, lev] for k, x in f.items()}, lev, chem)
        for k in out:
            out[k][:, lev] = res[k]
        for x, v, d in ((lim[0], vr2, "delxr2"), (lim[1], vh2, "delxh2")):
            x[lev] = torch.where(v > 0, torch.sqrt(sh.prof[d][lev] / torch.clamp(v, min=1e-300)), 1e10)
    for x in out.values():
        x[:, 0] = x[:, -1] = 0.0
    return out, lim[0], lim[1]


def _exact_levels(sh, H, f, lev, chem):
    P = {k: v[lev][:, None, None] for k, v in sh.prof.items()}
    r, or1, or2, or4, beta, orho1 = (P[k] for k in ("r", "or1", "or2", "or4", "beta", "orho1"))
    o2, dL, ost2, cosn = sh.prof["or2"][lev][None, :], sh.dL, H.ost2, H.cosn
    lf = sh.LFfac
    vr, vt, vp = H.vector(dL * f["w"], f["dw"], f["z"])
    inner = torch.ones(sh.n_r, dtype=RD, device=sh.dev)
    if sh.anel:  # the boundary levels' velocity is zero
        inner[0] = inner[-1] = 0.0
        vr, vt, vp = (x * inner[lev][:, None, None] for x in (vr, vt, vp))
    s = H.scalar(f["s"])
    out = {}
    LF = [0.0, 0.0, 0.0]
    if sh.mag:
        br, bt, bp = H.vector(dL * f["b"], f["db"], f["aj"])
        cbr, cbt, cbp = H.vector(dL * f["aj"], f["dj"], o2 * dL * f["b"] - f["ddb"])
        LF = [lf * ost2 * (cbt * bp - cbp * bt), lf * or4 * (cbp * br - cbr * bp),
              lf * or4 * (cbr * bt - cbt * br)]
    heat = 0.0
    if sh.anel:
        vrr, vtr, vpr = H.vector(dL * f["dw"], f["ddw"], f["dz"])
        cvr = H.scalar(dL * f["z"])
        vrt, vrp = H.grid(("dP", 1.0, dL * f["w"])), H.grid(("P", H.im, dL * f["w"]))
        im = 1j * sh.m.to(CD)[:, None]
        _, vtp, vpp = H.vector(0.0 * f["dw"], im * f["dw"], im * f["z"])
        vtp, vpp = vtp * ost2, vpp * ost2
        adv = (-or2 * orho1 * (vr * (vrr - (2 * or1 + beta) * vr)
                               + ost2 * (vt * (vrt - r * vt) + vp * (vrp - r * vp))),
               or4 * orho1 * (-vr * (vtr - beta * vt) + vt * (cosn * vt + vpp + vrr)
                              + vp * (cosn * vp - vtp)),
               or4 * orho1 * (-vr * (vpr - beta * vp) - vt * (vtp + cvr) - vp * vpp))
        e = (vrr - (2 * or1 + beta) * vr, cosn * vt + vpp + vrr - or1 * vr,
             vpp + cosn * vt + or1 * vr, 2 * vtp + cvr - 2 * cosn * vp,
             r * vtr - (2 + beta * r) * vt + or1 * vrt, r * vpr - (2 + beta * r) * vp + or1 * vrp)
        heat = sh.visc_heat * or4 * orho1 * P["otemp1"] * P["visc"] * (
            2 * (e[0] ** 2 + e[1] ** 2 + e[2] ** 2) + e[3] ** 2 + ost2 * (e[4] ** 2 + e[5] ** 2)
            - 2.0 / 3.0 * (beta * vr) ** 2)
        if sh.mag and sh.ohm:
            heat = heat + sh.ohm * P["lambda_"] * or2 * P["otemp1"] * (
                or2 * cbr ** 2 + ost2 * (cbt ** 2 + cbp ** 2))
        out["heat"] = H.scalar_back(heat)
        del vrr, vtr, vpr, cvr, vrt, vrp, vtp, vpp, e, heat
    else:
        cvr, cvt, cvp = H.vector(dL * f["z"], f["dz"], o2 * dL * f["w"] - f["ddw"])
        adv = (-ost2 * (cvt * vp - cvp * vt), -or4 * (cvp * vr - cvr * vp),
               -or4 * (cvr * vt - cvt * vr))
        del cvr, cvt, cvp
    out["Advr"] = H.scalar_back(adv[0] + LF[0])
    out["Advt"], out["Advp"] = H.vector_back(adv[1] + LF[1], adv[2] + LF[2])
    for x, a, b in ((s, "VSr", "VSt"),) + (((H.scalar(f["xi"]), "VXir", "VXit"),) if chem else ()):
        out[a] = H.scalar_back(vr * x)
        out[b] = H.vector_back(or2 * vt * x, or2 * vp * x)[0]
    if sh.mag:
        rho = orho1 if sh.anel else 1.0
        out["VxBr"] = H.scalar_back(rho * ost2 * (vt * bp - vp * bt))
        out["VxBt"], out["VxBp"] = H.vector_back(rho * or4 * (vp * br - vr * bp),
                                                 rho * or4 * (vr * bt - vt * br))
    big = lambda x: x.amax(dim=(1, 2))
    fr, fh = P["orho2"] * vr ** 2, (vt ** 2 + vp ** 2) * ost2 * P["orho2"]
    if not sh.mag:
        return out, big(COURFAC ** 2 * or4 * fr), big(COURFAC ** 2 * or2 * fh)
    ar, ah = br ** 2 * lf * orho1, (bt ** 2 + bp ** 2) * lf * ost2 * orho1
    q = (0.5 * (1.0 + sh.opm)) ** 2
    ar, ah = ar * ar / (ar + q / P["delxr2"]), ah * ah / (ah + q / P["delxh2"])
    return (out, big(or4 * (COURFAC ** 2 * fr + ALFFAC ** 2 * ar)),
            big(or2 * (COURFAC ** 2 * fh + ALFFAC ** 2 * ah)))


# -------------------------------------------------------- radial matrices

def _weights(z, x, m):
    """Weights at z of the derivatives 0..m from values at x: the columns of the solution of
    the moment equations, by Fornberg's recursion (Math. Comp. 51 (1988) 699)."""
    c = np.zeros((len(x), m + 1))
    c[0, 0] = 1.0
    a, d = 1.0, x[0] - z
    for i in range(1, len(x)):
        b, last, d = 1.0, d, x[i] - z
        for j in range(i):
            gap = x[i] - x[j]
            b *= gap
            if j == i - 1:
                prev = c[i - 1].copy()
                for k in range(m + 1):
                    c[i, k] = a * ((k * prev[k - 1] if k else 0.0) - last * prev[k]) / b
            old = c[j].copy()
            for k in range(m + 1):
                c[j, k] = (d * old[k] - (k * old[k - 1] if k else 0.0)) / gap
        a = b
    return c


def _matrices(sh):
    """Derivative matrices D1..D4 on grid values; on Chebyshev levels also the polynomials."""
    n, r = sh.n_r, sh.r
    if sh.cheb:
        x = np.cos(math.pi * np.arange(n) / (n - 1))
        T = np.zeros((4, n, n))
        T[0, :, 0], T[0, :, 1], T[1, :, 1] = 1.0, x, 2.0
        for c in range(2, n):  # d^k of T_c = 2 x T_{c-1} - T_{c-2}; dx/dr = 2
            for k in range(4):
                T[k, :, c] = 2 * x * T[k, :, c - 1] - T[k, :, c - 2] + (
                    4.0 * k * T[k - 1, :, c - 1] if k else 0.0)
        inv = np.linalg.inv(T[0])
        D = [T[k] @ inv for k in (1, 2, 3)]
        cos = 2.0 * np.cos(math.pi * (np.outer(np.arange(n), np.arange(n)) % (2 * n - 2)) / (n - 1))
        cos[:, 0] = 1.0
        cos[:, -1] = (-1.0) ** np.arange(n)
        mats = dict(T=T, C=cos / math.sqrt(2.0 * (n - 1)))
    else:
        D = [np.zeros((n, n)) for _ in range(4)]
        for j in range(n):
            for k in range(4):  # fourth order inside, one-sided second order at the ends
                half = 2 if k < 2 else 3
                if half <= j < n - half:
                    at = list(range(j - half, j + half + 1))
                else:
                    at = [i if j < n // 2 else n - 1 - i for i in range(3 + k)]
                w = _weights(0.0, np.array([r[i] - r[j] for i in at]), k + 1)
                D[k][j, at] = w[:, k + 1]
        mats = dict(D4=D[3])
    mats.update(D1=D[0], D2=D[1], D3=D[2])
    return {k: torch.as_tensor(v, device=sh.dev) for k, v in mats.items()}


# --------------------------------------------------- the terms of one time step

def _generic_terms(sh, e, x, dx, d2x):
    """old and implicit terms of the entropy, toroidal and magnetic equations."""
    or1, or2, beta, dbeta = (sh.row(k) for k in ("or1", "or2", "beta", "dbeta"))
    if e == "s":
        c1 = beta + sh.row("dLtemp0") + 2.0 * or1
        return dict(old=x.clone(), impl=sh.opr * (d2x + c1 * dx - sh.dL * or2 * x))
    size = sh.dL * or2
    if e == "z":
        return dict(old=size * x, impl=size * (d2x - beta * dx - (dbeta + 2 * beta * or1 + size) * x))
    return dict(old=size * x, impl=sh.opm * size * (d2x - size * x))


def _wp_terms(sh, f):
    or1, or2, beta, dbeta = (sh.row(k) for k in ("or1", "or2", "beta", "dbeta"))
    size = sh.dL * or2
    w, dw, ddw, dddw, p, dp = (f[k] for k in ("w", "dw", "ddw", "dddw", "p", "dp"))
    wt = dict(old=size * w, impl=-dp + beta * p + size * (
        ddw - beta / 3.0 * dw - (size + 4.0 / 3.0 * (dbeta + beta * or1)) * w)
        + sh.BuoFac * sh.row("rho0") * sh.row("rgrav") * f["s"])
    pt = dict(old=-size * dw, impl=size * p + size * (
        -dddw + beta * ddw + (size + dbeta + 2 * beta * or1) * dw
        - size * (2 * or1 + 2.0 / 3.0 * beta) * w))
    return wt, pt


def _w_terms(sh, f, dddw, ddddw):
    """Double-curl poloidal terms (finite differences, Boussinesq profiles)."""
    or1, or2 = sh.row("or1"), sh.row("or2")
    size = sh.dL * or2
    w, dw, ddw = f["w"], f["dw"], f["ddw"]
    old = size * (size * w - ddw)
    impl = sh.BuoFac * size * sh.row("rgrav") * f["s"] - size * (
        ddddw - 2 * size * ddw + 4 * sh.dL * or1 * or2 * dw + size * (size - 6 * or2) * w)
    for x in (old, impl):
        x[:, 0] = x[:, -1] = 0.0
    return dict(old=old, impl=impl)


def _exact_td(sh, f, nl):
    """Explicit terms from the stage's outputs, by equation."""
    D1 = _matrices(sh)["D1"].T.to(CD)
    l, m = sh.l.to(RD)[:, None], sh.m.to(RD)[:, None]
    clm = lambda k: torch.sqrt(torch.clamp((k + m) * (k - m), min=0.0)
                               / torch.clamp((2 * k - 1) * (2 * k + 1), min=1.0))
    lo, hi = clm(l), clm(l + 1)
    or1, or2, or4 = (sh.row(k) for k in ("or1", "or2", "or4"))
    last = (sh.l == sh.l_max)[:, None]
    up = lambda x: torch.where(last, 0.0, torch.roll(x, -1, 0))   # l + 1 at the same m
    dn = lambda x: torch.roll(x, 1, 0)                            # l - 1: factor 0 at l = m
    dL, im, cf = sh.dL, 1j * m.to(CD), 2.0 * sh.CorFac
    a3, s3 = l * (l + 2) * hi, (l - 1) * (l + 1) * lo
    a4, s4 = l * hi * (l + 1) * (l + 2), (l + 1) * lo * (l - 1) * l
    w, dw, ddw, z, dz = (f[k] for k in ("w", "dw", "ddw", "z", "dz"))

    def ends(x):
        x[:, 0] = x[:, -1] = 0.0
        return x

    out = {}
    if sh.cheb:
        out["w"] = ends(or2 * nl["Advr"] + cf * or1 * (
            im * dw + (l + 2) * hi * up(z) - (l - 1) * lo * dn(z)))
        out["p"] = ends(-dL * nl["Advt"] + cf * or2 * (
            -im * (dw + or1 * dL * w) + a3 * up(z) + s3 * dn(z)))
    else:
        x = dL * or4 * nl["Advr"] + cf * or2 * (
            im * (or2 * dL * w - ddw) + a3 * up(dz) + s3 * dn(dz)
            + or1 * (a4 * up(z) - s4 * dn(z)))
        x[0] = or2[0] * nl["Advr"][0] + cf * or1[0] * 2.0 * hi[0] * z[1]
        q = ends(-(sh.row("r") ** 2) * dL * nl["Advt"])
        out["w"] = ends(x) + or2 * (q @ D1)
    out["z"] = ends(dL * nl["Advp"] + cf * or2 * (
        im * z + a3 * up(dw) + s3 * dn(dw) + or1 * (a4 * up(w) - s4 * dn(w))))
    x = dL * nl["VSt"] - or2 * (nl["VSr"] @ D1)
    out["s"] = sh.row("orho1") * (x + nl["heat"]) if sh.anel else x
    if sh.mag:
        out["b"] = ends(dL * nl["VxBp"])
        q = -dL * nl["VxBt"] * sh.row("r") ** 2
        out["j"] = ends(dL * or4 * nl["VxBr"]) + or2 * (q @ D1)
    return out


def _solve(sh, A, rhs, cols=False):
    """Rows rhs (lm_max, N) through the matrices A (l_max + 1, N, N) of their degrees."""
    fr = 1.0 / A.abs().amax(dim=2)
    A = fr[:, :, None] * A
    fc = 1.0 / A.abs().amax(dim=1) if cols else torch.ones_like(fr)
    A = A * fc[:, None, :]
    n_l, N, M = sh.l_max + 1, rhs.shape[1], sh.m // sh.minc
    X = torch.zeros(n_l, sh.n_m, N, dtype=CD, device=sh.dev)
    X[sh.l, M] = rhs
    X = torch.view_as_real(fr[:, None, :] * X).permute(0, 2, 1, 3).reshape(n_l, N, -1).contiguous()
    X = torch.linalg.solve(A, X).reshape(n_l, N, sh.n_m, 2).permute(0, 2, 1, 3)
    X = fc[:, None, :] * torch.view_as_complex(X.contiguous())
    x = X[sh.l, M]
    x[sh.m0] = x[sh.m0].real.to(CD)
    return x


def _exact_lm(sh, f, ta):
    """The implicit updates S, Z, W (P), B, J: fields and time arrays afterwards."""
    k = _matrices(sh)
    n, dev = sh.n_r, sh.dev
    dt = sh.phys["dt"]
    wi, w_impl, e0, e1 = 0.6 * dt, 0.4 * dt, 1.5 * dt, -0.5 * dt
    rhs_of = lambda e: (ta[e]["old"] + w_impl * ta[e]["impl"] + e0 * ta[e]["expl0"]
                        + e1 * ta[e]["expl1"])
    l = torch.arange(sh.l_max + 1, dtype=RD, device=dev)[:, None, None]
    dL = l * (l + 1)
    col = lambda name: sh.prof[name][None, :, None]
    or1, or2, beta, dbeta = (col(c) for c in ("or1", "or2", "beta", "dbeta"))
    eye = torch.eye(n, dtype=RD, device=dev)
    R = [k["T"][i] for i in range(4)] if sh.cheb else [eye, k["D1"], k["D2"], k["D3"], k["D4"]]
    rn, bf = (math.sqrt(2.0 / (n - 1)), 0.5) if sh.cheb else (1.0, 1.0)
    bot, top = n - 1, 0
    DT = [k[c].T.to(CD) for c in ("D1", "D2", "D3")]
    res, new = {}, {}

    def keep(e, terms):
        res[e + "_old"], res[e + "_impl"] = terms["old"], terms["impl"]
        res[e + "_expl1"] = ta[e]["expl0"]

    def field(e, x, dx, d2x, A, rows, bval=0.0, l0=False):
        for i, v in rows.items():
            A[:, i] = v
        A[:, :, [0, -1]] *= bf
        q = rhs_of(e)
        q[:, 0] = q[:, -1] = 0.0
        q[0, -1] = bval
        if l0:  # degree 0: the right-hand side on finite differences, else zero
            A[0] = eye
            if sh.cheb:
                q[0] = 0.0
        y = _solve(sh, A, q)
        if sh.cheb:
            y = y @ k["C"].T.to(CD)
        new[x], new[dx] = y, y @ DT[0]
        second = y @ DT[1]
        if d2x:
            new[d2x] = second
        keep(e, _generic_terms(sh, e, y, new[dx], second))

    lap = dL * or2
    c1 = beta + col("dLtemp0") + 2.0 * or1
    wall = {top: rn * R[0][0], bot: rn * R[0][-1]}
    field("s", "s", "ds", None, rn * (R[0] - wi * sh.opr * (R[2] + c1 * R[1] - lap * R[0])), wall,
          bval=math.sqrt(4 * math.pi))
    free = {i: rn * (R[1][i] - (2 * sh.np["or1"][i] + sh.np["beta"][i]) * R[0][i])
            for i in (top, bot)}
    field("z", "z", "dz", None, rn * lap * (R[0] - wi * (
        R[2] - beta * R[1] - (lap + dbeta + 2 * beta * or1) * R[0])),
        free if sh.anel else wall, l0=True)
    if sh.anel:
        _angular_momentum(sh, new, res, k)
    if sh.cheb:
        _exact_wp(sh, k, R, rn, wi, rhs_of, ta, new, keep, DT)
    else:
        _exact_w(sh, k, wi, rhs_of, ta, new, keep, DT)
    if sh.mag:
        A = rn * lap * (R[0] - wi * sh.opm * (R[2] - lap * R[0]))
        lr = l[:, :, 0]
        field("b", "b", "db", "ddb", A.clone(), {
            top: rn * (R[1][0] + lr * sh.np["or1"][0] * R[0][0]),
            bot: rn * (R[1][-1] - (lr + 1) * sh.np["or1"][-1] * R[0][-1])}, l0=True)
        field("j", "aj", "dj", "ddj", A, wall, l0=True)
    res.update(new)
    return res


def _l0_forces(sh, s00, ta):
    """Right-hand side of the l = 0 pressure: buoyancy and the explicit radial force."""
    q = sh.prof["rho0"] * sh.BuoFac * sh.prof["rgrav"] * s00 + ta["w"]["expl0"][0].real
    q[0] = 0.0
    return q


def _radial_weights(sh, k):
    """Clenshaw-Curtis weights of the Chebyshev levels."""
    n = sh.n_r
    c = np.zeros(n)
    c[0::2] = [1.0 if i == 0 else -1.0 / ((i + 1.0) * (i - 1.0)) for i in range(0, n, 2)]
    c[[0, -1]] *= 0.5
    return 2.0 * math.sqrt(2.0 / (n - 1)) / 2.0 * torch.as_tensor(c, device=sh.dev) @ k["C"]


def _angular_momentum(sh, new, res, k):
    """Stress-free runs keep their angular momentum: a rigid rotation taken off z."""
    p = sh.prof
    r, rho = p["r"], p["rho0"]
    rw = _radial_weights(sh, k)
    a = rho * r ** 2
    da = rho * (2 * r + r ** 2 * p["beta"])
    d2a = rho * (2 + 4 * p["beta"] * r + (p["dbeta"] + p["beta"] ** 2) * r ** 2)
    inertia = float((rw * r ** 4 * rho).sum())
    terms = _generic_terms(sh, "z", torch.ones(sh.lm_max, 1, dtype=RD, device=sh.dev) * a,
                           torch.ones(sh.lm_max, 1, dtype=RD, device=sh.dev) * da,
                           torch.ones(sh.lm_max, 1, dtype=RD, device=sh.dev) * d2a)
    for m in (0, 1):
        at = torch.nonzero((sh.l == 1) & (sh.m == m))
        if not at.numel():
            continue
        i = int(at[0])
        c = (rw * r ** 2 * new["z"][i]).sum() / inertia
        new["z"][i] -= c * a
        new["dz"][i] -= c * da
        res["z_old"][i] -= c * terms["old"][i]
        res["z_impl"][i] -= c * terms["impl"][i]


def _exact_wp(sh, k, R, rn, wi, rhs_of, ta, new, keep, DT):
    """The coupled (w, p) equations on Chebyshev levels."""
    n, dev = sh.n_r, sh.dev
    l = torch.arange(sh.l_max + 1, dtype=RD, device=dev)[:, None, None]
    dL = l * (l + 1)
    col = lambda name: sh.prof[name][None, :, None]
    or1, or2, beta, dbeta = (col(c) for c in ("or1", "or2", "beta", "dbeta"))
    lap = dL * or2
    A = torch.zeros(sh.l_max + 1, 2 * n, 2 * n, dtype=RD, device=dev)
    A[:, :n, :n] = rn * lap * (R[0] - wi * (
        R[2] - beta / 3.0 * R[1] - (lap + 4.0 / 3.0 * (beta * or1 + dbeta)) * R[0]))
    A[:, :n, n:] = rn * wi * (R[1] - beta * R[0])
    A[:, n:, :n] = rn * lap * (-R[1] - wi * (
        -R[3] + beta * R[2] + (lap + dbeta + 2 * beta * or1) * R[1]
        - lap * (2 * or1 + 2.0 / 3.0 * beta) * R[0]))
    A[:, n:, n:] = -rn * wi * lap * R[0]
    for i in (0, n - 1):
        A[:, [i, n + i]] = 0.0
        A[:, i, :n] = rn * R[0][i]
        A[:, n + i, :n] = rn * (R[2][i] - (2 * sh.np["or1"][i] + sh.np["beta"][i]) * R[1][i]
                                if sh.anel else R[1][i])
    A[:, :, [0, n - 1, n, 2 * n - 1]] *= 0.5
    A[0] = torch.eye(2 * n, dtype=RD, device=dev)
    buoy = sh.row("rho0") * sh.row("rgrav")
    q = torch.cat((rhs_of("w") + wi * sh.BuoFac * buoy * new["s"], rhs_of("p")), 1)
    q[:, [0, n - 1, n, 2 * n - 1]] = 0.0
    q[0] = 0.0
    x = _solve(sh, A, q, cols=True)
    del A
    Ct = k["C"].T.to(CD)
    w, p = x[:, :n] @ Ct, x[:, n:] @ Ct
    # l = 0: the hydrostatic pressure
    B = rn * (R[1] - beta[0] * R[0])
    s00 = new["s"][0].real
    q0 = _l0_forces(sh, s00, ta)
    if sh.anel:  # the integral of the density perturbation in place of p = 0
        pr = sh.prof
        g = k["C"] @ (sh.visc_heat * sh.polind / pr["temp0"] * pr["r"] ** 2) * rn
        g[[0, -1]] *= 0.5
        j = np.arange(n, dtype=np.float64)
        d = [1.0 - (j[:, None] - j[None, :]) ** 2, 1.0 - (j[:, None] + j[None, :]) ** 2]
        K = sum(np.where(x != 0, 1.0 / np.where(x != 0, x, 1.0), 0.0) for x in d)
        K = np.where((j[:, None] + j[None, :]) % 2 == 0, 0.5 * rn * K, 0.0)
        B[0] = torch.as_tensor(K, device=dev) @ g
        q0[0] = (_radial_weights(sh, k) * pr["rho0"] * pr["r"] ** 2 * s00).sum()
    else:
        B[0] = rn * R[0][0]
    B[:, [0, -1]] *= 0.5
    p[0] = (k["C"] @ torch.linalg.solve(B, q0)).to(CD)
    new.update(w=w, dw=w @ DT[0], ddw=w @ DT[1], p=p, dp=p @ DT[0])
    wt, pt = _wp_terms(sh, dict(new, dddw=w @ DT[2]))
    if not sh.anel:
        for t in (wt, pt):
            t["impl"][0] = 0.0
            t["impl"][:, [0, -1]] = 0.0
    keep("w", wt)
    keep("p", pt)


def _exact_w(sh, k, wi, rhs_of, ta, new, keep, DT):
    """The double-curl poloidal equation on finite differences (Boussinesq, no-slip)."""
    n, dev = sh.n_r, sh.dev
    l = torch.arange(sh.l_max + 1, dtype=RD, device=dev)[:, None, None]
    dL = l * (l + 1)
    or1, or2 = sh.prof["or1"][None, :, None], sh.prof["or2"][None, :, None]
    lap = dL * or2
    eye = torch.eye(n, dtype=RD, device=dev)
    A = lap * (lap * eye - k["D2"]) + wi * lap * (
        k["D4"] - 2 * lap * k["D2"] + 4 * dL * or1 * or2 * k["D1"] + lap * (lap - 6 * or2) * eye)
    A[:, 0], A[:, 1], A[:, -2], A[:, -1] = eye[0], k["D1"][0], k["D1"][-1], eye[-1]
    A[0] = eye
    q = rhs_of("w") + wi * sh.BuoFac * sh.dL * sh.row("or2") * sh.row("rgrav") * new["s"]
    q[:, [0, 1, -2, -1]] = 0.0
    q[0] = 0.0
    w = _solve(sh, A, q, cols=True)
    new.update(w=w, dw=w @ DT[0], ddw=w @ DT[1])
    keep("w", _w_terms(sh, new, new["ddw"] @ DT[0], new["ddw"] @ DT[1]))
    # l = 0: the hydrostatic pressure, the last row a backward difference
    B = k["D1"].clone()
    gap = sh.r[-1] - sh.r[-2]
    B[0] = eye[0]
    B[-1, -1], B[-1, -2] = 1.0 / gap, -1.0 / gap
    q0 = _l0_forces(sh, new["s"][0].real, ta)
    p = torch.zeros(sh.lm_max, n, dtype=CD, device=dev)
    p[0] = torch.linalg.solve(B, q0).to(CD)
    new["p"] = p
