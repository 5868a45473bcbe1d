"""The implicit updates with dense operators (magic_b200/csrc/implicit.cu) on either
side of every change of kernel or tile: n_r around multiples of the 8-level
n-tiles, of the 16-row chunks and of the limits of the tensor-pipe forms (72, 144
and 256 levels for a field, 72, 144 and 192 for the coupled (w, p) update), degrees
whose orders do not fill the 16 of a CTA, minc > 1.

Random well-scaled operators (entries ~ 1 / sqrt(n)), against the same formulas in
plain FP64 torch on the host.  Each value is a sum of n to 2 n products of order
1 / sqrt(n) followed by another such sum: rounding of either order is below
2 n eps ~ 1e-13 of the largest value, so 1e-12."""

import types

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
TOL = 1e-12
WEIGHTS = (1.0, 0.3, 0.2, 0.7, -0.25)  # w_old, w_impl_now, w_impl, w_expl0, w_expl1


def _setup(l_max, minc, n_r, seed):
    from magic_b200 import Plan
    from magic_b200.radial import RadialOp

    rng = np.random.default_rng(seed)
    plan = Plan(l_max, minc)
    mat = lambda n: rng.standard_normal((n, n)) / np.sqrt(n)
    D = [mat(n_r) for _ in range(3)]
    sch = types.SimpleNamespace(**{f"D{i + 1}": RadialOp(D[i]) for i in range(3)})
    cplx = lambda: torch.from_numpy(rng.standard_normal((plan.lm_max, n_r))
                                    + 1j * rng.standard_normal((plan.lm_max, n_r)))
    vec = lambda n: torch.from_numpy(rng.standard_normal(n))
    return rng, plan, [torch.from_numpy(d) for d in D], sch, cplx, vec


def _solve(plan, M, rhs):
    x = torch.stack([torch.from_numpy(M[l]).to(torch.complex128) @ rhs[i]
                     for i, l in enumerate(plan.lm2l)])
    m0 = torch.from_numpy(plan.lm2m == 0)
    x[m0] = x[m0].real.to(torch.complex128)
    return x


def _check(got, ref):
    for k in ref:
        err = (got[k].cpu() - ref[k]).abs().max().item()
        assert err <= TOL * max(ref[k].abs().max().item(), 1e-300), (k, err)


@pytest.mark.parametrize("l_max,minc", [(16, 1), (12, 2)])
@pytest.mark.parametrize("n_r", [3, 7, 8, 9, 16, 17, 33, 72, 73, 129, 144, 145, 256, 257])
def test_field_update(n_r, l_max, minc):
    from magic_b200 import implicit as I

    rng, plan, D, sch, cplx, vec = _setup(l_max, minc, n_r, 100 * n_r + l_max)
    M = rng.standard_normal((l_max + 1, n_r, n_r)) / np.sqrt(n_r)
    ta = {k: cplx() for k in ("old", "impl", "expl0", "expl1")}
    coef = {k: vec(l_max + 1 if k.endswith("_l") else n_r) for k in
            ("so_l", "so_r", "ia_l", "ia_r", "ib_r", "ic_r", "ic_l", "ic_r2")}
    bot = cplx()[:, 0].contiguous()
    w_old, _, wi, e0, e1 = WEIGHTS
    rhs = w_old * ta["old"] + wi * ta["impl"] + e0 * ta["expl0"] + e1 * ta["expl1"]
    rhs[:, 0], rhs[:, -1] = 0.0, bot
    x = _solve(plan, M, rhs)
    dx, d2x = x @ D[0].T.to(x.dtype), x @ D[1].T.to(x.dtype)
    L = torch.from_numpy(plan.lm2l)
    c = lambda l, r: coef[l][L][:, None] * coef[r][None, :]
    ref = dict(x=x, dx=dx, d2x=d2x, old=c("so_l", "so_r") * x, expl1=ta["expl0"],
               impl=c("ia_l", "ia_r") * (d2x + coef["ib_r"] * dx
                                         - (coef["ic_r"] + c("ic_l", "ic_r2")) * x))
    cu = lambda t: t.cuda()
    tg = {k: cu(v) for k, v in ta.items()}
    got = {k: torch.full_like(tg["old"], 7.0) for k in ("x", "dx", "d2x")}
    I.update_field(plan, sch, I.LOp(M), got["x"], got["dx"], tg, WEIGHTS,
                   {k: cu(v) for k, v in coef.items()}, bot=cu(bot), d2x=got["d2x"])
    _check(dict(got, old=tg["old"], impl=tg["impl"], expl1=tg["expl1"]), ref)


@pytest.mark.parametrize("interior", [False, True])
@pytest.mark.parametrize("n_r", [3, 8, 9, 33, 36, 37, 72, 73, 129, 144, 145, 193])
def test_wp_update(n_r, interior):
    from magic_b200 import implicit as I
    from magic_b200.radial import RadialOp

    l_max = 16
    rng, plan, D, sch, cplx, vec = _setup(l_max, 1, n_r, 10 * n_r + interior)
    M = rng.standard_normal((l_max + 1, 2 * n_r, 2 * n_r)) / np.sqrt(2 * n_r)
    M[0] = 0.0
    P0 = rng.standard_normal((n_r, n_r)) / np.sqrt(n_r)
    tw, tp = ({k: cplx() for k in ("old", "impl", "expl0", "expl1")} for _ in range(2))
    s = cplx()
    names = ("or1", "or2", "beta", "dbeta", "visc", "dLvisc", "rgrav", "rho0")
    P = {k: vec(n_r) for k in names}
    hd, buo = vec(l_max + 1), 1.7
    w_old, w0, wi, e0, e1 = WEIGHTS
    comb = lambda t: w_old * t["old"] + wi * t["impl"] + e0 * t["expl0"] + e1 * t["expl1"]
    rw, rp = comb(tw) + w0 * P["rho0"] * P["rgrav"] * buo * s, comb(tp)
    for r in (rw, rp):
        r[:, 0] = r[:, -1] = 0.0
    sol = _solve(plan, M, torch.cat((rw, rp), 1))
    w, p = sol[:, :n_r].clone(), sol[:, n_r:].clone()
    q = P["rho0"] * buo * P["rgrav"] * s[0].real + tw["expl0"][0].real
    q[0] = 0.0
    p[0] = (torch.from_numpy(P0) @ q).to(p.dtype)
    d = lambda x, i: x @ D[i].T.to(x.dtype)
    dw, ddw, dddw, dp = d(w, 0), d(w, 1), d(w, 2), d(p, 0)
    L = torch.from_numpy(plan.lm2l).double()[:, None]
    dLo = L * (L + 1) * P["or2"]
    or1, beta, dbeta, dLv = (P[k] for k in ("or1", "beta", "dbeta", "dLvisc"))
    f = hd[torch.from_numpy(plan.lm2l)][:, None] * dLo * P["visc"]
    w_impl = -dp + beta * p + f * (ddw + (2 * dLv - beta / 3) * dw - (
        dLo + 4 / 3 * (dbeta + dLv * beta + (3 * dLv + beta) * or1)) * w) \
        + buo * P["rho0"] * P["rgrav"] * s
    p_impl = dLo * p + f * (-dddw + (beta - dLv) * ddw + (
        dLo + dLv * beta + dbeta + 2 * (dLv + beta) * or1) * dw
        - dLo * (2 * or1 + 2 / 3 * beta + dLv) * w)
    if interior:
        for x in (w_impl, p_impl):
            x[0] = 0.0
            x[:, 0] = x[:, -1] = 0.0
    ref = dict(w=w, dw=dw, ddw=ddw, p=p, dp=dp, w_old=dLo * w, w_impl=w_impl,
               w_expl1=tw["expl0"], p_old=-dLo * dw, p_impl=p_impl, p_expl1=tp["expl0"])
    cu = lambda t: t.cuda()
    gw, gp = ({k: cu(v) for k, v in t.items()} for t in (tw, tp))
    got = {k: torch.full_like(gw["old"], 7.0) for k in ("w", "dw", "ddw", "p", "dp")}
    I.update_wp(plan, sch, I.LOp(M), RadialOp(P0), got["w"], got["dw"], got["ddw"], got["p"],
                got["dp"], gw, gp, WEIGHTS, cu(s), {k: cu(v) for k, v in P.items()}, cu(hd), buo,
                impl_interior=interior)
    got.update({f"w_{k}": gw[k] for k in ("old", "impl", "expl1")},
               **{f"p_{k}": gp[k] for k in ("old", "impl", "expl1")})
    _check(got, ref)


def _banded(rng, n):
    """A random operator with a band of two on either side (one-sided at the ends)."""
    D = np.zeros((n, n))
    for j in range(n):
        k = min(max(j - 2, 0), max(n - 5, 0))
        D[j, k:k + 5] = rng.standard_normal(min(5, n))
    return D


@pytest.mark.parametrize("n_r", [7, 16, 65, 128, 129, 192, 193])
def test_wp_update_banded_derivatives(n_r, monkeypatch):
    """Banded derivative operators take the other form of the coupled solve, with two
    limits (128 and 192 levels)."""
    dense = _setup

    def banded(l_max, minc, n, seed):
        from magic_b200.radial import RadialOp

        rng, plan, _, _, cplx, vec = dense(l_max, minc, n, seed)
        D = [_banded(rng, n) for _ in range(3)]
        sch = types.SimpleNamespace(**{f"D{i + 1}": RadialOp(D[i]) for i in range(3)})
        return rng, plan, [torch.from_numpy(d) for d in D], sch, cplx, vec

    monkeypatch.setitem(globals(), "_setup", banded)
    test_wp_update(n_r, False)


@pytest.mark.parametrize("n_r", [144, 145, 170, 171])
def test_field_update_on_few_waves(n_r):
    """l_max 64 is 165 CTAs: between one and three waves of SMs the derivatives of 145
    to 170 levels run by FMAs."""
    test_field_update(n_r, 64, 1)
