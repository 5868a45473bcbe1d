"""Arrays with a lazy bit (x.conj() is a view of x's memory, and so is the imaginary
part of one): kernels read memory, so each entry point has to carry the bit out
first, and has to leave an array that it updates in place with the right values.
On the CPU what the argument helpers hand to the library; on the GPU every entry
point against its result for the resolved array, bit for bit (the same kernel on
the same values)."""

import ctypes as C
import types

import pytest
import torch

from magic_b200 import _lib
from magic_b200.plan import Plan
from magic_b200.radial import RadialOp

CD, RD = torch.complex128, torch.float64


def _neg(*shape, device="cpu"):
    """A contiguous real array with the negation bit."""
    return torch._neg_view(torch.randn(*shape, dtype=RD, device=device))


def test_arguments_are_read_as_values():
    p = object.__new__(Plan)
    p._h, p.device = None, torch.device("cpu")
    p.lm_max, p.n_theta_max, p.n_phi_max = 6, 4, 8
    for x in (torch.randn(6, 3, dtype=CD), torch.randn(6, dtype=CD)):
        y = p._spec(x.conj(), "x")[0]
        assert not y.is_conj() and torch.equal(y.view_as(x), x.conj())
    g = _neg(2, 4, 8)
    assert g.is_neg() and g.is_contiguous()
    for y in (p._grid(g, "g")[0], p._grids([g], 2, "g")[0]):
        assert not y.is_neg() and torch.equal(y, g)
    assert not p._prof(_neg(5), 5).is_neg()
    op = object.__new__(RadialOp)
    op._h, op.device, op.n_r = None, p.device, 3
    x = torch.randn(6, 3, dtype=CD)
    assert not op._rows(x.conj()).is_conj()


@pytest.mark.parametrize("rc", [0, 1])
def test_arrays_updated_in_place(monkeypatch, rc):
    """A call that doubles what it finds in memory (and fails for rc = 1)."""
    monkeypatch.setattr(_lib, "lib", lambda: types.SimpleNamespace(mt_last_error=lambda: b"no"))
    a, b = torch.randn(5, dtype=CD), torch.randn(5, dtype=CD).conj()
    want = (2 * a, 2 * b.resolve_conj())

    def call(pa, pb):
        for ptr in (pa, pb):
            m = (C.c_double * 10).from_address(ptr)
            for i in range(10):
                m[i] *= 2
        return rc

    if rc:
        with pytest.raises(_lib.MagicError):
            _lib.check_writes([a, b], call, a.data_ptr(), b.data_ptr())
    else:
        _lib.check_writes([a, b], call, a.data_ptr(), b.data_ptr())
    assert b.is_conj() and torch.equal(a, want[0]) and torch.equal(b, want[1])


# ------------------------------------------------------------------- on the GPU

L_MAX, N_R = 12, 5
ARGS = dict(nl_bouss=(200.0, 2.5, 1.0, 0.2), nl_anel=(200.0, 0.3, 0.2, 2.5, 1.0, 0.2))
FIELDS = ("w", "dw", "ddw", "z", "dz", "s", "b", "db", "ddb", "aj", "dj", "xi")


def _same(a, b):
    a, b = (x if isinstance(x, tuple) else (x,) for x in (a, b))
    assert all(torch.equal(x, y) for x, y in zip(a, b))


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "split"])
def test_transforms(precision):
    p = Plan(L_MAX, precision=precision)
    for shape in ((p.lm_max,), (p.lm_max, 3)):
        x, y, z = (torch.randn(shape, dtype=CD, device="cuda").conj() for _ in range(3))
        rx, ry, rz = (v.resolve_conj() for v in (x, y, z))
        for f in (p.scal_to_spat, p.scal_to_grad_spat, p.pol_to_grad_spat):
            _same(f(x), f(rx))
        _same(p.torpol_to_spat(x, y, z), p.torpol_to_spat(rx, ry, rz))
    g, h = (_neg(3, p.n_theta_max, p.n_phi_max, device="cuda") for _ in range(2))
    assert g.is_neg()
    rg, rh = g.resolve_neg(), h.resolve_neg()
    _same(p.scal_to_SH(g), p.scal_to_SH(rg))
    _same(p.spat_to_sphertor(g, h), p.spat_to_sphertor(rg, rh))


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "split", "ozaki"])
@pytest.mark.parametrize("name", ["nl_bouss", "nl_anel"])
def test_stages(name, precision):
    from magic_b200.profiles import anelastic_profiles

    p = Plan(L_MAX, precision=precision)
    prof = anelastic_profiles(N_R, L_MAX)
    f = {k: torch.randn(p.lm_max, N_R, dtype=CD, device="cuda").conj() for k in FIELDS}
    stage = lambda f, **kw: getattr(p, name)(f, prof, *ARGS[name], l_mag=True, l_chem=True, **kw)
    ref, dtr, dth = stage({k: v.resolve_conj() for k, v in f.items()})
    lazy = {k: torch.zeros(p.lm_max, N_R, dtype=CD, device="cuda").conj() for k in ref}
    for out in (None, lazy):
        got, a, b = stage(f, out=out)
        assert torch.equal(a, dtr) and torch.equal(b, dth)
        for k in ref:
            assert torch.equal(got[k], ref[k]), k


@pytest.mark.gpu
def test_explicit_terms_updates_and_energies():
    from magic_b200 import implicit as I
    from magic_b200.output import EnergyIntegrals

    p = Plan(L_MAX)
    new = lambda *s: torch.randn(*(s or (p.lm_max, N_R)), dtype=CD, device="cuda").conj()
    pos = lambda n: torch.rand(n, dtype=RD, device="cuda") + 0.5
    val = lambda d: {k: v.resolve_conj() for k, v in d.items()}
    D = [RadialOp(torch.randn(N_R, N_R, dtype=RD).numpy()) for _ in range(4)]
    sch = types.SimpleNamespace(D1=D[0], D2=D[1], D3=D[2])
    x = new()
    assert torch.equal(D[0](x), D[0](x.resolve_conj()))
    ins = {k: new() for k in ("Advr", "Advt", "Advp", "VSr", "VSt", "VxBr", "VxBt", "VxBp", "w",
                              "dw", "z")}
    prof = {k: pos(N_R) for k in ("r", "or1", "or2", "or4", "orho1", "beta", "dbeta", "visc",
                                  "dLvisc", "rgrav", "rho0")}
    ref = p.get_td(val(ins), prof, 3.0, D[0])
    for out in (None, {k: new() for k in ref}):
        got = p.get_td(ins, prof, 3.0, D[0], out=out)
        assert all(torch.equal(got[k], ref[k]) for k in ref)
    e = EnergyIntegrals(p, torch.linspace(1.5, 0.5, N_R), prof["or2"].cpu(), prof["orho1"].cpu(),
                        prof["r"].cpu())
    a = [new() for _ in range(3)]
    assert e.kin(*a) == e.kin(*(v.resolve_conj() for v in a))
    # in place: state, time arrays and results with the bit set
    W = (1.0, 0.3, 0.2, 0.7, -0.25)
    lm = p.l_max + 1
    coef = {k: pos(lm if k.endswith("_l") else N_R) for k in
            ("so_l", "so_r", "ia_l", "ia_r", "ib_r", "ic_r", "ic_l", "ic_r2")}
    ta = {f"{v}{k}": new() for v in "wp" for k in ("old", "impl", "expl0", "expl1")}
    f = {k: new() for k in ("x", "dx", "d2x", "p", "dp")}
    bot, s = new(p.lm_max), new()
    op = lambda n: I.LOp(torch.randn(lm, n, n, dtype=RD).numpy() / n)
    ops = op(N_R), op(2 * N_R)

    def run(ta, f, bot, s):
        t = [{k: ta[v + k] for k in ("old", "impl", "expl0", "expl1")} for v in "wp"]
        I.update_field(p, sch, ops[0], f["x"], f["dx"], t[0], W, coef, bot=bot, d2x=f["d2x"])
        I.update_wp(p, sch, ops[1], D[3], f["x"], f["dx"], f["d2x"], f["p"], f["dp"], *t, W, s,
                    prof, coef["so_l"], 1.5)
        I.update_poloidal_dc(p, sch, ops[0], D[3], f["x"], f["dx"], f["d2x"], f["p"], t[0], W, s,
                             prof, coef["so_l"], 1.5, wcoef=[prof["or1"]] * 5)

    rta, rf = val(ta), val(f)
    run(rta, rf, bot.resolve_conj(), s.resolve_conj())
    run(ta, f, bot, s)
    for k in ta:
        assert ta[k].is_conj() and torch.equal(ta[k], rta[k]), k
    for k in f:
        assert torch.equal(f[k], rf[k]), k
