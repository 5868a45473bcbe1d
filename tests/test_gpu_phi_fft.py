"""The row FFTs of the phi stages (magic_b200/csrc/phi_fft.cuh) at every row
length the plan accepts: all even n_phi = 2^a 3^b 5^c up to 1168, so every radix
and every pair, F = 1 (odd half length) included, full spectra (n_m up to
n_phi / 2) and short ones.

Drop-in transforms on a grid of four colatitudes against torch's FFT of the
same Fourier rows in FP64 on the host: a coefficient passes through
log2(n_phi) <= 11 butterfly levels of rounding error eps each, and the Legendre
sums of at most n_phi / 2 terms add eps sqrt(terms), so 1e-12 of the largest
value covers both by two orders of magnitude (FP32 rows: 2e-5, the split
transforms' bound).  The fused stages at row lengths outside their other tests
against the oracle, with those tests' tolerances."""

import numpy as np
import pytest
import torch

from oracle import grid as og
from oracle import stage as ostage

pytestmark = pytest.mark.gpu


def _smooth(n):
    for p in (2, 3, 5):
        while n % p == 0:
            n //= p
    return n == 1


SIZES = [n for n in range(4, 1170, 2) if _smooth(n)]


def _case(n_phi, precision, cols, rng, frac):
    from magic_b200 import Plan

    l_max = max(1, int((n_phi // 2 - 1) * frac))
    if precision == "split":
        l_max = min(l_max, 383)  # the largest the split tables are used at
    p = Plan(l_max, precision=precision, n_theta_max=4, n_phi_max=n_phi)
    P = p.tables()["Plm"].cpu().numpy()  # (lm_max, 2)
    X = rng.standard_normal((p.lm_max, cols)) + 1j * rng.standard_normal((p.lm_max, cols))
    X[p.lm2m == 0] = X[p.lm2m == 0].real
    return p, P, X


def _rows(p, P, X):
    """(n_m, 4, cols) Fourier rows, interleaved north and south."""
    F = np.zeros((p.n_m_max, 4, X.shape[1]), dtype=complex)
    sign = np.where((p.lm2l - p.lm2m) % 2 == 0, 1.0, -1.0)
    for mc in range(p.n_m_max):
        s = slice(p.lStart[mc], p.lStart[mc] + p.l_max - mc + 1)
        F[mc, 0::2] = P[s].T @ X[s]
        F[mc, 1::2] = P[s].T @ (sign[s, None] * X[s])
    return F


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("split", 2e-5)])
@pytest.mark.parametrize("n_phi", SIZES)
def test_rows_of_every_length(n_phi, precision, tol):
    rng = np.random.default_rng(n_phi)
    for cols, frac in ((3, 1.0), (9, 0.4)):
        p, P, X = _case(n_phi, precision, cols, rng, frac)
        F = torch.from_numpy(_rows(p, P, X))
        full = torch.zeros(n_phi // 2 + 1, 4, cols, dtype=torch.complex128)
        full[:p.n_m_max] = F
        ref = torch.fft.irfft(full, n=n_phi, dim=0, norm="forward").permute(2, 1, 0)
        got = p.scal_to_spat(torch.from_numpy(X).cuda()).cpu()
        assert (got - ref).abs().max() < tol * ref.abs().max(), (n_phi, cols)
        # analysis of rough grids: sum over the four rows of w P rfft
        g = torch.from_numpy(rng.standard_normal((cols, 4, n_phi)))
        G = torch.fft.rfft(g, dim=2, norm="forward")[:, :, :p.n_m_max].permute(2, 1, 0).numpy()
        w = 2 * np.pi * p.tables()["gauss"].cpu().numpy()[:2]
        ref = np.zeros((p.lm_max, cols), dtype=complex)
        for mc in range(p.n_m_max):
            s = slice(p.lStart[mc], p.lStart[mc] + p.l_max - mc + 1)
            sg = np.where((p.lm2l[s] - p.lm2m[s]) % 2 == 0, 1.0, -1.0)[:, None]
            N, S = G[mc, 0::2] * w[:, None], G[mc, 1::2] * w[:, None]
            ref[s] = P[s] @ N + sg * (P[s] @ S)
        back = p.scal_to_SH(g.cuda()).cpu().numpy()
        assert np.abs(back - ref).max() < tol * np.abs(ref).max(), (n_phi, cols)


# n_phi 30 (F = 1), 300 (15 x 5), 500 (25 x 5), 1000 (25 x 10)
STAGES = [(40, 4, 5, True, True), (100, 1, 4, True, False), (166, 1, 3, True, False),
          (333, 1, 3, False, False)]
PAIR = {"Advt": "Advp", "Advp": "Advt", "VxBt": "VxBp", "VxBp": "VxBt"}


@pytest.mark.parametrize("l_max,minc,N,l_mag,l_chem", STAGES)
@pytest.mark.parametrize("anel", [False, True])
def test_stages_at_other_row_lengths(l_max, minc, N, l_mag, l_chem, anel):
    from magic_b200 import Plan

    g = og.Grid(l_max, minc)
    rng = np.random.default_rng(l_max + N)
    amp = (g.lm2l + 1.0) ** -1.5
    names = ["w", "dw", "ddw", "z", "dz", "s"] + (["b", "db", "ddb", "aj", "dj"] if l_mag else [])
    f = {}
    for k in names + (["xi"] if l_chem else []):
        x = rng.standard_normal((g.lm_max, N)) + 1j * rng.standard_normal((g.lm_max, N))
        x *= amp[:, None]
        x[g.lm2m == 0] = x[g.lm2m == 0].real
        f[k] = x
    cu = lambda d: {k: torch.as_tensor(np.ascontiguousarray(v)).cuda() for k, v in d.items()}
    if anel:
        prof = ostage.anel_profiles(N, l_max=l_max)
        args = (200.0, 0.3, 0.2, 2.5, 1.0, 0.2)
        ref, rdt, _ = ostage.nl_anel_stage(g, f, prof, *args, l_mag, l_chem)
    else:
        prof = ostage.bouss_profiles(N, l_max=l_max)
        args = (200.0, 2.5, 1.0, 0.2)
        ref, rdt, _ = ostage.nl_bouss_stage(g, f, prof, *args, l_mag, l_chem)
    tols = {"fp64": 1e-12 if l_max <= 127 else 4e-12, "ozaki": 5e-13 * l_max ** 2,
            "split": 2e-5 if l_max <= 127 else 5e-5}
    for precision, tol in tols.items():
        p = Plan(l_max, minc, precision=precision)
        stage = p.nl_anel if anel else p.nl_bouss
        out, dt, _ = stage(cu(f), cu(prof), *args, l_mag=l_mag, l_chem=l_chem)
        p.poll_status(block=True)
        for k in ref:
            scale = max(np.abs(ref[k]).max(), np.abs(ref[PAIR.get(k, k)]).max())
            err = np.abs(out[k].cpu().numpy() - ref[k]).max() / scale
            assert err < tol, (precision, k, err)
        assert np.abs(dt.cpu().numpy() - rdt).max() < max(tol, 1e-12) * np.abs(rdt).max()


@pytest.mark.parametrize("anel", [False, True])
def test_compiled_shapes(anel):
    """The FP64 phi stages at every row length they compile in (512 to 1152, outer
    radix 16) against the run-time shape of n_phi 600: the products are quadratic, so
    at l_max 64 any n_phi above 192 gives the same spectra, to the stages' FP64 and
    digit-split tolerances."""
    from magic_b200 import Plan

    l_max, N = 64, 5
    rng = np.random.default_rng(16)
    make = lambda n, prec: Plan(l_max, precision=prec, n_theta_max=100, n_phi_max=n)
    q = make(600, "fp64")
    names = ("w", "dw", "ddw", "z", "dz", "s", "b", "db", "ddb", "aj", "dj", "xi")
    f = {}
    for k in names:
        x = rng.standard_normal((q.lm_max, N)) + 1j * rng.standard_normal((q.lm_max, N))
        x *= ((q.lm2l + 1.0) ** -1.5)[:, None]
        x[q.lm2m == 0] = x[q.lm2m == 0].real
        f[k] = torch.from_numpy(x).cuda()
    if anel:
        prof, args = ostage.anel_profiles(N, l_max=l_max), (200.0, 0.3, 0.2, 2.5, 1.0, 0.2)
    else:
        prof, args = ostage.bouss_profiles(N, l_max=l_max), (200.0, 2.5, 1.0, 0.2)
    prof = {k: torch.as_tensor(np.ascontiguousarray(v)).cuda() for k, v in prof.items()}
    run = lambda p, **kw: (p.nl_anel if anel else p.nl_bouss)(f, prof, *args, **kw)[0]
    for kw in (dict(l_mag=True, l_chem=False), dict(l_mag=False, l_chem=True)):
        ref = run(q, **kw)
        for n_phi in (512, 640, 768, 960, 1024, 1152):
            for precision, tol in (("fp64", 1e-12), ("ozaki", 5e-13 * l_max ** 2)):
                out = run(make(n_phi, precision), **kw)
                for k in ref:
                    scale = max(ref[j].abs().max().item() for j in (k, PAIR.get(k, k)))
                    err = (out[k] - ref[k]).abs().max().item()
                    assert err < tol * scale, (n_phi, precision, k, err / scale)


def test_longer_rows_are_refused():
    """1200 is the first length of factors 2, 3, 5 above the limit, which the error names."""
    from magic_b200 import MagicError, Plan

    with pytest.raises(MagicError, match=r"limit \(1168\)"):
        Plan(16, n_theta_max=24, n_phi_max=1200)
