"""The digit-split GEMMs sum their accumulator groups through int32 pairs up to
800 terms a sum and in FP64 above (ozaki.cu).

The sums themselves on group words as large as 800 terms make them, where a limit
set too high would wrap an int32: both against the integer sum rounded once, bit
for bit.

The stage on either side of the line, for the synthesis (one term per degree:
l_max 799, 800) and for the analysis (one per theta pair: 800 and 804 of them on a
refined colatitude grid), against the FP64 plan's stage: that both forms of the
kernels run there and are as accurate as the digit-split stage is, 5e-13 l_max^2
of scale, written with n_theta = 1.5 l_max, as what sets it is the 1/sin^2 weight
of the polar rows.  (The terms' signs vary, so these sums stay far below the
largest.)"""

import ctypes as C
import itertools

import pytest
import torch

from oracle import stage as ostage

pytestmark = pytest.mark.gpu

PAIR = {"Advt": "Advp", "Advp": "Advt"}


def test_group_sums_at_the_pair_limit():
    from magic_b200 import _lib

    L = _lib.lib()

    def run(rows):
        g = torch.tensor(rows, dtype=torch.int32, device="cuda")
        a, b = (torch.empty(len(rows), dtype=torch.float64, device="cuda") for _ in range(2))
        terms = C.c_int(0)
        _lib.check(L.mt_selftest_oz_combine(g.data_ptr(), len(rows), a.data_ptr(), b.data_ptr(),
                                            C.byref(terms), None))
        torch.cuda.synchronize()
        return a.tolist(), b.tolist(), terms.value

    terms = run([[0] * 6])[2]
    top = [(g + 1) * 4096 * terms for g in range(6)]  # digits up to 64, g + 1 pairs of them
    assert terms == 800 and max(top) < 2 ** 31
    rows = [[s * t for s, t in zip(sign, top)] for sign in itertools.product((1, -1), repeat=6)]
    gen = torch.Generator().manual_seed(6)
    for _ in range(2000):
        f = (2 * torch.rand(6, dtype=torch.float64, generator=gen) - 1) ** 3
        rows.append([int(x * t) for x, t in zip(f.tolist(), top)])
    paired, plain, _ = run(rows)
    for r, a, b in zip(rows, paired, plain):
        exact = float(sum(c << (7 * (5 - g)) for g, c in enumerate(r)))  # rounded once
        assert a == b == exact, r


@pytest.mark.parametrize("l_max,minc,n_theta,n_phi",
                         [(799, 8, 0, 0), (800, 8, 0, 0), (48, 1, 1600, 144), (48, 1, 1608, 144)])
def test_group_sums_either_side_of_the_pair_limit(l_max, minc, n_theta, n_phi):
    from magic_b200 import Plan

    n_r = 3
    make = lambda prec: Plan(l_max, minc, precision=prec, n_theta_max=n_theta, n_phi_max=n_phi)
    p, q = make("ozaki"), make("fp64")
    g = torch.Generator(device="cuda").manual_seed(l_max + n_theta)
    amp = (torch.as_tensor(p.lm2l).cuda().double() + 1.0) ** -1.5
    f = {}
    for k in ("w", "dw", "ddw", "z", "dz", "s"):
        x = torch.randn(p.lm_max, n_r, dtype=torch.complex128, device="cuda", generator=g)
        f[k] = x * amp[:, None]
    prof = {k: torch.as_tensor(v).cuda() for k, v in ostage.bouss_profiles(n_r, l_max=l_max).items()}
    args = (200.0, 2.5, 1.0, 0.2)
    got, dtr, dth = p.nl_bouss(f, prof, *args, l_mag=False, l_chem=False)
    ref, rdt, rdh = q.nl_bouss(f, prof, *args, l_mag=False, l_chem=False)
    torch.cuda.synchronize()
    p.poll_status(block=True)
    tol = 5e-13 * (p.n_theta_max / 1.5) ** 2
    for k in ref:
        scale = max(ref[j].abs().max().item() for j in (k, PAIR.get(k, k)))
        assert scale > 0 and (got[k] - ref[k]).abs().max().item() < tol * scale, k
    assert ((dtr - rdt).abs().max() / rdt.abs().max()).item() < tol
    assert ((dth - rdh).abs().max() / rdh.abs().max()).item() < tol
