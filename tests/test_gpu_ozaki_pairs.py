"""The digit-split GEMMs sum their accumulator groups through int32 pairs up to
800 terms a sum and in FP64 above (ozaki.cu): the stage on either side of that
line, for the synthesis (one term per degree: l_max 799, 800) and for the analysis
(one per theta pair: 800 and 804 of them on a refined colatitude grid), against
the FP64 plan's stage.  A sum that wrapped around would be off by 2^32 units of
its last pair, many orders above the tolerance: that of the digit-split stage,
5e-13 l_max^2 of scale, written with n_theta = 1.5 l_max, as what sets it is the
1/sin^2 weight of the polar rows."""

import pytest
import torch

from oracle import stage as ostage

pytestmark = pytest.mark.gpu

PAIR = {"Advt": "Advp", "Advp": "Advt"}


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
