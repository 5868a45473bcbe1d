"""The FP64 anelastic stage writes whatever output arrays its caller hands over:
none, contiguous ones, a row stride of its own, columns first, filled with
garbage; boundary columns come back zero.  Against the stage's own result in
fresh arrays (bit for bit: only the destination differs), which
tests/test_gpu_anel.py and tests/test_gpu_phi_fft.py compare with the oracle.
n_r = 3 is the smallest stage, 10 and 11 end a tile of eight columns."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_r", [3, 10, 11])
@pytest.mark.parametrize("mag,chem", [(False, False), (True, True)])
def test_output_layouts(n_r, mag, chem):
    from magic_b200 import Plan
    from magic_b200.profiles import anelastic_profiles

    l_max = 20
    p = Plan(l_max)
    prof = anelastic_profiles(n_r, l_max)
    g = torch.Generator(device="cuda").manual_seed(n_r)
    names = ["w", "dw", "ddw", "z", "dz", "s"] + (["b", "db", "ddb", "aj", "dj"] if mag else [])
    names += ["xi"] if chem else []
    f = {k: torch.randn(p.lm_max, n_r, dtype=torch.complex128, device="cuda", generator=g)
         for k in names}
    args = (200.0, 0.3, 0.2, 2.5, 1.0, 0.2)
    ref, dtr, dth = p.nl_anel(f, prof, *args, l_mag=mag, l_chem=chem)
    for x in ref.values():
        assert (x[:, 0] == 0).all() and (x[:, -1] == 0).all()
        assert n_r < 4 or x[:, 1:-1].abs().max() > 0
    new = lambda *shape: torch.full(shape, float("nan"), dtype=torch.complex128, device="cuda")
    layouts = dict(
        contiguous=lambda k: new(p.lm_max, n_r),
        wide=lambda k: new(p.lm_max, n_r + 5)[:, :n_r],
        columns=lambda k: new(n_r, p.lm_max).T,
        mixed=lambda k: new(p.lm_max, n_r + (3 if k == "heat" else 0))[:, :n_r])
    for name, make in layouts.items():
        out = {k: make(k) for k in ref}
        got, a, b = p.nl_anel(f, prof, *args, l_mag=mag, l_chem=chem, out=out)
        assert torch.equal(a, dtr) and torch.equal(b, dth)
        for k in ref:
            assert got[k] is out[k] and torch.equal(out[k], ref[k]), (name, k)
