"""The FP64 Legendre kernels at the edges of their tiles, against the oracle: odd
and even numbers of theta pairs (75 and 72: 8- and 16-byte table copies, a last
tile of 11 or 8 of 32), column counts around the tiles of 4, 8 and 16, orders
with fewer degrees than a ring of chunks holds, and the fused stages' synthesis
(l(l+1) factors and the curl's difference on fragments) on a last tile of one and
of three columns.  Tolerance 1e-12 of scale, as for the other FP64 transforms."""

import numpy as np
import pytest
import torch

from conftest import rel_err
from oracle import grid as og
from oracle import sht as osht
from oracle import stage as ostage

pytestmark = pytest.mark.gpu

TOL = 1e-12
PAIR = {"Advt": "Advp", "Advp": "Advt", "VxBt": "VxBp", "VxBp": "VxBt"}


def _spec(g, n, rng):
    x = rng.standard_normal((g.lm_max, n)) + 1j * rng.standard_normal((g.lm_max, n))
    x *= ((g.lm2l + 1.0) ** -1.5)[:, None]
    x[g.lm2m == 0] = x[g.lm2m == 0].real
    return x


@pytest.mark.parametrize("l_max,minc,nhs", [(100, 1, 75), (96, 4, 72)])
@pytest.mark.parametrize("cols", [1, 4, 5, 17])
def test_transforms(l_max, minc, nhs, cols):
    from magic_b200 import Plan

    g, p = og.Grid(l_max, minc), Plan(l_max, minc)
    assert p.nhs == nhs
    rng = np.random.default_rng(l_max + cols)
    cu = lambda x: torch.as_tensor(np.ascontiguousarray(x)).cuda()
    npy = lambda x: x.cpu().numpy()
    Q, S, T = (_spec(g, cols, rng) for _ in range(3))
    sc = osht.scal_to_spat(g, Q)
    assert rel_err(npy(p.scal_to_spat(cu(Q))), sc) < TOL
    for fun in ("scal_to_grad_spat", "pol_to_grad_spat"):
        for a, b in zip(getattr(p, fun)(cu(Q)), getattr(osht, fun)(g, Q)):
            assert rel_err(npy(a), b) < TOL
    ref = osht.torpol_to_spat(g, Q, S, T)
    for a, b in zip(p.torpol_to_spat(cu(Q), cu(S), cu(T)), ref):
        assert rel_err(npy(a), b) < TOL
    assert rel_err(npy(p.scal_to_SH(cu(sc))), osht.scal_to_SH(g, sc)) < TOL
    want = osht.spat_to_sphertor(g, ref[1], ref[2])
    scale = max(np.abs(x).max() for x in want)
    for a, b in zip(p.spat_to_sphertor(cu(ref[1]), cu(ref[2])), want):
        assert np.abs(npy(a) - b).max() < TOL * scale


@pytest.mark.parametrize("l_max,n_r", [(100, 5), (48, 3)])
def test_stage(l_max, n_r):
    from magic_b200 import Plan

    g, p = og.Grid(l_max), Plan(l_max)
    rng = np.random.default_rng(l_max)
    names = ["w", "dw", "ddw", "z", "dz", "s", "b", "db", "ddb", "aj", "dj", "xi"]
    f = {k: _spec(g, n_r, rng) for k in names}
    prof = ostage.bouss_profiles(n_r, l_max=l_max)
    cu = lambda x: torch.as_tensor(np.ascontiguousarray(x)).cuda()
    args = (200.0, 2.5, 1.0, 0.2)
    ref, rdt, rdh = ostage.nl_bouss_stage(g, f, prof, *args, True, True)
    out, dt, dh = p.nl_bouss({k: cu(v) for k, v in f.items()}, {k: cu(v) for k, v in prof.items()},
                             *args, l_mag=True, l_chem=True)
    for k in ref:
        scale = max(np.abs(ref[j]).max() for j in (k, PAIR.get(k, k)))
        assert np.abs(out[k].cpu().numpy() - ref[k]).max() < TOL * scale, k
    assert rel_err(dt.cpu().numpy(), rdt) < TOL and rel_err(dh.cpu().numpy(), rdh) < TOL
