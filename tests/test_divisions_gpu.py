"""Divisions that leave the ordinary range: equal hybgen targets (the heat
diffusion divides by their difference, and the clamp takes the neighbour that
the infinite quotient's sign names) and infinite pressures."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import fimocn_subx_realtime_hera_apr2020_gb300 as F  # noqa: E402
from helpers import make_case, oracle_for, rel_l2  # noqa: E402

pytestmark = pytest.mark.gpu

HYB = ["us3d", "vs3d", "tr3d", "sdot", "ex3d", "dp3d", "pr3d"]
CNU = ["us3d", "vs3d", "u_edg", "v_edg", "dp_edg", "lp_edg", "dp3d", "pr3d", "ex3d", "dp_tdcy", "dpl_tdcy",
       "massfx", "ws3d"]


def test_equal_targets():
    th, dp = F.vertical_tables(38)
    th = th.copy()
    th[15:17] = th[14]  # quotients of both signs
    th[24] = th[23]
    grid, cfg, fields = make_case(glvl=3, nvl=38, ntra=5, dt=200.0, seed=7, thetac=th, dpsig=dp)
    o = oracle_for(grid, cfg)
    s = o.new_state(fields)
    NL = grid.nip * 38
    s["tr3d"][:NL] += np.random.default_rng(8).normal(0.0, 0.2, NL)
    dyc = F.Dycore(grid, cfg)
    g = {n: torch.from_numpy(s[n].copy()).cuda() for n in HYB}
    o.hybgen(4, *[s[n] for n in HYB])
    dyc.hybgen(4, None, *[g[n] for n in HYB])
    for n in ("us3d", "vs3d", "tr3d", "ex3d", "pr3d"):
        assert np.isfinite(s[n]).all(), n
        assert rel_l2(g[n].cpu().numpy(), s[n]) <= 1e-12, n


@pytest.mark.parametrize("value", [np.inf, -np.inf])
def test_infinite_pressures(value):
    """An infinite thickness tendency leaves the pressure and the vertical
    motion below it infinite, and the Exner function with them."""
    grid, cfg, fields = make_case(glvl=2, nvl=38, ntra=5, dt=200.0, seed=7)
    o = oracle_for(grid, cfg)
    s = o.init_state(o.new_state(fields))
    for its in (1, 2):
        o.abstart(its)
    dyc = F.Dycore(grid, cfg)
    dyc.set_ab(o.c.nf + 1, o.c.of + 1, o.c.vof + 1, o.c.ab1, o.c.ab2, o.c.ab3)
    for i in (3, 50, 120):
        s["dp_tdcy"].reshape(3, grid.nip, 38)[o.c.of, i, 20] = value
    g = {n: torch.from_numpy(s[n].copy()).cuda() for n in CNU}
    o.cnuity(*[s[n] for n in CNU])
    dyc.cnuity(2, *[g[n] for n in CNU])
    assert np.isinf(s["ws3d"]).any()
    for n in ("pr3d", "ex3d", "ws3d"):
        got = g[n].cpu().numpy()
        for kind in (np.isnan, np.isinf):
            assert np.array_equal(kind(s[n]), kind(got)), n
