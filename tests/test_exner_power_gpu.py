"""The FP64 build's Exner function (cnuity) and the column remap's pressures
from it against extended precision, column heights that split the remap's warps
and blocks unevenly, and columns with massless layers."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import fimocn_subx_realtime_hera_apr2020_gb300 as F  # noqa: E402
from helpers import make_case, oracle_for, rel_l2  # noqa: E402

pytestmark = pytest.mark.gpu

CP, RD = 1004.6855, 287.0586


def _dev(a, dtype=torch.float64):
    return torch.from_numpy(np.ascontiguousarray(a)).to(device="cuda", dtype=dtype)


def test_exner_power():
    """exner = cp (p / p0)^(rd/cp) over p = 30 Pa .. 1100 hPa: two roundings
    (quotient, product) and a power within an ulp: 4 x 2^-53."""
    grid, cfg, fields = make_case(glvl=4, nvl=38, ntra=5, dt=100.0, seed=6, sigma_ps=2000.0)
    o = oracle_for(grid, cfg)
    s = o.init_state(o.new_state(fields))
    dyc = F.Dycore(grid, cfg)
    dyc.set_ab(1, 3, 2, cfg.dt, 0.0, 0.0)
    names = ["us3d", "vs3d", "u_edg", "v_edg", "dp_edg", "lp_edg", "dp3d", "pr3d", "ex3d", "dp_tdcy", "dpl_tdcy",
             "massfx", "ws3d"]
    g = {n: _dev(s[n]) for n in names}
    dyc.cnuity(1, *[g[n] for n in names])
    p = g["pr3d"].cpu().numpy().reshape(grid.nip, -1)[:, :-1].astype(np.longdouble)
    ex = g["ex3d"].cpu().numpy().reshape(grid.nip, -1)[:, :-1].astype(np.longdouble)
    assert p.min() < 400.0 and p.max() > 1.0e5
    want = np.longdouble(CP) * (p / np.longdouble(1.0e5)) ** np.longdouble(RD / CP)
    if np.finfo(np.longdouble).eps < 1e-17:  # extended precision on this machine
        assert float(np.abs(ex / want - 1).max()) <= 4 * 2.0 ** -53


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("glvl,nvl", [(1, 38), (2, 20), (3, 64), (2, 100), (4, 33)])
def test_column_adjustment(glvl, nvl, precision):
    """hybgen after a perturbation on columns of 1, 2 and 4 levels a lane, one
    and two columns a warp, grids whose last warp and block are partly idle."""
    kw = {}
    if nvl != 38:
        th, dp = F.vertical_tables(64)
        at = np.linspace(0.0, 63.0, nvl)
        kw = dict(thetac=np.interp(at, np.arange(64.0), th), dpsig=np.interp(at, np.arange(64.0), dp) * 64.0 / nvl)
    grid, cfg, fields = make_case(glvl=glvl, nvl=nvl, ntra=5, dt=200.0, seed=7, **kw)
    o = oracle_for(grid, cfg)
    s = o.new_state(fields)
    NL = grid.nip * nvl
    rng = np.random.default_rng(8)
    s["tr3d"][:NL] += rng.normal(0.0, 0.2, NL)
    gcfg = F.FimConfig(**{k: getattr(cfg, k) for k in cfg.__dataclass_fields__})
    gcfg.precision = precision
    dt = torch.float64 if precision == "f64" else torch.float32
    dyc = F.Dycore(grid, gcfg)
    names = ["us3d", "vs3d", "tr3d", "sdot", "ex3d", "dp3d", "pr3d"]
    if precision == "f32":  # both start from the rounded columns
        for n in names:
            s[n][:] = s[n].astype(np.float32)
    # FP32 interface pressures are up to 2^-7 Pa apart: an interface is off by
    # that at each of its three steps (old, smoothed, new), which moves the
    # same share of a layer's value into the next one
    tol = 1e-12 if precision == "f64" else 3 * 2.0 ** -7 / s["dp3d"][s["dp3d"] > 1.0].min()
    g = {n: _dev(s[n], dt) for n in names}
    o.hybgen(4, *[s[n] for n in names])
    dyc.hybgen(4, None, *[g[n] for n in names])
    for n in ("us3d", "vs3d", "tr3d", "ex3d", "pr3d"):
        assert rel_l2(g[n].double().cpu().numpy(), s[n]) <= tol, n
