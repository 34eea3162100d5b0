"""The per-routine trcadv on the patch kernels: column heights and alignments
that take each level-vector width, small grids (the general staging loop, pole
patches), tracers of both signs and zero, AB3 weights, a member whose own
tracer count is smaller; against the CPU oracle."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import fimocn_subx_realtime_hera_apr2020_gb300 as F  # noqa: E402
from helpers import make_case, oracle_for, rel_l2  # noqa: E402

pytestmark = pytest.mark.gpu

NAMES = ["trc_edg", "tr3d", "trdp", "trc_tdcy", "trl_tdcy", "massfx", "dp3d"]


def _inputs(glvl, nvl, ntra):
    kw = {}
    if nvl != 38:
        th, dp = F.vertical_tables(64)
        kw = dict(thetac=th[:nvl], dpsig=dp[:nvl])
    grid, cfg, fields = make_case(glvl=glvl, nvl=nvl, ntra=ntra, dt=400.0, seed=77, **kw)
    o = oracle_for(grid, cfg)
    s = o.init_state(o.new_state(fields))
    N, L = grid.nip, nvl
    rng = np.random.default_rng(78)
    tr = s["tr3d"].reshape(ntra, N, L)
    tr[1:] = rng.uniform(-2e-3, 1e-2, (ntra - 1, N, L))  # the bounds' clamp at zero acts
    tr[2] = 0.0                                           # zero fluxes, zero sums
    s["trdp"][:ntra * N * L] = (tr * s["dp3d"].reshape(1, N, L)).ravel()
    for _ in range(3):  # AB3 weights, three filled slots
        its = _ + 1
        o.abstart(its)
        o.edgvar1(s["us3d"], s["vs3d"], s["dp3d"], s["pr3d"], s["ex3d"], s["ph3d"], s["mp3d"], s["tr3d"],
                  s["u_edg"], s["v_edg"], s["dp_edg"], s["lp_edg"], s["geop_edg"], s["mont_edg"], s["uvsq_edg"],
                  s["trc_edg"])
        o.edgvar3(s["dp3d"], s["tr3d"], s["dp_edg"], s["trc_edg"])
        o.cnuity(s["us3d"], s["vs3d"], s["u_edg"], s["v_edg"], s["dp_edg"], s["lp_edg"], s["dp3d"], s["pr3d"],
                 s["ex3d"], s["dp_tdcy"], s["dpl_tdcy"], s["massfx"], s["ws3d"])
        before = {n: s[n].copy() for n in NAMES}
        o.trcadv(s["trc_edg"], s["tr3d"], s["trdp"], s["trc_tdcy"], s["trl_tdcy"], s["massfx"], s["dp3d"])
    return grid, cfg, o, before, s


@pytest.mark.parametrize("precision,tol", [("f64", 1e-12), ("f32", 1e-5)])
@pytest.mark.parametrize("glvl,nvl,ntra,shift", [(1, 38, 5, 0), (2, 37, 4, 0), (3, 64, 6, 0), (3, 40, 5, 1), (3, 9, 5, 2)])
def test_trcadv_routes(glvl, nvl, ntra, shift, precision, tol):
    """shift: elements every array starts past a 256-byte boundary."""
    grid, cfg, o, before, after = _inputs(glvl, nvl, ntra)
    gcfg = F.FimConfig(**{k: getattr(cfg, k) for k in cfg.__dataclass_fields__})
    gcfg.precision = precision
    dyc = F.Dycore(grid, gcfg)
    dyc.set_ab(o.c.nf + 1, o.c.of + 1, o.c.vof + 1, o.c.ab1, o.c.ab2, o.c.ab3)
    st = dyc.state()
    st.set_tracers(0, 2)  # the routine transports every tracer it is given
    dt = torch.float64 if precision == "f64" else torch.float32

    def dev(a):
        b = torch.zeros(a.size + shift, dtype=dt, device="cuda")
        b[shift:] = torch.from_numpy(a).to(dt)
        return b[shift:]

    g = {n: dev(before[n]) for n in NAMES}
    dyc.trcadv(3, *[g[n] for n in NAMES])
    for n in ("tr3d", "trdp", "trc_tdcy", "trl_tdcy"):
        got = g[n].double().cpu().numpy()
        assert rel_l2(got, after[n]) <= tol, n
        if n == "tr3d":
            assert (got.reshape(ntra, -1)[2] == 0.0).all()
