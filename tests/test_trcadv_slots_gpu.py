"""AB3 slots that are the same one (fim_set_ab takes any three of 1..3): the
tendency a call writes is then also one it reads, and the limiters of the cells
around see none of it.  Against the CPU oracle, twice alike."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import fimocn_subx_realtime_hera_apr2020_gb300 as F  # noqa: E402
from test_trcadv_routes_gpu import NAMES, _inputs  # noqa: E402
from helpers import rel_l2  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("f64", 1e-12), ("f32", 1e-5)])
@pytest.mark.parametrize("nf,of,vof", [(1, 1, 1), (2, 2, 3), (3, 1, 3), (1, 2, 2)])
@pytest.mark.parametrize("ab2,ab3", [(0.0, 0.0), (-0.25, 0.125)])
def test_equal_slots(nf, of, vof, ab2, ab3, precision, tol):
    grid, cfg, o, before, _ = _inputs(4, 38, 4)
    dt = 300.0
    o.c.nf, o.c.of, o.c.vof = nf - 1, of - 1, vof - 1
    o.c.ab1, o.c.ab2, o.c.ab3 = dt, ab2 * dt, ab3 * dt
    gcfg = F.FimConfig(**{k: getattr(cfg, k) for k in cfg.__dataclass_fields__})
    gcfg.precision = precision
    dyc = F.Dycore(grid, gcfg)
    dyc.set_ab(nf, of, vof, dt, ab2 * dt, ab3 * dt)
    # the mass fluxes of the new slot, whichever it is, are the case's
    mf = before["massfx"].reshape(3, -1)
    mf[:] = mf[np.abs(mf).sum(axis=1).argmax()]
    tdt = torch.float64 if precision == "f64" else torch.float32
    runs = []
    for _ in range(2):
        g = {n: torch.from_numpy(before[n]).to(device="cuda", dtype=tdt) for n in NAMES}
        dyc.trcadv(3, *[g[n] for n in NAMES])
        runs.append(g)
    s = {n: before[n].copy() for n in NAMES}
    o.trcadv(*[s[n] for n in NAMES])
    for n in ("tr3d", "trdp", "trc_tdcy", "trl_tdcy"):
        assert torch.equal(runs[0][n], runs[1][n]), n
        assert rel_l2(runs[0][n].double().cpu().numpy(), s[n]) <= tol, n
