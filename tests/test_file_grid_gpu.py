"""Grid tables that are not exact rotations: a grid read from glvl.dat holds
real*4 cosines and sines, whose cs^2 + sn^2 is off by up to 6e-8.  The edge
winds' magnitudes are those of the rotated components, so the FP64 build keeps
its bound against the CPU oracle on such tables too."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import fimocn_subx_realtime_hera_apr2020_gb300 as F  # noqa: E402
from fimocn_subx_realtime_hera_apr2020_gb300.grid_io import read_glvl_dat, write_glvl_dat  # noqa: E402
from helpers import PROGNOSTIC, oracle_for, rel_l2  # noqa: E402

pytestmark = pytest.mark.gpu

EDG = ["us3d", "vs3d", "dp3d", "pr3d", "ex3d", "ph3d", "mp3d", "tr3d", "u_edg", "v_edg", "dp_edg", "lp_edg",
       "geop_edg", "mont_edg", "uvsq_edg", "trc_edg"]


def _case(glvl, tmp_path, precision="f64"):
    grid = F.Grid(glvl)
    write_glvl_dat(grid, tmp_path / "glvl.dat")
    tables = read_glvl_dat(tmp_path / "glvl.dat", glvl=glvl)
    for n in grid.NAMES_I + grid.NAMES_D:
        getattr(grid, n)[:] = getattr(tables, n)
    cfg = F.FimConfig(nvl=38, ntra=5, dt=300.0, precision=precision)
    return grid, cfg, F.synthetic_state(grid, cfg, seed=17, sigma_ps=300.0, noise=1.0)


@pytest.mark.parametrize("glvl", [2, 4])
def test_edgvar1(glvl, tmp_path):
    grid, cfg, fields = _case(glvl, tmp_path)
    o = oracle_for(grid, cfg)
    s = o.init_state(o.new_state(fields))
    s["us3d"][7::11] = 0.0  # still air: the magnitude's floor
    s["vs3d"][7::11] = 0.0
    dyc = F.Dycore(grid, cfg)
    g = {n: torch.from_numpy(s[n].copy()).cuda() for n in EDG}
    o.edgvar1(*[s[n] for n in EDG])
    dyc.edgvar1(1, *[g[n] for n in EDG])
    for n in ("u_edg", "v_edg", "uvsq_edg"):
        assert rel_l2(g[n].cpu().numpy(), s[n]) <= 1e-12, n


@pytest.mark.parametrize("precision,tol", [("f64", 1e-12), ("f32", 1e-5)])
def test_step(precision, tol, tmp_path):
    grid, cfg, fields = _case(3, tmp_path, precision)
    o = oracle_for(grid, cfg)
    s = o.init_state(o.new_state(fields))
    st = F.Dycore(grid, cfg).state()
    st.load(fields)
    st.init()
    o.step(s, 1)
    st.step(1)
    for n in PROGNOSTIC:
        assert rel_l2(st.download(n), s[n]) <= tol, n
