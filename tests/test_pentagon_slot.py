"""A pentagon's sixth prox entry may be any cell (the routines' one-ring bounds
read it, no edge uses it).  Without high-order edge fluxes a context takes such
a grid; the patches' frames then hold that cell too."""
import numpy as np
import pytest

import fimocn_subx_realtime_hera_apr2020_gb300 as F
from fimocn_subx_realtime_hera_apr2020_gb300 import _lib as L
from helpers import PROGNOSTIC, oracle_for, rel_l2


def far_sixth(glvl):
    """A grid whose pentagons' sixth entries name cells far away."""
    g = F.Grid(glvl)
    prox = g.prox.reshape(-1, 6)
    for j, i in enumerate(np.nonzero(np.asarray(g.nprox) == 5)[0]):
        prox[i, 5] = 1 + (int(i) + g.nip // 2 + 3 * j) % g.nip
    return g


@pytest.mark.gpu
@pytest.mark.parametrize("precision,tol", [("f64", 1e-12), ("f32", 1e-5)])
def test_step_without_high_order_fluxes(precision, tol):
    pytest.importorskip("torch")
    grid = far_sixth(4)
    cfg = F.FimConfig(nvl=38, ntra=5, dt=300.0, precision=precision, hi_order_flux_comp=0)
    fields = F.synthetic_state(grid, cfg, seed=5, sigma_ps=200.0, noise=1.0)
    o = oracle_for(grid, cfg)
    s = o.init_state(o.new_state(fields))
    st = F.Dycore(grid, cfg).state()
    st.load(fields)
    st.init()
    for its in range(1, 4 if precision == "f64" else 2):
        o.step(s, its)
        st.step(its)
        for n in PROGNOSTIC:
            assert rel_l2(st.download(n), s[n]) <= tol, (its, n)


@pytest.mark.gpu
def test_high_order_context_refuses():
    pytest.importorskip("torch")
    with pytest.raises(RuntimeError):
        F.Dycore(far_sixth(4), F.FimConfig(nvl=38, ntra=5, dt=300.0))


@pytest.mark.gpu
def test_no_coefficients_where_none_are_read():
    """An FP64 context without high-order fluxes holds no copy of the
    least-squares coefficients (36 a cell and the ring edges')."""
    pytest.importorskip("torch")
    grid = F.Grid.cached(4)
    size = [F.Dycore(grid, F.FimConfig(nvl=38, ntra=5, dt=300.0, hi_order_flux_comp=h)) for h in (0, 1)]
    size = [d.lib.fim_ctx_device_bytes(d.ctx) for d in size]
    assert size[1] - size[0] >= 8 * 36 * grid.nip
