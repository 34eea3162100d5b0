"""edgvar3's two-sided edge values on cell patches (FP32): column heights and
alignments of each level-vector width, small grids (pole patches, the general
staging loop), fields split over blocks or not; and the tracer transport with
edgvar1's edge values (hi_order_flux_comp = 0).  Against the CPU oracle."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import fimocn_subx_realtime_hera_apr2020_gb300 as F  # noqa: E402
from helpers import make_case, oracle_for, rel_l2  # noqa: E402

pytestmark = pytest.mark.gpu

EDG = ["us3d", "vs3d", "dp3d", "pr3d", "ex3d", "ph3d", "mp3d", "tr3d", "u_edg", "v_edg", "dp_edg", "lp_edg",
       "geop_edg", "mont_edg", "uvsq_edg", "trc_edg"]


def _case(glvl, nvl, ntra, **kw):
    if nvl != 38:
        th, dp = F.vertical_tables(64)
        kw.update(thetac=th[:nvl], dpsig=dp[:nvl])
    return make_case(glvl=glvl, nvl=nvl, ntra=ntra, dt=300.0, seed=91, **kw)


# 6 products and their sum in FP32, one rounding of inputs and coefficients:
# ~10 roundings of 6e-8 of the largest term
@pytest.mark.parametrize("glvl,nvl,ntra,shift", [(1, 38, 4, 0), (2, 37, 6, 0), (3, 64, 5, 0), (3, 40, 5, 1), (3, 40, 5, 2),
                                                 (5, 64, 4, 0)])
def test_edges_patch(glvl, nvl, ntra, shift):
    grid, cfg, fields = _case(glvl, nvl, ntra)
    o = oracle_for(grid, cfg)
    s = o.init_state(o.new_state(fields))
    rng = np.random.default_rng(92)
    s["tr3d"][grid.nip * nvl:] = rng.uniform(0.0, 1e-2, (ntra - 1) * grid.nip * nvl)
    gcfg = F.FimConfig(**{k: getattr(cfg, k) for k in cfg.__dataclass_fields__})
    gcfg.precision = "f32"
    dyc = F.Dycore(grid, gcfg)

    def dev(a):
        b = torch.zeros(a.size + shift, dtype=torch.float32, device="cuda")
        b[shift:] = torch.from_numpy(a).float()
        return b[shift:]

    g = {n: dev(s[n]) for n in EDG}
    o.edgvar1(*[s[n] for n in EDG])
    o.edgvar3(s["dp3d"], s["tr3d"], s["dp_edg"], s["trc_edg"])
    args = [g[n] for n in EDG]
    dyc.edgvar1(1, *args)
    dyc.edgvar3(1, *args)
    for n in ("u_edg", "v_edg", "lp_edg", "mont_edg", "uvsq_edg", "dp_edg", "trc_edg"):
        assert rel_l2(g[n].double().cpu().numpy(), s[n]) <= 1e-6, n
    five = np.asarray(grid.nprox) == 5
    te = g["trc_edg"].cpu().numpy().reshape(ntra, grid.nip, 6, nvl)
    assert not te[:, five, 5].any()
    # both cells of an edge hold the same average
    npx, prox, proxs = grid.zero_based()
    prox, proxs = prox.reshape(-1, 6), proxs.reshape(-1, 6)
    for e in range(5):
        assert np.array_equal(te[1:, :, e], te[1:, prox[:, e], proxs[:, e]])


@pytest.mark.parametrize("precision,tol", [("f64", 1e-12), ("f32", 1e-5)])
def test_step_without_high_order_fluxes(precision, tol):
    """hi_order_flux_comp = 0: edgvar1's dp and tracer edge values feed cnuity
    and the tracer kernels."""
    grid, cfg, fields = _case(3, 38, 5, precision=precision, hi_order_flux_comp=0)
    o = oracle_for(grid, cfg)
    s = o.init_state(o.new_state(fields))
    dyc = F.Dycore(grid, cfg)
    st = dyc.state()
    st.load(fields)
    st.init()
    for its in range(1, 4 if precision == "f64" else 2):
        o.step(s, its)
        st.step(its, use_graph=True)
        for n in ("us3d", "vs3d", "dp3d", "pr3d", "ex3d", "tr3d", "trdp"):
            assert rel_l2(st.download(n), s[n]) <= tol, (its, n)
