"""The column kernels' routes by launch size: regrid's column arrays in shared
or local memory, the smoothing's wide or narrow blocks and the columns a warp
remaps follow the columns of a launch, so a member alone and the same member in
a large batch take different ones and have to come out alike, bit for bit.
Column heights that fill the remap's lanes (32, 64, 128 levels), with massless
layers, and heights whose shared memory needs the opt-in (FP64 cnuity5 and
hystat above 95 levels), against the CPU oracle."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import fimocn_subx_realtime_hera_apr2020_gb300 as F  # noqa: E402
from helpers import PROGNOSTIC, make_case, oracle_for, rel_l2  # noqa: E402

pytestmark = pytest.mark.gpu

HYB = ["us3d", "vs3d", "tr3d", "sdot", "ex3d", "dp3d", "pr3d"]
CNU = ["us3d", "vs3d", "u_edg", "v_edg", "dp_edg", "lp_edg", "dp3d", "pr3d", "ex3d", "dp_tdcy", "dpl_tdcy",
       "massfx", "ws3d"]


def _tables(nvl):
    if nvl == 38:
        return {}
    th, dp = F.vertical_tables(64)
    at = np.linspace(0.0, 63.0, nvl)
    return dict(thetac=np.interp(at, np.arange(64.0), th), dpsig=np.interp(at, np.arange(64.0), dp) * 64.0 / nvl)


# 81 blocks of 32 columns a member at glvl 4.  152 SMs of 227 KB hold 1064 (FP32)
# or 456 (FP64) one-warp regrid blocks at nvl 64, and blocks turn narrow above 608
@pytest.mark.parametrize("precision,nvl,members", [("f32", 64, 16), ("f64", 64, 8), ("f64", 38, 12)])
def test_member_alone_and_in_a_batch(precision, nvl, members):
    grid, cfg, fields = make_case(glvl=4, nvl=nvl, ntra=5, dt=300.0, seed=41, precision=precision)
    runs = []
    for m in (1, members):
        c = F.FimConfig(**{k: getattr(cfg, k) for k in cfg.__dataclass_fields__})
        c.members = m
        st = F.Dycore(grid, c).state()
        for q in range(m):
            st.load(fields, member=q)
        st.init()
        for its in (1, 2, 3):
            st.step(its)
        runs.append(st)
    for n in PROGNOSTIC + ["sdot", "ws3d"]:
        want = runs[0].download(n)
        for q in (0, members - 1):
            assert np.array_equal(runs[1].download(n, member=q), want), (n, q)


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("nvl", [32, 38, 64, 128])
@pytest.mark.parametrize("thktop", [30.0, 0.0])
def test_massless_layers(nvl, precision, thktop):
    grid, cfg, fields = make_case(glvl=2, nvl=nvl, ntra=5, dt=200.0, seed=9, thktop=thktop, **_tables(nvl))
    o = oracle_for(grid, cfg)
    s = o.new_state(fields)
    N = grid.nip
    ex, pr = s["ex3d"].reshape(N, nvl + 1), s["pr3d"].reshape(N, nvl + 1)
    for i in range(0, N, 3):  # two collapsed layers and one of 1e-5 Pa
        for k, thin in ((3 + i % 5, 0.0), (nvl // 2, 0.0), (nvl - 6, 1e-5)):
            pr[i, k + 1] = pr[i, k] - thin
            ex[i, k + 1] = 1004.6855 * (pr[i, k + 1] / 1e5) ** (287.0586 / 1004.6855)
    s["dp3d"][:] = (pr[:, :-1] - pr[:, 1:]).ravel()
    gcfg = F.FimConfig(**{k: getattr(cfg, k) for k in cfg.__dataclass_fields__})
    gcfg.precision = precision
    dt = torch.float64 if precision == "f64" else torch.float32
    if precision == "f32":
        for n in HYB:
            s[n][:] = s[n].astype(np.float32)
    dyc = F.Dycore(grid, gcfg)
    g = {n: torch.from_numpy(s[n]).to(device="cuda", dtype=dt) for n in HYB}
    # FP32 pressures are up to 2^-7 Pa apart: an interface is off by that at
    # each of its three steps (old, smoothed, new), which moves the same share
    # of a layer's value into the next one
    tol = 1e-12 if precision == "f64" else 3 * 2.0 ** -7 / s["dp3d"][s["dp3d"] > 1.0].min()
    o.hybgen(4, *[s[n] for n in HYB])
    dyc.hybgen(4, None, *[g[n] for n in HYB])
    # a layer's value weighs by its thickness: a massless layer's is arbitrary
    w = s["dp3d"]
    for n in ("us3d", "vs3d", "tr3d"):
        x = np.tile(w, s[n].size // w.size)
        assert rel_l2(g[n].double().cpu().numpy() * x, s[n] * x) <= tol, n
    for n in ("ex3d", "pr3d"):
        assert rel_l2(g[n].double().cpu().numpy(), s[n]) <= tol, n


@pytest.mark.parametrize("nvl", [96, 128])
def test_tall_columns(nvl):
    grid, cfg, fields = make_case(glvl=2, nvl=nvl, ntra=5, dt=200.0, seed=10, **_tables(nvl))
    o = oracle_for(grid, cfg)
    s = o.init_state(o.new_state(fields))
    o.abstart(1)
    dyc = F.Dycore(grid, cfg)
    dyc.set_ab(o.c.nf + 1, o.c.of + 1, o.c.vof + 1, o.c.ab1, o.c.ab2, o.c.ab3)
    o.edgvar1(*[s[n] for n in ["us3d", "vs3d", "dp3d", "pr3d", "ex3d", "ph3d", "mp3d", "tr3d", "u_edg", "v_edg",
                               "dp_edg", "lp_edg", "geop_edg", "mont_edg", "uvsq_edg", "trc_edg"]])
    o.edgvar3(s["dp3d"], s["tr3d"], s["dp_edg"], s["trc_edg"])
    g = {n: torch.from_numpy(s[n].copy()).cuda() for n in CNU}
    o.cnuity(*[s[n] for n in CNU])
    dyc.cnuity(1, *[g[n] for n in CNU])
    for n in ("dp3d", "pr3d", "ex3d", "ws3d"):
        assert rel_l2(g[n].cpu().numpy(), s[n]) <= 1e-12, n
    names = ["ph3d", "ex3d", "mp3d", "dp3d", "tr3d", "trdp", "psrf", "ptdcy"]
    g = {n: torch.from_numpy(s[n].copy()).cuda() for n in names}
    o.hystat(1, *[s[n] for n in names])
    dyc.hystat(1, *[g[n] for n in names])
    for n in ("ph3d", "mp3d", "trdp", "psrf"):
        assert rel_l2(g[n].cpu().numpy(), s[n]) <= 1e-12, n
    # the tendency is the difference of two column sums of ~1e5 Pa
    assert np.abs(g["ptdcy"].cpu().numpy() - s["ptdcy"]).max() <= 2 * nvl * 2.0 ** -53 * 1.1e5
