"""Values that are not finite in the column kernels: a wind beside interfaces
that do not move, NaNs in theta, the Exner function, pressures and tracers.  The
comparisons keep or drop a NaN as they are written (a < b ? a : b)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import fimocn_subx_realtime_hera_apr2020_gb300 as F  # noqa: E402
from helpers import make_case, oracle_for  # noqa: E402

pytestmark = pytest.mark.gpu

HYB = ["us3d", "vs3d", "tr3d", "sdot", "ex3d", "dp3d", "pr3d"]
NAN, NEG_NAN = np.frombuffer(np.array([0x7ff8 << 48, 0xfff8 << 48], np.uint64).tobytes(), np.float64)


def _setup(precision, glvl=2, nvl=38, **kw):
    grid, cfg, fields = make_case(glvl=glvl, nvl=nvl, ntra=5, dt=200.0, seed=7, **kw)
    o = oracle_for(grid, cfg)
    s = o.new_state(fields)
    rng = np.random.default_rng(8)
    NL = grid.nip * nvl
    s["tr3d"][:NL] += rng.normal(0.0, 0.2, NL)
    gcfg = F.FimConfig(**{k: getattr(cfg, k) for k in cfg.__dataclass_fields__})
    gcfg.precision = precision
    if precision == "f32":
        for n in HYB:
            s[n][:] = s[n].astype(np.float32)
    return grid, o, s, F.Dycore(grid, gcfg)


def _dev(s, precision):
    dt = torch.float64 if precision == "f64" else torch.float32
    return {n: torch.from_numpy(s[n]).to(device="cuda", dtype=dt) for n in HYB}


def _cells(grid, g):
    """Columns without thin layers (whose fill couples layers by a factor 1e-22);
    FP32 takes two columns a warp, whose fills run together."""
    dp = g["dp3d"].double().cpu().numpy().reshape(grid.nip, 38)
    cells = set(np.nonzero(dp.min(axis=1) > 1.0)[0])
    cells = sorted(c for c in cells if c ^ 1 in cells)[:8]
    assert len(cells) == 8
    return cells


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("value", [np.inf, NAN])
def test_unmoved_interfaces(precision, value):
    """slak = 0 leaves every interface where it is: nothing passes through
    them, so a wind that is not finite stays in its layer."""
    grid, o, s, dyc = _setup(precision, slak=0.0)
    g = _dev(s, precision)
    dyc.hybgen(4, None, *[g[n] for n in HYB])  # pressures that belong to the Exner function
    cells = _cells(grid, g)
    before = {n: g[n].clone() for n in HYB}
    u = g["us3d"].view(grid.nip, 38)
    for j, c in enumerate(cells):
        u[c, 4 + 4 * j] = float(value)
    dyc.hybgen(4, None, *[g[n] for n in HYB])
    assert torch.equal(g["ex3d"], before["ex3d"])
    bad = ~torch.isfinite(g["us3d"].view(grid.nip, 38)).cpu().numpy()
    want = np.zeros_like(bad)
    for j, c in enumerate(cells):
        want[c, 4 + 4 * j] = True
    assert np.array_equal(bad, want), np.argwhere(bad != want)[:5]


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("value", [NAN, NEG_NAN])
def test_nan_layer(precision, value):
    """Of a NaN layer q's neighbours the one below takes a NaN slope and the one
    above none (f <= min(f-, f+) or f >= max(f-, f+), with a < b ? a : b): the
    flux through an interface that moved is a NaN if its donor is q or q - 1."""
    grid, o, s, dyc = _setup(precision)
    g = _dev(s, precision)
    dyc.hybgen(4, None, *[g[n] for n in HYB])
    cells = _cells(grid, g)
    old = g["pr3d"].clone().view(grid.nip, 39)
    u = g["us3d"].view(grid.nip, 38)
    for j, c in enumerate(cells):
        u[c, 4 + 4 * j] = float(value)
    dyc.hybgen(4, None, *[g[n] for n in HYB])
    move = (g["pr3d"].view(grid.nip, 39) - old).cpu().numpy()  # < 0: up, the layer above gives
    bad = torch.isnan(g["us3d"].view(grid.nip, 38)).cpu().numpy()
    want = np.zeros_like(bad)
    for j, c in enumerate(cells):
        q = 4 + 4 * j
        want[c, q] = True
        want[c, q - 1] = move[c, q] != 0
        want[c, q + 1] = move[c, q + 1] > 0
        if move[c, q - 1] < 0:
            want[c, q - 2:q] = True
    assert np.array_equal(bad, want), np.argwhere(bad != want)[:5]
