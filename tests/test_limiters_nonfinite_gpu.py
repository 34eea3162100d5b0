"""Values that are not finite in the flux-corrected transport: the limiters'
comparisons pass a NaN on (or drop it) as the routines are written, a = max(b,
c) being b > c ? b : c, so the same cell-levels come out finite as in the CPU
oracle, in both precisions and for NaNs of either sign."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import fimocn_subx_realtime_hera_apr2020_gb300 as F  # noqa: E402
from helpers import make_case, oracle_for  # noqa: E402

pytestmark = pytest.mark.gpu

EDG = ["us3d", "vs3d", "dp3d", "pr3d", "ex3d", "ph3d", "mp3d", "tr3d", "u_edg", "v_edg", "dp_edg", "lp_edg",
       "geop_edg", "mont_edg", "uvsq_edg", "trc_edg"]
CNU = ["us3d", "vs3d", "u_edg", "v_edg", "dp_edg", "lp_edg", "dp3d", "pr3d", "ex3d", "dp_tdcy", "dpl_tdcy",
       "massfx", "ws3d"]
TRC = ["trc_edg", "tr3d", "trdp", "trc_tdcy", "trl_tdcy", "massfx", "dp3d"]
NAN, NEG_NAN = np.frombuffer(np.array([0x7ff8 << 48, 0xfff8 << 48], np.uint64).tobytes(), np.float64)
NVL, NTRA = 38, 4


@pytest.fixture(scope="module")
def case():
    """The inputs of edgvar1, cnuity and trcadv in the third step."""
    grid, cfg, fields = make_case(glvl=3, nvl=NVL, ntra=NTRA, dt=400.0, seed=31)
    o = oracle_for(grid, cfg)
    s = o.init_state(o.new_state(fields))
    rng = np.random.default_rng(32)
    s["tr3d"][grid.nip * NVL:] = rng.uniform(1e-4, 1e-2, (NTRA - 1) * grid.nip * NVL)
    s["trdp"][:] = (s["tr3d"].reshape(NTRA, -1) * s["dp3d"].reshape(1, -1)).ravel()
    for its in (1, 2, 3):
        o.abstart(its)
        before_e = {n: s[n].copy() for n in EDG}
        o.edgvar1(*[s[n] for n in EDG])
        o.edgvar3(s["dp3d"], s["tr3d"], s["dp_edg"], s["trc_edg"])
        before = {n: s[n].copy() for n in CNU}
        o.cnuity(*[s[n] for n in CNU])
        before_t = {n: s[n].copy() for n in TRC}
        if its < 3:
            o.trcadv(*[s[n] for n in TRC])
    return grid, cfg, o, before_e, before, before_t


def _run(case, precision, routine, poison, before, names, outs, kinds=(np.isfinite,)):
    grid, cfg, o = case[:3]
    gcfg = F.FimConfig(**{k: getattr(cfg, k) for k in cfg.__dataclass_fields__})
    gcfg.precision = precision
    dyc = F.Dycore(grid, gcfg)
    dyc.set_ab(o.c.nf + 1, o.c.of + 1, o.c.vof + 1, o.c.ab1, o.c.ab2, o.c.ab3)
    dt = torch.float64 if precision == "f64" else torch.float32
    b = {n: before[n].copy() for n in names}
    if precision == "f32":  # both start from the rounded values
        for n in names:
            b[n] = b[n].astype(np.float32).astype(np.float64)
    poison(b)
    g = {n: torch.from_numpy(b[n]).to(device="cuda", dtype=dt) for n in names}
    getattr(o, routine)(*[b[n] for n in names])
    getattr(dyc, routine)(3, *[g[n] for n in names])
    for n in outs:
        got = g[n].cpu().numpy()
        assert not np.isfinite(b[n]).all() or n == "massfx", n
        for kind in kinds:
            assert np.array_equal(kind(b[n]), kind(got)), (n, int(kind(b[n]).sum()), int(kind(got).sum()))


# (FP32 takes the magnitude as x rsqrt(x), a NaN where x is infinite)
@pytest.mark.parametrize("name,value", [("us3d", np.inf), ("us3d", -np.inf), ("vs3d", NAN), ("vs3d", NEG_NAN)])
def test_edgvar1(case, name, value):
    """The edge winds' magnitude is floored only where it is a number below the floor."""
    N = case[0].nip

    def poison(b):
        for i in CELLS:
            for k in LEVELS:
                b[name].reshape(N, NVL)[i, k] = value

    _run(case, "f64", "edgvar1", poison, case[3], EDG, ["u_edg", "v_edg", "uvsq_edg"], (np.isnan, np.isinf))


CELLS = (3, 100, 317, 640)  # poles' neighbourhood, patch interiors and edges
LEVELS = (0, 13, 37)


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("name,value", [("tr3d", NAN), ("tr3d", NEG_NAN), ("tr3d", np.inf), ("massfx", NAN),
                                        ("massfx", NEG_NAN), ("massfx", -np.inf), ("trc_tdcy", NAN), ("trc_tdcy", NEG_NAN),
                                        ("trc_edg", NAN), ("trc_edg", NEG_NAN)])
def test_trcadv(case, precision, name, value):
    grid, _, o, _, _, before = case
    N = grid.nip

    def poison(b):
        for i in CELLS:
            for k in LEVELS:
                if name == "tr3d":
                    b[name].reshape(NTRA, N, NVL)[2, i, k] = value
                elif name == "massfx":
                    b[name].reshape(3, N, 6, NVL)[o.c.nf, i, 2, k] = value
                elif name == "trc_tdcy":
                    b[name].reshape(NTRA, 3, N, NVL)[2, o.c.of, i, k] = value
                else:
                    b[name].reshape(NTRA, N, 6, NVL)[2, i, 3, k] = value

    outs = ["tr3d", "trdp", "trc_tdcy"] + (["trl_tdcy"] if name in ("tr3d", "massfx") else [])
    _run(case, precision, "trcadv", poison, before, TRC, outs)


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("name,value", [("dp3d", NAN), ("dp3d", NEG_NAN), ("u_edg", NAN), ("u_edg", NEG_NAN),
                                        ("dp_tdcy", NAN), ("dp_tdcy", NEG_NAN)])
def test_cnuity(case, precision, name, value):
    grid, _, o, _, before, _ = case
    N = grid.nip

    def poison(b):
        for i in CELLS:
            for k in LEVELS[1:]:
                if name == "dp3d":
                    b[name].reshape(N, NVL)[i, k] = value
                elif name == "u_edg":
                    b[name].reshape(N, 6, NVL)[i, 2, k] = value
                else:
                    b[name].reshape(3, N, NVL)[o.c.of, i, k] = value

    _run(case, precision, "cnuity", poison, before, CNU, ["dp3d", "dp_tdcy", "massfx"])
