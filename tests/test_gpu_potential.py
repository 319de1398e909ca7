"""The couple in potential form (lcs_potential.cuh) against the oracle's
element-wise sweeps.

Both visit the same cells in the same order with the same divergence up to
rounding.  FP64: a sweep rounds Phi and the sums of its div by a few ulp, and
red-black relaxation does not amplify them, so after up to 61 sweeps U, V, W
and P agree to 61 x 10 ulp = 1.4e-13; the bound is 1e-12.  FP32: U, V, W to
1e-5 and P to 1e-3 of FP64, the bounds of the element-wise FP32 sweeps.
Sweep counts are equal; the residual, while it is far above rounding, agrees to
1e-9 (differences of U, each 1e-16 of values about 1e4 times the residual).
"""

import numpy as np
import pytest

import serve_cases
from helpers import make_config, rel_l2
from lcs_b200 import Engine, _abi
from oracle_engine import OracleEngine

F = _abi
pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def potential(monkeypatch):
    monkeypatch.setenv("LCS_B200_FUSED_SWEEP", "potential")


def couple(cls, dims, ov, itrmin, itrmax, epsp, precision=F.PRECISION_FP64, stage=2):
    cfg = make_config(dims=dims, mode=F.MODE_FLOW, time_blocking=True, overlap=ov, itrmin=itrmin, itrmax=itrmax,
                      epsp=epsp, Re=50.0, precision=precision)
    e = cls(cfg)
    rng = np.random.default_rng(sum(dims))
    fields = (0, 1, 2, 6) if stage == 2 else (3, 4, 5, 6)
    for f in fields:
        e.field_set(f, rng.standard_normal(e.interior_shape) * (0.1 if f == 6 else 0.5))
    lg = e.couple(stage, 0.004)
    out = [e.field_get(f) for f in fields]
    e.close()
    return lg, out


# the tiles give 52 x 20 columns and the slab tiles 26 x 26: one column or row
# less, equal and more; few planes; the smallest grid; several tiles and chunks
DIMS = [(8, 8, 8), (24, 26, 30), (50, 18, 40), (52, 20, 32), (54, 22, 20), (106, 42, 16), (72, 64, 130), (96, 96, 96)]


@pytest.mark.parametrize("ov", [True, False])
@pytest.mark.parametrize("dims", DIMS)
def test_fp64_equals_the_element_wise_order(dims, ov):
    lg, g = couple(Engine, dims, ov, 6, 61, 1e-12)
    lo, o = couple(OracleEngine, dims, ov, 6, 61, 1e-12)
    assert lg["itr"] == lo["itr"] and lg["sweeps"] == lo["sweeps"]
    if min(dims) >= 32:  # smaller boxes relax to a residual of rounding alone
        assert abs(lg["div"] - lo["div"]) <= 1e-9 * lo["div"]
    for a, b in zip(g, o):
        assert rel_l2(a, b) <= 1e-12


@pytest.mark.parametrize("tile", ["0", "1", "2"])
@pytest.mark.parametrize("dims", [(24, 26, 30), (54, 38, 66), (106, 74, 16)])
def test_sweep_tiles(dims, tile, monkeypatch):
    """The three tile heights (FP64: two) on the same grids."""
    monkeypatch.setenv("LCS_B200_POT_TILE", tile)
    _, g = couple(Engine, dims, True, 6, 12, 1e-12)
    _, o = couple(OracleEngine, dims, True, 6, 12, 1e-12)
    for a, b in zip(g, o):
        assert rel_l2(a, b) <= 1e-12
    _, f = couple(Engine, dims, True, 6, 12, 1e-12, F.PRECISION_FP32_MIXED)
    errs = [rel_l2(a, b) for a, b in zip(f, o)]
    assert max(errs[:3]) <= 1e-5 and errs[3] <= 1e-3, errs


@pytest.mark.parametrize("itrmin", [6, 7, 8])
@pytest.mark.parametrize("itrmax", [9, 60])
@pytest.mark.parametrize("ov", [True, False])
def test_exit_inside_a_group(itrmin, itrmax, ov):
    """An exit after the first, second and third sweep of a group: the group
    runs again up to that sweep (also when it is the loop's last)."""
    lg, g = couple(Engine, (40, 24, 32), ov, itrmin, itrmax, 1e3, stage=1)
    lo, o = couple(OracleEngine, (40, 24, 32), ov, itrmin, itrmax, 1e3, stage=1)
    assert lg["itr"] == lo["itr"] == itrmin and lg["sweeps"] == lo["sweeps"]
    for a, b in zip(g, o):
        assert rel_l2(a, b) <= 1e-12


@pytest.mark.parametrize("dims", [(24, 26, 30), (54, 38, 20), (272, 250, 252)])
def test_fp32_close_to_fp64(dims):
    l32, a = couple(Engine, dims, True, 6, 12, 1e-12, F.PRECISION_FP32_MIXED)
    l64, b = couple(Engine, dims, True, 6, 12, 1e-12)
    assert l32["sweeps"] == l64["sweeps"]
    errs = [rel_l2(x, y) for x, y in zip(a, b)]
    assert max(errs[:3]) <= 1e-5 and errs[3] <= 1e-3, errs


@pytest.mark.parametrize("epsp", [1e-12, 2e-3])
def test_step_graph_equals_direct_calls(epsp):
    """The device-side loop (with and without an early exit) takes the same
    groups as the host's."""
    out = []
    for graphs in (0, 1):
        cfg = make_config(40, mode=F.MODE_FLOW, Re=50.0, itrmin=6, itrmax=40, epsp=epsp, graphs=graphs)
        e = Engine(cfg)
        rng = np.random.default_rng(3)
        e.upload_flow(*[rng.standard_normal(e.interior_shape) * 0.3 for _ in range(4)])
        logs = e.step(3)
        out.append((logs, e.download_flow()))
        e.close()
    (la, fa), (lb, fb) = out
    for x, y in zip(la, lb):
        assert x["couple1"] == y["couple1"] and x["couple2"] == y["couple2"]
    for a, b in zip(fa, fb):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("precision", [F.PRECISION_FP64, F.PRECISION_FP32_MIXED])
def test_group_equals_members_alone(precision):
    from lcs_b200 import _abi as abi

    serve_cases.check_group_equals_members_alone(Engine, abi.load_library(), precision, count=5, nsteps=2, n=28)
