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
import test_gpu_parity as parity
from helpers import make_config, rel_l2
from lcs_b200 import Engine, LCSError, _abi
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


# the sweep's tiles give 52 x 20 columns, of n + 1 (dims are even): just below,
# and above one and two of them; few planes; the smallest grid; several tiles and
# chunks.  A slab tile gives 22 x 22 of n + 5 or n - 1: 22 | 24 and 44 | 46 (n - 1),
# 38 | 40 (n + 5) lie on either side, along each axis.
DIMS = [(8, 8, 8), (24, 26, 30), (50, 18, 40), (52, 20, 32), (54, 22, 20), (106, 42, 16), (72, 64, 130), (96, 96, 96),
        (22, 38, 44), (24, 40, 46), (44, 22, 38), (46, 24, 40), (38, 44, 22), (40, 46, 24)]


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


@pytest.mark.parametrize("n", [8, 32, 54])
def test_fp32_uniform_flow_leaves_at_itrmin(n):
    """A uniform flow is free of divergence in FP32 too: residual 0, the exit
    and the counts of the oracle."""
    out = []
    for cls in (Engine, OracleEngine):
        e = cls(make_config(n, mode=F.MODE_FLOW, itrmin=7, itrmax=60, epsp=1e-8 * 2 * np.pi / n,
                            precision=F.PRECISION_FP32_MIXED))
        for f, v in ((0, 1.0), (1, -0.3), (2, 0.1), (6, 0.0)):
            e.field_set(f, np.full(e.interior_shape, v))
        out.append(e.couple(2, 0.004))
        e.close()
    assert out[0] == out[1] and out[0]["itr"] == 7 and out[0]["div"] == 0.0


def smooth(shape, rng, share=1e-3):
    """U, V, W of 24 Fourier modes each (|k| <= 3 an axis, rms about 0.5) without
    divergence, and `share` of it with: a thousandth is what a time step hands to
    a couple."""
    nz, ny, nx = shape
    pts = np.meshgrid(*(np.arange(m) * (2 * np.pi / m) for m in (nz, ny, nx)), indexing="ij")[::-1]
    out = []
    for a in range(3):
        f = np.zeros(shape)
        for _ in range(24):
            k = rng.integers(-3, 4, 3)
            whole = rng.random() < 0.5
            amp = 0.15 if whole else 0.15 * share
            if whole:
                k[a] = 0
            f += amp * np.sin(sum(k[b] * pts[b] for b in range(3)) + rng.random() * 6.3)
        out.append(f)
    return out


@pytest.mark.parametrize("ov", [True, False])
@pytest.mark.parametrize("n", [24, 32, 48])
def test_fp32_residual_is_the_stored_velocitys(n, ov):
    """Long FP32 couples.  Rounding the stored faces (about 0.5, 1.2e-8 rms)
    leaves a divergence of sqrt(6) 1.2e-8 / dx = 1.1e-7 to 2.2e-7; the sweeps
    relax Phi (5e-4) until its own rounding stops them, below 1e-8.  So with an
    exit at 4e-8 the couple must not leave, although the potential alone would,
    and the logged residual is the stored velocity's divergence up to twice
    1e-8, 15 % of the former."""
    e = Engine(make_config(n, mode=F.MODE_FLOW, overlap=ov, itrmin=6, itrmax=900, epsp=4e-8 * 2 * np.pi / n,
                           precision=F.PRECISION_FP32_MIXED))
    for f, a in enumerate(smooth(e.interior_shape, np.random.default_rng(n))):
        e.field_set(f, a)
    lg = e.couple(2, 0.004)
    rms, _ = e.flow_divergence()
    e.close()
    assert lg["itr"] == lg["sweeps"] == 900
    assert abs(lg["div"] - rms) <= 0.15 * rms, (lg, rms)


@pytest.mark.parametrize("itrmin", [6, 7, 8])
@pytest.mark.parametrize("epsp", [1e3, 3e-3])
@pytest.mark.parametrize("ov", [True, False])
def test_fp32_exit_equals_the_oracles(itrmin, epsp, ov):
    """Exits after each sweep of a group, and on the residual far above the
    rounding: the oracle's counts (a residual falls by 1 % or more a sweep, FP32
    changes it by 1e-6)."""
    dims = (40, 24, 32)
    lg, g = couple(Engine, dims, ov, itrmin, 200, epsp, F.PRECISION_FP32_MIXED)
    lo, o = couple(OracleEngine, dims, ov, itrmin, 200, epsp)
    assert lg["itr"] == lo["itr"] < 200 and lg["sweeps"] == lo["sweeps"]
    for a, b in zip(g[:3], o[:3]):
        assert rel_l2(a, b) <= 1e-5


@pytest.mark.parametrize("rms,itrmax", [(3e-8, 420), (1e-4, 420)])
def test_fp32_step_graph_equals_direct_calls(rms, itrmax):
    """The device-side loop in FP32: with the rounding measured and above the
    exit (3e-8), and with an exit (1e-4)."""
    out = []
    for graphs in (0, 1):
        e = Engine(make_config(32, mode=F.MODE_FLOW, Re=50.0, itrmin=6, itrmax=itrmax, epsp=rms * 2 * np.pi / 32,
                               graphs=graphs, precision=F.PRECISION_FP32_MIXED))
        e.upload_flow(*smooth(e.interior_shape, np.random.default_rng(4)), np.zeros(e.interior_shape))
        logs = e.step(2)
        out.append((logs, e.download_flow()))
        e.close()
    (la, fa), (lb, fb) = out
    for x, y in zip(la, lb):
        assert x["couple1"] == y["couple1"] and x["couple2"] == y["couple2"]
        assert (x["couple2"]["itr"] == itrmax) == (rms < 1e-7)
    for a, b in zip(fa, fb):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("n", [32, 64, 128])
def test_fp64_error_of_long_couples(n):
    """No bias of the operator: a relative error b of one coefficient changes the
    longest waves of P by b 6 n^2 / 4 pi^2 (b = 1.1e-16 at 64^3: 7e-14 of their
    share).  Element by element the roundings of 300 sweeps leave 1e-15 in P,
    the potential less; bound 4e-15."""
    out = []
    for cls in (Engine, OracleEngine):
        e = cls(make_config(n, mode=F.MODE_FLOW, overlap=False, itrmin=300, itrmax=300, epsp=1e-30))
        for f, a in enumerate(smooth(e.interior_shape, np.random.default_rng(1), share=1.0)):
            e.field_set(f, a)
        e.field_set(6, np.zeros(e.interior_shape))
        e.couple(2, 0.004)
        out.append([e.field_get(f) for f in (0, 1, 2, 6)])
        e.close()
    errs = [rel_l2(a, b) for a, b in zip(*out)]
    assert max(errs) <= 4e-15, errs


@pytest.mark.parametrize("precision", [F.PRECISION_FP64, F.PRECISION_FP32_MIXED])
@pytest.mark.parametrize("dims,h,ov", [((24, 26, 30), 3, True), ((8, 8, 8), 3, True), ((10, 32, 8), 5, False)])
def test_halos_after_a_couple(dims, h, ov, precision):
    """The halos of U, V, W and P are the images of the interior, whatever they
    held: exactly."""
    e = Engine(make_config(dims=dims, h=h, mode=F.MODE_FLOW, overlap=ov, itrmin=6, itrmax=9, epsp=1e-12,
                           precision=precision))
    rng = np.random.default_rng(2)
    for f in (0, 1, 2, 6):
        e.field_set(f, rng.standard_normal(e.haloed_shape), haloed=True)
    e.couple(2, 0.004)
    for f in (0, 1, 2, 6):
        a = e.field_get(f, haloed=True)
        assert np.array_equal(a, np.pad(a[h:-h, h:-h, h:-h], h, mode="wrap")), f
    e.close()


@pytest.mark.parametrize("precision", [F.PRECISION_FP64, F.PRECISION_FP32_MIXED])
def test_group_members_leave_at_different_sweeps(precision, monkeypatch):
    """The ensemble's loop (four groups a body from itrmax 24): members whose
    couples end in different groups and bodies, after the first, second or third
    sweep, each as alone, bit for bit."""
    from lcs_b200 import _abi as abi

    def configs(prec, n, count):
        cfgs = plain(prec, n=n, count=count)
        for c in cfgs:
            c.itrmax, c.epsp = 70, 1e-3
        return cfgs

    def scaled(cfg, seed):
        flow, parts = inputs(cfg, seed)
        return [f * 0.25 * 3.0 ** (seed % 5) for f in flow], parts

    plain, inputs = serve_cases.group_configs, serve_cases.inputs
    monkeypatch.setattr(serve_cases, "group_configs", configs)
    monkeypatch.setattr(serve_cases, "inputs", scaled)
    sweeps = []
    for i, c in enumerate(configs(precision, 28, 5)):
        c.use_graphs = 1
        logs = serve_cases.run_alone(Engine, c, 200 + i, 4)[2]
        sweeps += [lg[k]["sweeps"] for lg in logs for k in ("couple1", "couple2")]
    assert {s % 3 for s in sweeps} == {0, 1, 2} and max(sweeps) - min(sweeps) > 12 and min(sweeps) < 70, sweeps
    serve_cases.check_group_equals_members_alone(Engine, abi.load_library(), precision, count=5, nsteps=2, n=28)


@pytest.mark.parametrize("tile", ["0", "2"])
@pytest.mark.parametrize("ov", [True, False])
def test_fp64_planes_without_masks(ov, tile, monkeypatch):
    """Interior tiles of one long z chunk: most planes run the form without
    masks (three tile columns, so that the middle one lies off both faces)."""
    monkeypatch.setenv("LCS_B200_POT_TILE", tile)
    monkeypatch.setenv("LCS_B200_ZCHUNK", "60")
    dims = (160, 64, 48)
    lg, g = couple(Engine, dims, ov, 6, 13, 1e-12)
    lo, o = couple(OracleEngine, dims, ov, 6, 13, 1e-12)
    assert lg["sweeps"] == lo["sweeps"] and abs(lg["div"] - lo["div"]) <= 1e-9 * lo["div"]
    for a, b in zip(g, o):
        assert rel_l2(a, b) <= 1e-12


@pytest.mark.parametrize("graphs", [0, 1])
def test_ten_steps_noncubic(graphs):
    """Whole steps (forcing, particles) of FP64 boxes that run element by element
    unless asked: the bounds of the element-wise form, 1e-10 after ten steps."""
    parity.test_ten_steps_noncubic_rel_l2(graphs)


@pytest.mark.parametrize("forcing", [F.FORCING_LINEAR_POWER, F.FORCING_RC_ENERGY, F.FORCING_NO])
@pytest.mark.parametrize("ov", [True, False])
def test_ten_steps(forcing, ov):
    cfg = make_config(32, forcing=forcing, power=0.5, energy=0.649, kmin=1, kmax=2, coarse=8, Re=100.0, overlap=ov,
                      itrmin=6, itrmax=40, epsp=1e-8 * 2 * np.pi / 32, graphs=1,
                      species=[{"n": 2000, "density_ratio": 843.0}, {"n": 1000, "density_ratio": 843.0}])
    (g, o), (lg, lo) = parity.evolve_pair(cfg, 10, nparts=(2000, 1000), graphs=True)
    assert g.couple_form() == "potential"
    for a, b in zip(lg, lo):
        assert [a[c]["itr"] for c in ("couple1", "couple2")] == [b[c]["itr"] for c in ("couple1", "couple2")]
        assert abs(a["dt"] - b["dt"]) <= 1e-13 * b["dt"]
    for a, b in zip(g.download_flow(), o.download_flow()):
        assert rel_l2(a, b) <= 1e-10
    for q in (0, 1):
        a, b = g.download_particles(q), o.download_particles(q)
        assert all(rel_l2(a[k], b[k]) <= 1e-10 for k in ("x", "y", "z", "u", "v", "w"))


@pytest.mark.parametrize("graphs", [0, 1])
@pytest.mark.parametrize("precision", [F.PRECISION_FP64, F.PRECISION_FP32_MIXED])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_nonfinite_residual_is_reported(bad, precision, graphs):
    """A non-finite P leaves the time step finite and reaches the couple through
    the rhs: the loop ends and the call reports it."""
    e = Engine(make_config(24, mode=F.MODE_FLOW, Re=50.0, itrmin=6, itrmax=60, graphs=graphs, precision=precision))
    rng = np.random.default_rng(1)
    flow = [rng.standard_normal(e.interior_shape) * 0.3 for _ in range(4)]
    flow[3][5, 6, 7] = bad
    e.upload_flow(*flow)
    with pytest.raises(LCSError) as ei:
        e.step(1)
    assert ei.value.code == F.ENONFINITE
    e.close()
