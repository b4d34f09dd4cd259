"""The layouts of a context.  Full: face geometry stored, LU-SGS rows with
all factors; compact: both formed where they are used (PHX_LAYOUT; by size
otherwise).  The same results.  The face fluxes, the SA face terms
and the staging buffer of state I/O live within one call each and lie in the
same memory: reading every array between the phases changes no bit of a step."""
import numpy as np
import pytest

from phenlei_b200 import cases
from phenlei_b200 import mesh as M
from phenlei_b200 import solver as S
from tests.conftest import rel_err

pytestmark = pytest.mark.gpu

COMMON = [S.PHX_Q, S.PHX_RES, S.PHX_DT, S.PHX_LIMIT, S.PHX_GRADX, S.PHX_GRADY, S.PHX_GRADZ, S.PHX_DQ, S.PHX_INVSPEC,
          S.PHX_VISSPEC]
SA = [S.PHX_Q_TURB, S.PHX_VISL, S.PHX_VIST, S.PHX_RES_TURB, S.PHX_GRAD_TURB]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("case", ["tets", "sa"])
def test_reads_between_phases_change_nothing(case, precision):
    # tetrahedra: the fewest faces a cell, so the least room beside the staging buffer
    m = M.tet_cube(6) if case == "tets" else M.channel_bump(24, 13, 7, thickness=0.08, prism_layers=5)
    params = dict(cases.LAMINAR, gradientName="lsq") if case == "tets" else cases.SA_BUMP
    wd = M.wall_distance(m) if case == "sa" else None
    q0 = cases.perturbed_state(m, params, seed=3)
    out = []
    for reads in (False, True):
        s = S.NSSolverUnstruct(m, precision=precision, wall_dist=wd, **params)
        s.set_q_cells(q0)
        phases = [s.Boundary, s.ComputeGradientAndLimiter, s.UpdateResiduals, s.LUSGSForward, s.LUSGSBackward,
                  s.UpdateFlowField]
        if case == "sa":
            phases += [s.TurbUpdateResiduals, s.TurbLUSGSForward, s.TurbLUSGSBackward, s.TurbUpdateFlowField]
        arrays = COMMON + (SA if case == "sa" else [])
        for step in range(1, 4):
            s.step = step
            for f in phases:
                f()
                if reads:
                    for a in arrays:
                        s.get(a)
        out.append([s.get(a) for a in arrays])
        s.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)


LAYOUTS = {
    "hex_vencat": (lambda: M.channel_bump(23, 11, 5), cases.EULER_BUMP),
    "hex_barth_rotate": (lambda: M.channel_bump(16, 8, 4),
                         dict(cases.EULER_BUMP, uns_limiter_name="barth", uns_scheme_name="vanleer_Rotate", flowInitStep=0)),
    "tets_lsq": (lambda: M.tet_cube(6), dict(cases.LAMINAR, gradientName="lsq", flowInitStep=1)),
    "hex_ggnode": (lambda: M.channel_bump(16, 9, 5), dict(cases.LAMINAR, gradientName="ggnode", flowInitStep=1)),
    "hex_clamped": (lambda: M.channel_bump(16, 9, 5), dict(cases.LAMINAR, ktmax=3.0, uns_scheme_name="ausmpw+", flowInitStep=0)),
    # cells of seven faces: more neighbours than lanes on one side
    "prism_sa": (lambda: M.channel_bump(24, 13, 7, thickness=0.08, prism_layers=5), dict(cases.SA_BUMP, flowInitStep=1)),
    "prism_sa_lsq": (lambda: M.channel_bump(24, 13, 7, thickness=0.08, prism_layers=5),
                     dict(cases.SA_BUMP, gradientName="lsq", flowInitStep=0)),
    "plate_sa": (lambda: M.flat_plate(20, 12, 6, first_spacing=1e-3), cases.SA_PLATE),
}
# geometry and sweep factors are formed by the same expressions where they are used or once before; a compiler may
# contract them otherwise, so a few roundings (2^-53, 2^-24) over three steps
TOL = {"fp64": 1e-13, "mixed": 2e-6}


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("name", sorted(LAYOUTS))
def test_every_layout_gives_the_same_results(monkeypatch, name, precision):
    make, params = LAYOUTS[name]
    m = make()
    sa = params["viscousType"] == 3
    wd = M.wall_distance(m) if sa else None
    q0 = cases.perturbed_state(m, params, seed=5)
    out, hist = [], []
    for layout, warps in (("full", None), ("compact", None), ("compact", "3")):
        monkeypatch.setenv("PHX_LAYOUT", layout)
        if warps:
            monkeypatch.setenv("PHX_LUSGS_MAX_BLOCKS", warps)
        s = S.NSSolverUnstruct(m, precision=precision, wall_dist=wd, **params)
        s.set_q_cells(q0)
        hist.append(s.Relaxation(3))
        out.append([s.get(a) for a in COMMON + (SA if sa else [])])
        s.close()
    for other in (1, 2):
        assert rel_err(hist[other], hist[0]) <= TOL[precision]
        for a, b in zip(out[0], out[other]):
            assert np.isfinite(a).all() and rel_err(b, a) <= TOL[precision]
    for a, b in zip(out[1], out[2]):   # few warps: the same sums in the same order
        assert np.array_equal(a, b)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("grad", ["ggcell", "lsq"])
def test_every_layout_across_zones(monkeypatch, grad, precision):
    """Interface faces: geometry behind them from the other zone, forward dq from the exchange."""
    from phenlei_b200.zones import ZoneSet

    m = M.channel_bump(24, 13, 7, thickness=0.08, prism_layers=5)
    params = dict(cases.SA_BUMP, gradientName=grad, flowInitStep=1)
    wd = M.wall_distance(m)
    q0 = cases.perturbed_state(m, params, seed=6)
    out = []
    for layout in ("full", "compact"):
        monkeypatch.setenv("PHX_LAYOUT", layout)
        z = ZoneSet(m, params, 3, wall_dist=wd, precision=precision)
        z.set_state(q0)
        out.append([z.iterate(3)] + [zz.get(a) for zz in z.zones for a in (S.PHX_Q, S.PHX_DQ, S.PHX_Q_TURB)])
    for a, b in zip(*out):
        assert np.isfinite(a).all() and rel_err(b, a) <= TOL[precision]
