"""Memory that the phases of a step share.  The face fluxes, the SA face terms
and the staging buffer of state I/O live within one call each and lie in the
same memory: reading every array between the phases changes no bit of a step."""
import numpy as np
import pytest

from phenlei_b200 import cases
from phenlei_b200 import mesh as M
from phenlei_b200 import solver as S

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
