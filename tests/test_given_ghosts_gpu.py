"""The residual of a state whose ghosts the caller gave (PHX_Q sets cells and
ghosts; phx_ns_boundary is not run after it): a wall's face velocity in the
viscous flux is zero all the same (GetVisFaceValue,
CFD/NSSolver/src/NSSolverUnstruct.cpp:7126-7375), and the other faces take the
mean of both sides.  Against the oracle's routines on the same arrays; 1e-12 is
the FP64 bound of the other laminar tests, and single precision carries its
own rounding, 1e-5 of the largest value."""
import ctypes as C

import numpy as np
import pytest

from phenlei_b200 import cases
from phenlei_b200 import mesh as M
from phenlei_b200 import solver as S
from tests.conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grad", ["ggcell", "lsq"])
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 1e-5)])
def test_residual_with_moving_wall_ghosts(precision, tol, grad):
    from oracle.oracle import Oracle, _p, lib

    m = M.channel_bump(24, 12, 3)
    params = dict(cases.LAMINAR, gradientName=grad, flowInitStep=0, refReNumber=50.0)
    nc, nt = m.n_cell, m.n_cell + m.n_bface
    q0 = cases.perturbed_state(m, params, seed=12)
    s = S.NSSolverUnstruct(m, precision=precision, **params)
    s.set_q_cells(q0)
    s.step = 1
    s.Boundary()
    s.ComputeGradientAndLimiter()
    q = s.get(S.PHX_Q)
    walls = np.isin(m.solver_regions()[1], np.flatnonzero(np.asarray(m.solver_regions()[0]) == M.BC_SOLID_SURFACE))
    ghosts = nc + np.flatnonzero(walls)
    assert len(ghosts)
    q[1:4, ghosts] += 0.2 * np.random.default_rng(1).standard_normal((3, len(ghosts)))
    s.set(S.PHX_Q, q)
    s.UpdateResiduals()

    o = Oracle(m, params)
    o.set_state(q0)
    L, w = lib(), o.work
    g, mm, p = C.byref(o.g), C.byref(o.m), C.byref(o.p)

    def gas():
        L.ox_gamma_temperature(g, p, _p(o.q), _p(w("gama")), _p(w("t")))

    gas()
    L.ox_ns_boundary(g, mm, p, _p(o.q), _p(w("gama")))
    gas()
    for k in range(5):
        L.ox_gradient(g, mm, p, _p(o.q[k]), _p(w("dqdx")[k]), _p(w("dqdy")[k]), _p(w("dqdz")[k]))
    L.ox_gradient(g, mm, p, _p(w("t")), _p(w("dtdx")), _p(w("dtdy")), _p(w("dtdz")))
    grads = [_p(w(a)) for a in ("dqdx", "dqdy", "dqdz")]
    L.ox_limiter(g, mm, p, _p(o.q), *grads, _p(w("limit")))
    o.q[:, nc:] = q[:, nc:]
    gas()
    L.ox_viscosity(g, p, _p(w("t")), _p(w("visl")), _p(w("vist")))
    res = w("res")
    L.ox_viscous_flux(g, mm, p, _p(o.q), _p(w("t")), _p(w("visl")), _p(w("vist")), *grads, _p(w("dtdx")),
                      _p(w("dtdy")), _p(w("dtdz")), _p(res))
    viscous = res[:, :nc].copy()
    L.ox_inviscid_flux(g, mm, p, _p(o.q), _p(w("gama")), *grads, _p(w("limit")), _p(res))
    assert o.q.shape == (5, nt)
    out = s.get(S.PHX_RES)[:, :nc]
    assert rel_err(out, res[:, :nc]) <= tol
    assert rel_err(out[4], res[4, :nc]) <= tol   # where a wall's velocity does work
    assert np.abs(viscous[4]).max() > 100 * tol * np.abs(res[4, :nc]).max()
