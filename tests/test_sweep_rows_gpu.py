"""The LU-SGS sweeps on few warps (every warp then runs many chains, and the
shared-memory slots are reused) give the results of the full grid bit for bit:
the sums of every cell are taken in the same order.  A grid of one, of three
warps, and of more than a mesh of this size fills, on hexahedra, prisms (cells of
seven faces) and tetrahedra, both precisions, with and without the SA sweep."""
import numpy as np
import pytest

from phenlei_b200 import cases
from phenlei_b200 import mesh as M
from phenlei_b200 import solver as S

pytestmark = pytest.mark.gpu

CASES = {
    "hex": (lambda: M.channel_bump(23, 11, 5), cases.EULER_BUMP),
    "prism_sa": (lambda: M.channel_bump(24, 13, 7, thickness=0.08, prism_layers=5), cases.SA_BUMP),
    "tets": (lambda: M.tet_cube(6), dict(cases.LAMINAR, gradientName="lsq")),
}


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_few_warps_give_the_same_bits(monkeypatch, name, precision):
    make, params = CASES[name]
    m = make()
    wd = M.wall_distance(m) if params["viscousType"] == 3 else None
    q0 = cases.perturbed_state(m, params, seed=4)
    out = []
    for warps in (None, "1", "3"):
        if warps is None:
            monkeypatch.delenv("PHX_LUSGS_MAX_BLOCKS", raising=False)
        else:
            monkeypatch.setenv("PHX_LUSGS_MAX_BLOCKS", warps)
        s = S.NSSolverUnstruct(m, precision=precision, wall_dist=wd, **params)
        s.set_q_cells(q0)
        s.Relaxation(2)
        out.append([s.get(S.PHX_Q), s.get(S.PHX_DQ)] + ([s.get(S.PHX_Q_TURB)] if wd is not None else []))
        s.close()
    for other in out[1:]:
        for a, b in zip(out[0], other):
            assert np.isfinite(a).all() and np.array_equal(a, b)
