"""phx_ns_relaxation runs the SA sweeps and update of a step on a second stream
beside the next step's boundary, gradient and residual.  PHX_OVERLAP=0 runs
every phase in order: the states after several steps are the same bit for bit,
for every gradient (GG-node forms node values after the SA update) and with the
learned source, on a mesh whose passes take longer than its sweeps and on one
where it is the other way round."""
import numpy as np
import pytest

from phenlei_b200 import cases
from phenlei_b200 import mesh as M
from phenlei_b200 import solver as S
from tests.conftest import rel_err

pytestmark = pytest.mark.gpu

MESHES = {"bump": lambda: M.channel_bump(48, 24, 24, thickness=0.08, prism_layers=6),
          "long": lambda: M.channel_bump(160, 6, 4)}


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("grad,source", [("ggcell", "exact"), ("lsq", "exact"), ("ggnode", "exact"),
                                         ("ggcell", "mlp_fallback")])
@pytest.mark.parametrize("mesh", sorted(MESHES))
def test_overlapped_steps_equal_steps_in_order(monkeypatch, mesh, grad, source, precision):
    m = MESHES[mesh]()
    wd = M.wall_distance(m)
    params = dict(cases.SA_BUMP, gradientName=grad, sa_source=source, flowInitStep=2)
    q0 = cases.perturbed_state(m, params, seed=8)
    blob, out, hist = None, [], []
    for overlap in ("0", "1"):
        monkeypatch.setenv("PHX_OVERLAP", overlap)
        s = S.NSSolverUnstruct(m, precision=precision, wall_dist=wd, **params)
        if source != "exact":
            if blob is None:
                a = S.NSSolverUnstruct(m, wall_dist=wd, **dict(params, sa_source="exact"))
                a.Relaxation(3)
                f, t, _, _ = a.capture_sa_samples()
                a.train_sa_mlp(f, t, epochs=2, batch=512, seed=1)
                blob = a.mlp_blob()
                a.close()
            s.set_mlp_blob(blob)
        s.set_q_cells(q0)
        hist.append(np.concatenate([s.Relaxation(5), s.Relaxation(3)]))
        out.append([s.get(a) for a in (S.PHX_Q, S.PHX_DQ, S.PHX_Q_TURB, S.PHX_VIST, S.PHX_VISL, S.PHX_RES,
                                       S.PHX_RES_TURB, S.PHX_GRAD_TURB)])
        s.close()
    # the monitor's sum over the blocks is taken as they end: the order of a thousand FP64 terms
    assert rel_err(hist[1], hist[0]) <= 1e-13
    for a, b in zip(*out):
        assert np.isfinite(a).all() and np.array_equal(a, b)
