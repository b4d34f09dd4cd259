"""The residual history of one call: a context has room for some thousands of
steps from its creation, and a longer call makes room for itself.  One call of
5000 steps, calls that grow, and single steps give the same history."""
import numpy as np
import pytest

from phenlei_b200 import cases
from phenlei_b200 import mesh as M
from phenlei_b200 import solver as S
from tests.conftest import rel_err

pytestmark = pytest.mark.gpu


def test_long_and_growing_calls_give_the_same_history():
    m = M.channel_bump(8, 4, 2)
    out = []
    for calls in ([5000], [1, 3, 0, 96, 4900], [2500] * 2):
        s = S.NSSolverUnstruct(m, **cases.EULER_BUMP)
        out.append(np.concatenate([s.Relaxation(n) for n in calls]))
        s.close()
    assert out[0].shape == (5000,) and np.isfinite(out[0]).all()
    # 64 cells: the monitor's blocks add in any order, and a history near 1e-17 is rounding alone
    for h in out[1:]:
        assert rel_err(h[:200], out[0][:200]) <= 1e-12 and np.abs(h - out[0]).max() <= 1e-12 * out[0].max()
