"""The LU-SGS sweep schedules, replayed on the host (tests/schedule_replay.cpp):
every cell once with all its neighbours on the sweep's side, every shared-memory
slot holding the result that it is read for, and no wait that nothing ends, for
few and many warps, for cells with more neighbours than lanes, and for a
numbering without any order."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from phenlei_b200 import mesh as M

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "phenlei_b200", "csrc")


@pytest.fixture(scope="module")
def replay(tmp_path_factory):
    lib = str(tmp_path_factory.mktemp("schedule") / "replay.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I/usr/local/cuda/include",
                    os.path.join(HERE, "schedule_replay.cpp"), os.path.join(CSRC, "phx_schedule.cpp"), "-o", lib],
                   check=True)
    return C.CDLL(lib)


def _graph(m, shuffled):
    nb, nf, nc = m.n_bface, m.n_face, m.n_cell
    number = np.random.default_rng(3).permutation(nc) if shuffled else np.arange(nc)
    left = number[m.left].astype(np.int32)
    right = np.array(m.right, np.int32)
    right[:nb] = nc + np.arange(nb)
    right[nb:] = number[right[nb:]]
    cell = np.concatenate([left, right[nb:]])
    face = np.concatenate([np.arange(nf), np.arange(nb, nf)])
    c2f = face[np.lexsort((face, cell))].astype(np.int32)
    off = np.concatenate([[0], np.cumsum(np.bincount(cell, minlength=nc))]).astype(np.int32)
    return off, c2f, left, right


MESHES = {
    "one_cell_wide": lambda: M.channel_bump(40, 1, 1, wall_spacing=0.5),
    "hex": lambda: M.channel_bump(17, 9, 5),
    "prism": lambda: M.channel_bump(24, 13, 7, thickness=0.08, prism_layers=5),
    "plate": lambda: M.flat_plate(20, 12, 6, first_spacing=1e-3),
    "tets": lambda: M.tet_cube(5),
}


@pytest.mark.parametrize("warps", [1, 3, 2368])
@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("name", sorted(MESHES))
def test_schedule_replays(replay, name, shuffled, warps):
    m = MESHES[name]()
    nb, nc = m.n_bface, m.n_cell
    off, c2f, left, right = _graph(m, shuffled)
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    for forward in (1, 0):
        used = C.c_int()
        assert replay.replay(nc, nb, p(off), p(c2f), p(left), p(right), forward, warps, C.byref(used)) == 0
        assert 1 <= used.value <= warps


@pytest.mark.parametrize("name,make,shuffled,rows,share", [
    # ducts and small blocks in order: chains, one row a level on the longest warp
    ("1_wide", lambda: M.channel_bump(400, 1, 1), False, 1.0, 1.0),
    ("3_wide", lambda: M.channel_bump(300, 3, 1), False, 1.0, 1.0),
    ("3x2_wide", lambda: M.channel_bump(200, 3, 2), False, 1.0, 0.7),
    ("4x4_wide", lambda: M.channel_bump(100, 4, 4), False, 1.0, 0.65),
    ("small", lambda: M.channel_bump(8, 6, 2), False, 1.0, 0.7),
    # a few thousand cells at random: still about a row a level
    ("few_at_random", lambda: M.channel_bump(16, 8, 8), True, 1.75, 0.2),
    # many cells at random: full rows dealt out, nothing held
    ("many_at_random", lambda: M.channel_bump(64, 48, 32), True, None, 0.0),
])
def test_which_schedule_is_taken(replay, name, make, shuffled, rows, share):
    """Rows of the longest warp a level at most (None: dealt-out rows, 1.3 times
    the full rows at most) and the share of held neighbours at least."""
    m = make()
    nc = m.n_cell
    off, c2f, left, right = _graph(m, shuffled)
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    for forward in (1, 0):
        out = (C.c_double * 4)()
        replay.shape(nc, m.n_bface, p(off), p(c2f), p(left), p(right), forward, 2368, out)
        total, _, longest, held = out
        assert replay.replay(nc, m.n_bface, p(off), p(c2f), p(left), p(right), forward, 2368, C.byref(C.c_int())) == 0
        lev = np.zeros(nc, int)
        for c in range(nc) if forward else range(nc - 1, -1, -1):
            f = c2f[off[c]:off[c + 1]]
            f = f[f >= m.n_bface]
            o = np.where(left[f] == c, right[f], left[f])
            o = o[o < c] if forward else o[o > c]
            lev[c] = lev[o].max() + 1 if len(o) else 0
        if rows is None:
            assert total <= 1.3 * nc / 8 and held < 0.01
        else:
            assert longest <= rows * (lev.max() + 1) and held >= share
