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
    return C.CDLL(lib).replay


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
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    for forward in (1, 0):
        used = C.c_int()
        assert replay(nc, nb, p(off), p(c2f), p(left), p(right), forward, warps, C.byref(used)) == 0
        assert 1 <= used.value <= warps
