"""Solver.marching_cubes raises the failed call's own error, after that call alone."""
import ctypes

import numpy as np
import pytest

import bubbles_gb300 as bb
from bubbles_gb300 import _native as N


class FailingLibrary:
    """bbg_marching_cubes counts the mesh, and fails where it would write it."""

    def __init__(self, status):
        self.status, self.calls = status, 0

    def bbg_marching_cubes(self, h, grid, values, iso, rotate, points, normals, np_cap, triangles, nt_cap, npt, ntr):
        self.calls += 1
        ctypes.cast(npt, ctypes.POINTER(ctypes.c_size_t))[0] = 3
        ctypes.cast(ntr, ctypes.POINTER(ctypes.c_size_t))[0] = 1
        return 4 if points is None else self.status

    def bbg_last_error(self):
        return b"marching cubes: as told"


@pytest.mark.parametrize("status", [1, 2, 3])
def test_the_error_is_the_calls_own(monkeypatch, status):
    lib = FailingLibrary(status)
    monkeypatch.setattr(N, "load", lambda: lib)
    monkeypatch.setattr(N, "_lib", lib)
    s = bb.Solver.__new__(bb.Solver)
    s.h = None
    with pytest.raises(bb.BbgError) as e:
        s.marching_cubes((2, 2, 2), (0, 0, 0), 0.1, np.zeros(8, np.float32))
    assert e.value.status == status and "as told" in str(e.value)
    assert lib.calls == 1
