"""Per-segment reductions of a packed solve, cut into pieces of 2,048 DOFs.

Segments below one piece, just above it, of several pieces and of a single
tet's few DOFs in one plan; each must reach the direct FP64 solution."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_multigrid import SOL_TOL, _direct, _hessian, _plan, _rhs, _solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[8], [1, 7, 8, 10, 13], [13, 1, 1, 2]])
@pytest.mark.parametrize("kind", ["jacobi", "multigrid"])
def test_every_segment_reaches_the_direct_solution(sizes, kind):
    import bartels_gb300 as bg
    from bartels_gb300 import _lib
    from bartels_gb300.meshes import kuhn_cube, material_params
    Vs, Es, voff, toff = [], [], [0], [0]
    for n in sizes:
        V, E = kuhn_cube(n)
        Vs.append(V)
        Es.append(E + voff[-1])
        voff.append(voff[-1] + len(V))
        toff.append(toff[-1] + len(E))
    V, E = np.concatenate(Vs), np.concatenate(Es).astype(np.int32)
    pinned = np.abs(V[:, 2]) < 1e-12
    plan = _plan(V, E, material_params("neohookean", len(E), 2e6, 0.45), pinned)
    vo, to = np.array(voff, np.int32), np.array(toff, np.int64)
    _lib.check(bg.lib().bartels_plan_set_segments(plan.handle, len(sizes), vo.ctypes.data_as(C.POINTER(C.c_int)),
                                                  to.ctypes.data_as(C.POINTER(C.c_int64))), "set_segments")
    rng = np.random.default_rng(0)
    vals = _hessian(plan, V + 0.002 * rng.uniform(-1, 1, V.shape))
    b = _rhs(len(V), pinned)
    x, rep = _solve(plan, vals, b, kind)
    ref = _direct(plan, vals, b, pinned)
    assert rep.converged
    for q in range(len(sizes)):
        s = slice(3 * voff[q], 3 * voff[q + 1])
        assert np.linalg.norm(x[s] - ref[s]) <= SOL_TOL * np.linalg.norm(ref[s])
    plan.close()
