"""The autotuner's choice reaches the kernel that the solves run: the PCG loop's SpMV
over the sliced-ELL copy takes the tuned warps per slice, a second plan of the size
bucket takes them from the cache, and the solution has the residual it should."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_multigrid import _cube, _hessian, _rhs, _solve

pytestmark = pytest.mark.gpu


def _tuning(plan):
    import bartels_gb300 as bg
    from bartels_gb300 import _lib
    v = [C.c_int(-1) for _ in range(3)]
    _lib.check(bg.lib().bartels_plan_tuning(plan.handle, *[C.byref(x) for x in v]), "tuning")
    return tuple(x.value for x in v)


@pytest.mark.parametrize("n", [24, 31])  # 15.6k and 32.8k vertices: the general loop, buckets of their own
def test_tuned_split(n):
    import bartels_gb300 as bg
    from bartels_gb300 import _lib
    seen = []
    for force in (1, 0):
        plan, V, q, pinned = _cube(n)
        assert _tuning(plan) == (0, 0, 0)
        vals = _hessian(plan, q)
        a, b = C.c_int(), C.c_int()
        _lib.check(bg.lib().bartels_plan_autotune(plan.ctx.handle, plan.handle, C.c_void_p(vals.data_ptr()), force,
                                                  C.byref(a), C.byref(b)), "tune")
        split, lanes, tri = _tuning(plan)
        assert split in (1, 2, 4) and (lanes, tri) == (a.value, b.value)
        seen.append((split, lanes, tri))
        rhs = _rhs(len(V), pinned)
        x, rep = _solve(plan, vals, rhs, "jacobi")
        A = plan.csr(vals.cpu().numpy().astype(np.float64))
        b = rhs.cpu().numpy()
        r = b - A @ x
        r[np.repeat(pinned, 3)] = 0.0
        # the solver's own criterion, 1e-8 |b|, evaluated there in pairs of FP32 numbers
        assert rep.converged and np.linalg.norm(r) <= 1.01e-8 * np.linalg.norm(b)
        plan.close()
    assert seen[0] == seen[1]
