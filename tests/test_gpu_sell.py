"""The PCG loop's SpMV over the sliced-ELL copy of the values, against FP64.

Row lengths and counts at the layout's edges: one tet, vertex counts around a
slice (32 rows) and a window (256 rows), a shuffled numbering with uneven rows,
pinned rows, and meshes with enough slices for two and for one warp per slice (four
below that)."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu

# FP32 sums of up to ~90 products, each rounded at 6e-8 of |A||x|, in any order
TOL = 90 * 6e-8


def _mesh(kind):
    from bartels_gb300.meshes import kuhn_cube
    if kind == "tet":
        return np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1.0]]), np.array([[0, 1, 2, 3]], np.int32)
    if kind.startswith("strip"):  # a chain of tets over exactly n vertices
        n = int(kind[5:])
        t = np.arange(n)
        V = np.stack([np.cos(2.0 * t), np.sin(2.0 * t), 0.3 * t], 1)
        E = np.stack([t[:-3], t[1:-2], t[2:-1], t[3:]], 1).astype(np.int32)
        d = np.linalg.det(V[E[:, 1:]] - V[E[:, :1]])
        E[d < 0] = E[d < 0][:, [0, 2, 1, 3]]
        return V, E
    n = int(kind[4:])
    V, E = kuhn_cube(n)
    if kind.startswith("shuf"):
        rng = np.random.default_rng(n)
        p = rng.permutation(len(V))
        W = np.empty_like(V)
        W[p] = V
        E = p[E][rng.permutation(len(E))].astype(np.int32)
        V = W
    return V, E


@pytest.mark.parametrize("kind", ["tet", "strip31", "strip33", "strip255", "strip256", "strip257", "strip1000",
                                  "shuf9", "shuf20", "cube35", "cube44"])
@pytest.mark.parametrize("pin", [False, True])
def test_spmv_matches_fp64(kind, pin):
    torch = pytest.importorskip("torch")
    import bartels_gb300 as bg
    from bartels_gb300 import _lib
    V, E = _mesh(kind)
    plan = bg.MeshPlan(V, E)
    rng = np.random.default_rng(1)
    pinned = rng.uniform(size=len(V)) < 0.2 if pin else np.zeros(len(V), bool)
    plan.set_problem(pinned=pinned.astype(np.uint8))
    vals = rng.standard_normal(plan.nnz).astype(np.float32)
    x = rng.standard_normal(3 * len(V)).astype(np.float32)
    vd, xd = torch.from_numpy(vals).cuda(), torch.from_numpy(x).cuda()
    yd = torch.full_like(xd, np.nan)
    torch.cuda.synchronize()
    us = C.c_double()
    _lib.check(bg.lib().bartels_plan_pcg_spmv_time_d(plan.ctx.handle, plan.handle, C.c_void_p(vd.data_ptr()),
                                                     C.c_void_p(xd.data_ptr()), C.c_void_p(yd.data_ptr()), 1,
                                                     C.byref(us)), "spmv")
    plan.ctx.synchronize()
    rp, ci = plan.pattern()
    A = sp.csr_matrix((vals.astype(np.float64), ci, rp), shape=(len(x), len(x)))
    ref = A @ x.astype(np.float64)
    scale = abs(A) @ np.abs(x.astype(np.float64))
    ref[np.repeat(pinned, 3)] = 0.0
    assert np.all(np.abs(yd.cpu().numpy() - ref) <= TOL * scale + 1e-30)
    plan.close()
