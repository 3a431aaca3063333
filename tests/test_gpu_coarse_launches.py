"""The multigrid's coarse levels as a launch per level, the form for a device that
cannot host the cluster: the same V-cycle as the cluster launch to FP32 rounding,
with a dense coarsest level alone, below one level and below several, and with a
block-diagonal one (packed meshes)."""
import numpy as np
import pytest

from test_gpu_coarse_cluster import AGREE, _vcycle
from test_gpu_multigrid import _cube, _direct, _hessian, _rhs, _solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 9, 17, 30])
def test_vcycle_agrees_with_the_cluster_launch(n, monkeypatch):
    zs = []
    for ctas in ("16", "0"):
        monkeypatch.setenv("BARTELS_MG_CLUSTER", ctas)
        monkeypatch.setenv("BARTELS_MG_DEGCL", "1")  # the same polynomial on level 1
        plan, V, q, pinned = _cube(n)
        vals = _hessian(plan, q)
        zs.append(_vcycle(plan, vals, _rhs(len(V), pinned).float()))
        plan.close()
    assert np.linalg.norm(zs[0]) > 0
    assert np.linalg.norm(zs[1] - zs[0]) <= AGREE * np.linalg.norm(zs[0])


@pytest.mark.parametrize("n", [3, 13])
def test_solution(n, monkeypatch):
    monkeypatch.setenv("BARTELS_MG_CLUSTER", "0")
    plan, V, q, pinned = _cube(n, seed=n)
    vals = _hessian(plan, q)
    b = _rhs(len(V), pinned)
    x, rep = _solve(plan, vals, b, "multigrid")
    ref = _direct(plan, vals, b, pinned)
    assert rep.converged and np.linalg.norm(x - ref) <= 1e-6 * np.linalg.norm(ref)
    plan.close()


def test_packed_meshes(monkeypatch):
    from test_gpu_segment_pieces import test_every_segment_reaches_the_direct_solution as packed
    monkeypatch.setenv("BARTELS_MG_CLUSTER", "0")
    packed([13, 1, 1, 2], "multigrid")
