"""The multigrid's coarse levels as one thread-block cluster launch.

How the coarse nodes are split over the cluster's CTAs changes no arithmetic
within a row, only which CTA computes it and how many lanes share a row, so
the V-cycle must agree across cluster sizes to FP32 rounding; and the split
must not show in the solution. Sizes: the coarsest (dense) level alone, a
level-1 of a few dozen nodes, level 1 inside and outside the cluster's shared
memory, a dense level at its upper limit; four CTAs up to sixteen, with more
CTAs than nodes."""
import numpy as np
import pytest

from test_gpu_multigrid import _cube, _direct, _hessian, _rhs, _solve

pytestmark = pytest.mark.gpu

# z is a fixed polynomial in FP32 operators: each of ~40 dependent steps rounds at 6e-8, the 6x6 row sums
# of up to 30 blocks at ~1e-6 worst case
AGREE = 2e-5


def _vcycle(plan, vals, r):
    import torch
    from bartels_gb300 import lpcg
    lpcg.use_multigrid(plan)
    z = torch.zeros_like(r)
    lpcg.precond_apply(plan, vals, r, z)
    return z.double().cpu().numpy()


@pytest.mark.parametrize("n", [2, 3, 9, 17, 30, 44])
def test_vcycle_does_not_depend_on_the_cluster_size(n, monkeypatch):
    ref = None
    for ctas in (16, 4, 7, 8):
        monkeypatch.setenv("BARTELS_MG_CLUSTER", str(ctas))
        monkeypatch.setenv("BARTELS_MG_DEGCL", "1")  # the same polynomial whether or not level 1 is in the cluster
        plan, V, q, pinned = _cube(n)  # the hierarchy is built with the plan's first solve
        vals = _hessian(plan, q)
        r = _rhs(len(V), pinned).float()
        z = _vcycle(plan, vals, r)
        plan.close()
        if ref is None:
            ref = z
            assert np.linalg.norm(ref) > 0 and np.all(ref[np.repeat(pinned, 3)] == 0.0)
        assert np.linalg.norm(z - ref) <= AGREE * np.linalg.norm(ref), ctas


@pytest.mark.parametrize("n", [3, 9, 13])
def test_solution_through_the_cluster_matches_the_direct_solve(n):
    plan, V, q, pinned = _cube(n, seed=n)
    vals = _hessian(plan, q)
    b = _rhs(len(V), pinned)
    x, rep = _solve(plan, vals, b, "multigrid")
    x_ref = _direct(plan, vals, b, pinned)
    assert rep.converged
    assert np.linalg.norm(x - x_ref) <= 1e-6 * np.linalg.norm(x_ref)
    plan.close()
