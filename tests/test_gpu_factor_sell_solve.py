"""A learned-smoother solve on a mesh large enough for the factor's sliced-ELL copies
(44^3 cells; the symmetry suite's solves are on smaller ones, in the lane form)."""
import numpy as np
import pytest

from test_gpu_multigrid import _cube, _hessian, _rhs, _solve

pytestmark = pytest.mark.gpu


def test_solve_over_the_factor_copies():
    from bartels_gb300 import lpcg
    plan, V, q, pinned = _cube(44)
    vals = _hessian(plan, q)
    b = _rhs(len(V), pinned)
    net = lpcg.LearnedPreconditioner.load(ctx=plan.ctx)
    x, lm = _solve(plan, vals, b, "learned_multigrid", net=net)
    A = plan.csr(vals.cpu().numpy().astype(np.float64))
    r = b.cpu().numpy() - A @ x
    r[np.repeat(pinned, 3)] = 0.0
    # the solver's own criterion, 1e-8 |b|, evaluated there in pairs of FP32 numbers
    assert lm.converged and np.linalg.norm(r) <= 1.01e-8 * np.linalg.norm(b.cpu().numpy())
    _, bj = _solve(plan, vals, b, "jacobi")
    assert lm.iterations <= 0.3 * bj.iterations  # as the smaller sizes are asked
    plan.close()
    net.close()
