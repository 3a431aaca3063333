"""The learned smoother over the factor's sliced-ELL copies: with G and G^T from
two layouts the V-cycle must still be symmetric, positive and zero on pinned rows,
and its solves must need few iterations. Vertex counts around a slice and a window,
and a mesh large enough for the sliced-ELL form (44^3; smaller ones keep the lane form)."""
import numpy as np
import pytest

from test_gpu_multigrid import _cube, _hessian, _rhs, _solve, _torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 6, 17, 35, 44])
def test_learned_vcycle_is_symmetric(n):
    torch = _torch()
    from bartels_gb300 import lpcg
    plan, V, q, pinned = _cube(n)
    vals = _hessian(plan, q)
    net = lpcg.LearnedPreconditioner.load(ctx=plan.ctx)
    net.attach(plan, multigrid=True)
    mask = torch.from_numpy(np.repeat(~pinned, 3).astype(np.float32)).cuda()
    g = torch.Generator(device="cuda").manual_seed(n)
    rs = [torch.randn(3 * len(V), device="cuda", generator=g) * mask for _ in range(3)]
    zs = []
    for r in rs:
        z = torch.empty_like(r)
        lpcg.precond_apply(plan, vals, r, z)
        zs.append(z.double())
    for i in range(3):
        assert float(rs[i].double() @ zs[i]) > 0.0
        assert torch.all(zs[i][~mask.bool()] == 0)
        for j in range(i):
            a, c = float(rs[j].double() @ zs[i]), float(rs[i].double() @ zs[j])
            # FP32 sums of a V-cycle, as in the multigrid suite
            assert abs(a - c) <= 2e-5 * float(torch.linalg.norm(rs[i].double()) * torch.linalg.norm(zs[j])), (i, j)
    if n in (17, 35):
        b = _rhs(len(V), pinned)
        _, bj = _solve(plan, vals, b, "jacobi")
        _, lm = _solve(plan, vals, b, "learned_multigrid", net=net)
        assert lm.converged and lm.iterations <= 0.3 * bj.iterations
    net.close()
    plan.close()
