"""The weight gradient's register tiles at row counts around them: fewer rows
than one tile of 32, one part of 64 rows and a remainder, and several parts; with
and without the residual probe, and on a system whose gradient follows a larger one
through the same network (the partials' scratch is reused)."""
import numpy as np
import pytest

from oracle import lpcg as L
from test_gpu_lpcg import _system, _theta

pytestmark = pytest.mark.gpu


def _check(net, th, n, seed):
    plan, vals, g, A = _system(n, seed=seed)
    npr = 3
    loss = net.train_step(plan, vals, None, nprobes=npr, seed=seed, lr=0.0)
    grad = net.grad().astype(np.float64)
    ref_loss, ref, _ = L.loss_and_grad(g, A, th.astype(np.float64), L.rademacher(seed, npr, 3 * g.nV), bf=True)
    assert abs(loss - ref_loss) <= 1e-4 * max(1.0, abs(ref_loss))
    # BF16 operands of the tensor-core products, as in the suite of the whole network
    assert np.linalg.norm(grad - ref) <= 3e-2 * np.linalg.norm(ref)
    for name, (o, s) in L.LAYOUT.items():
        k = int(np.prod(s))
        if np.linalg.norm(ref[o:o + k]) > 1e-6 * np.linalg.norm(ref):
            assert np.linalg.norm(grad[o:o + k] - ref[o:o + k]) <= 5e-2 * np.linalg.norm(ref[o:o + k]), name
    plan.close()
    return grad


@pytest.mark.parametrize("sizes", [(2,), (3,), (5,), (7, 2)])
def test_gradient_matches_oracle(sizes):
    import bartels_gb300 as bg
    from bartels_gb300.lpcg import LearnedPreconditioner
    th = _theta(4)
    net = LearnedPreconditioner(bg.Context.default(), params=th)
    for i, n in enumerate(sizes):
        a = _check(net, th, n, 11 + i)
        assert np.array_equal(a, _check(net, th, n, 11 + i))  # fixed order
    net.close()
