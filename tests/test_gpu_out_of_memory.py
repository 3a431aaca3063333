"""A device allocation that fails leaves an error, and no half-built state: the
next call builds again and gives the same bits.

Each allocation of a call is made to fail in turn (reported by the library instead
of being made), on a new plan. What a plan keeps between calls has to be published
only when it is complete, or the next call would hand kernels null pointers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _plan(n, seed=1):
    from bartels_gb300.meshes import kuhn_cube, material_params
    from test_gpu_multigrid import _plan as make
    V, E = kuhn_cube(n)
    pinned = np.abs(V[:, 2]) < 1e-12
    q = V + 0.05 / n * np.random.default_rng(seed).uniform(-1, 1, V.shape)
    return make(V, E, material_params("neohookean", len(E), 2e6, 0.45), pinned), V, q, pinned


def _sweep(make, call, at_most):
    """call(state) on make()'s state: undisturbed, then with its 1st, 2nd, ... allocation failing."""
    import bartels_gb300 as bg
    L = bg.lib()
    state = make()
    ref = call(state)
    state[0].close()
    for k in range(1, at_most):
        state = make()
        L.bartels_fail_alloc(k)
        try:
            got = call(state)
        except bg.BartelsError:
            got = None
        left = L.bartels_fail_alloc(0)
        if left == 0:  # it was reported: the plan still works
            for _ in range(2):
                assert np.array_equal(call(state), ref), k
        state[0].close()
        if left:
            assert k > 1 and np.array_equal(got, ref)
            return
    raise AssertionError("more allocations than expected")


def _solver(kind, net=None):
    from test_gpu_multigrid import _rhs, _solve

    def call(state):
        plan, V, vals, pinned = state
        x, rep = _solve(plan, vals, _rhs(len(V), pinned), kind, **({} if net is None else {"net": net}))
        assert rep.converged
        return x
    return call


def _with_values(n):
    from test_gpu_multigrid import _hessian

    def make():
        plan, V, q, pinned = _plan(n)
        return plan, V, _hessian(plan, q), pinned
    return make


@pytest.mark.parametrize("n", [6, 21])  # the cluster's small solve, and the loop over the sliced-ELL copy
def test_block_jacobi_solve(n):
    _sweep(_with_values(n), _solver("jacobi"), 30)
