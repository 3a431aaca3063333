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


def test_packed_segments():
    import ctypes as C
    import bartels_gb300 as bg
    from bartels_gb300 import _lib
    from bartels_gb300.meshes import kuhn_cube, material_params
    from test_gpu_multigrid import _hessian, _plan as make_plan, _rhs, _solve
    Vs, Es, voff, toff = [], [], [0], [0]
    for n in (2, 9, 5):
        V, E = kuhn_cube(n)
        Vs.append(V)
        Es.append(E + voff[-1])
        voff.append(voff[-1] + len(V))
        toff.append(toff[-1] + len(E))
    V, E = np.concatenate(Vs), np.concatenate(Es).astype(np.int32)
    pinned = np.abs(V[:, 2]) < 1e-12
    vo, to = np.array(voff, np.int32), np.array(toff, np.int64)

    def make():
        plan = make_plan(V, E, material_params("neohookean", len(E), 2e6, 0.45), pinned)
        return plan, _hessian(plan, V + 0.002 * np.random.default_rng(0).uniform(-1, 1, V.shape))

    def call(state):
        plan, vals = state
        _lib.check(bg.lib().bartels_plan_set_segments(plan.handle, 3, vo.ctypes.data_as(C.POINTER(C.c_int)),
                                                      to.ctypes.data_as(C.POINTER(C.c_int64))), "set_segments")
        x, rep = _solve(plan, vals, _rhs(len(V), pinned), "jacobi")
        assert rep.converged
        return x

    _sweep(make, call, 60)


@pytest.mark.parametrize("what", ["factor", "train"])
def test_learned_preconditioner(what):
    from bartels_gb300 import lpcg
    from bartels_gb300.lpcg import LearnedPreconditioner
    from test_gpu_multigrid import _rhs, _torch
    torch = _torch()

    class Both:  # a plan and its network, closed together
        def __init__(self, plan, net):
            self.plan, self.net = plan, net

        def close(self):
            self.plan.close()
            self.net.close()

    values = _with_values(5)

    def make():
        plan, V, vals, pinned = values()
        net = LearnedPreconditioner.load(ctx=plan.ctx)
        if what == "factor":
            net.attach(plan)
        return Both(plan, net), V, vals, pinned

    def call(state):
        both, V, vals, pinned = state
        if what == "train":
            loss = both.net.train_step(both.plan, vals, None, nprobes=2, seed=3, lr=0.0)
            return np.append(both.net.grad(), loss)
        b = _rhs(len(V), pinned)
        x = torch.zeros_like(b)
        assert lpcg.plan_pcg(both.plan, vals, b, x, rel_tol=1e-8, max_iters=20000).converged
        return x.cpu().numpy()

    _sweep(make, call, 120)


@pytest.mark.parametrize("kind", ["multigrid", "learned_multigrid"])
def test_multigrid_solve(kind):
    import bartels_gb300 as bg
    from bartels_gb300.lpcg import LearnedPreconditioner
    net = LearnedPreconditioner.load(ctx=bg.Context.default())
    _sweep(_with_values(8), _solver(kind, net), 160)
    net.close()
