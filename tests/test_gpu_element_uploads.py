"""Element data whose upload reads host memory that the library owns.

Column-major parameters are laid out per tet in a buffer of the call, and linear
elasticity's (E, nu) become (lambda, mu) in another; both must live until the
device has read them. On 105k tets (1.7 MB of parameters), with the host's memory
reused at once after each call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _reuse():
    """Allocations of the sizes that the calls above have just freed, filled with rubbish."""
    return [np.full(n, 7e33) for n in (2 * 6 * 26 ** 3, 6 * 26 ** 3, 3 * 27 ** 3)]


@pytest.mark.parametrize("model", ["stvk", "linear_elasticity"])
def test_parameters_reach_the_device(model):
    import bartels_gb300 as bg
    from bartels_gb300 import _lib
    from bartels_gb300.api import MODELS, _dptr
    from bartels_gb300.meshes import kuhn_cube, material_params
    V, E = kuhn_cube(26)
    rng = np.random.default_rng(0)
    q = (1.02 * V + 1e-3 * rng.uniform(-1, 1, V.shape)).ravel()
    params = material_params(model, len(E), 2e6, 0.45) * rng.uniform(0.5, 1.0, (len(E), 1))
    plan = bg.MeshPlan(V, E)
    lam = params
    if model == "linear_elasticity":
        young, nu = params.T
        lam = np.stack([young * nu / ((1 + nu) * (1 - 2 * nu)), young / (2 * (1 + nu))], 1)
    plan.set_element_data(params=lam)  # the plan's own form, waited for
    ref = plan.q(model, q), plan.dq(model, q)
    L = bg.lib()
    for _ in range(3):
        for form in ("rows", "columns"):
            plan.set_element_data(params=np.ones_like(params))
            if form == "rows":
                p = params.copy()
                _lib.check(L.bartels_plan_set_element_rows(plan.handle, MODELS[model], None, None, _dptr(p)), "rows")
                got = None
            else:
                p = np.ascontiguousarray(params.T)
                got = plan.q(model, q, params=np.asfortranarray(params))
            junk = _reuse()
            if got is None:
                got = plan.q(model, q)
            assert got == ref[0]
            assert (plan.dq(model, q) == ref[1]).all()
            del junk, p
    plan.close()
