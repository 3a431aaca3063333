"""Energy and gradient on the device against the oracle where the FP64 laws
change form: volume ratios over the rows of the logarithm's table and past its
end, rotations of every quaternion branch, and inverted elements, whose
corotational law takes the general SVD."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# The oracle's textbook energy cancels to eps mu / psi ~ 1e-13 at these strains.
TOL = 1e-11

_AXES = {"x": (1, -1, -1), "y": (-1, 1, -1), "z": (-1, -1, 1), "none": (1, 1, 1)}


@pytest.mark.parametrize("model", ["neohookean", "neohookean_isochoric", "stvk", "corotational", "arap"])
@pytest.mark.parametrize("scale,turn", [(0.72, "none"), (0.9, "x"), (1.0, "y"), (1.06, "z"), (1.18, "none"), (1.6, "x")])
def test_energy_and_gradient(model, scale, turn):
    import bartels_gb300 as bg
    from bartels_gb300.meshes import kuhn_cube, material_params
    from oracle import oracle as o
    V, E = kuhn_cube(4)
    rng = np.random.default_rng(int(100 * scale))
    q = (scale * V * np.array(_AXES[turn]) + 0.02 * rng.uniform(-1, 1, V.shape)).ravel()
    _compare(bg, o, material_params(model, len(E), 2e6, 0.45), model, V, E, q)


@pytest.mark.parametrize("model", ["corotational", "arap", "stvk"])
def test_inverted_elements(model):
    import bartels_gb300 as bg
    from bartels_gb300.meshes import kuhn_cube, material_params
    from oracle import oracle as o
    V, E = kuhn_cube(3)
    rng = np.random.default_rng(9)
    q = (V * np.array([1.0, -0.8, 1.1]) + 0.02 * rng.uniform(-1, 1, V.shape)).ravel()
    _compare(bg, o, material_params(model, len(E), 2e6, 0.45), model, V, E, q)


def _compare(bg, o, params, model, V, E, q):
    dphi, vol = o.dphi_dX(V, E), o.volume(V, E)
    plan = bg.MeshPlan(V, E)
    e = plan.q(model, q, dphi, vol, params)
    ref = o.tetmesh_q(model, E, q, dphi, vol, params)
    assert abs(e - ref) <= TOL * abs(ref)
    g = plan.dq(model, q, dphi, vol, params)
    gr = o.tetmesh_dq(model, len(V), E, q, dphi, vol, params)
    assert np.abs(g - gr).max() <= TOL * np.abs(gr).max()
    plan.close()
