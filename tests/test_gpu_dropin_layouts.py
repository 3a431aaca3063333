"""Element data by layout and meshes by content: row-major arrays (which go to the
device as they are), column-major, strided, FP32 and list forms give the same bits
for every law, and an in-place change of a mesh or of its data is seen."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MODELS = ["neohookean", "stvk", "corotational", "neohookean_isochoric", "arap", "linear_elasticity"]


def _case(model, n=3):
    import bartels_gb300 as bg
    from bartels_gb300.meshes import kuhn_cube, material_params
    V, E = kuhn_cube(n)
    rng = np.random.default_rng(n)
    q = (V * 1.02 + 0.02 * rng.uniform(-1, 1, V.shape)).ravel()
    params = material_params(model, len(E), 2e6, 0.45) * rng.uniform(0.5, 1, (len(E), 1))
    return V, E, q, bg.linear_tetmesh_dphi_dX(V, E), bg.volume(V, E), params


def _strided(a):
    b = np.zeros((len(a), 2 * a.shape[1]))
    b[:, ::2] = a
    return b[:, ::2]


@pytest.mark.parametrize("model", MODELS)
def test_layouts(model):
    import bartels_gb300 as bg
    V, E, q, dphi, vol, params = _case(model)
    plan = bg.MeshPlan(V, E)

    def both(d, v, p):
        return plan.q(model, q, d, v, p), plan.dq(model, q, d, v, p), plan.dq2_values(model, q, d, v, p)

    ref = both(np.asfortranarray(dphi), vol, np.asfortranarray(params))
    for d, v, p in ((dphi, vol, params), (_strided(dphi), vol.reshape(-1, 1), params), (dphi, list(vol), _strided(params)),
                    (dphi, vol, params.tolist()), (None, None, params), (dphi, None, None)):
        got = both(d, v, p)
        assert got[0] == ref[0] and (got[1] == ref[1]).all() and (got[2] == ref[2]).all()
    with pytest.raises(bg.BartelsError):
        plan.q(model, q, dphi + 1.0, vol, params)  # row 0 is not minus the others' sum
    plan.close()


def test_changes_in_place_are_seen():
    import bartels_gb300 as bg
    V, E, q, dphi, vol, params = _case("stvk")
    e0 = bg.linear_tetmesh_stvk_q(V, E, q, dphi, vol, params)
    params *= 2
    assert bg.linear_tetmesh_stvk_q(V, E, q, dphi, vol, params) == pytest.approx(2 * e0, rel=1e-13)
    params /= 2
    meshes = []
    for k in range(6):  # more meshes than are kept
        V *= 1.1
        d, v = bg.linear_tetmesh_dphi_dX(V, E), bg.volume(V, E)
        meshes.append((V.copy(), bg.linear_tetmesh_stvk_q(V, E, 1.02 * V.ravel(), d, v, params)))
    for W, e in meshes + meshes[::-1]:
        d, v = bg.linear_tetmesh_dphi_dX(W, E), bg.volume(W, E)
        assert bg.linear_tetmesh_stvk_q(W, E, 1.02 * W.ravel(), d, v, params) == e
