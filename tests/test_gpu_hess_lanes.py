"""The assembly kernel with one, two and four lanes per vertex, against the oracle.

Mesh sizes on all sides of the rule that picks the lane count (four up to 128
vertices per SM, one for the cheap laws from 190 up to three chunks per SM, two
elsewhere; on 152 SMs 22.0k is above the first line, 42.9k between the others), and a
shuffled numbering with uneven incidence counts; with and without projection,
and under both CTA shapes (whose values must be the same bits)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-5  # FP32 element Hessians: per row, of the row's largest entry (as the parity suite)


def _mesh(kind):
    from bartels_gb300.meshes import kuhn_cube
    n = int(kind[4:])
    V, E = kuhn_cube(n)
    if kind.startswith("shuf"):
        rng = np.random.default_rng(n)
        p = rng.permutation(len(V))
        W = np.empty_like(V)
        W[p] = V
        V, E = W, p[E][rng.permutation(len(E))].astype(np.int32)
    return V, E, 1.0 / n


@pytest.mark.parametrize("kind", ["cube1", "cube3", "shuf4", "shuf12", "cube27", "shuf34"])
@pytest.mark.parametrize("psd", [None, 1e-6])
def test_values_match_the_oracle(kind, psd):
    import bartels_gb300 as bg
    from bartels_gb300 import _lib
    from bartels_gb300.meshes import material_params
    from oracle import oracle as o
    V, E, h = _mesh(kind)
    rng = np.random.default_rng(2)
    q = (V * np.array([0.97, 1.0, 0.95]) + 0.02 * h * rng.uniform(-1, 1, V.shape)).ravel()
    params = material_params("neohookean", len(E), 2e6, 0.45)
    dphi, vol = o.dphi_dX(V, E), o.volume(V, E)
    plan = bg.MeshPlan(V, E)
    H = plan.dq2("neohookean", q, dphi, vol, params, psd_tol=psd)
    ref = o.tetmesh_dq2("neohookean", len(V), E, q, dphi, vol, params, psd_tol=psd)
    assert (H.indptr == ref.indptr).all() and (H.indices == ref.indices).all()
    rowmax = np.maximum.reduceat(np.abs(ref.data), ref.indptr[:-1])
    err = np.maximum.reduceat(np.abs(H.data - ref.data), ref.indptr[:-1])
    assert (err <= TOL * rowmax).all(), (err / rowmax).max()
    for chunk in (128, 64):
        _lib.check(bg.lib().bartels_plan_set_hessian_tuning(plan.handle, chunk, 128), "tuning")
        assert (plan.dq2_values("neohookean", q, dphi, vol, params, psd_tol=psd) == H.data).all()
    plan.close()
