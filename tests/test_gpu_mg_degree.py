"""BARTELS_MG_DEGC sets the degree of multigrid level 1 where the cluster kernel runs the
level too (unless BARTELS_MG_DEGCL says otherwise)."""
import numpy as np
import pytest

from test_gpu_coarse_cluster import _vcycle
from test_gpu_multigrid import _cube, _hessian, _rhs

pytestmark = pytest.mark.gpu


def test_degree_of_level_1(monkeypatch):
    def z(**env):
        for k in ("BARTELS_MG_DEGC", "BARTELS_MG_DEGCL"):
            monkeypatch.delenv(k, raising=False)
        for k, v in env.items():
            monkeypatch.setenv(k, v)
        plan, V, q, pinned = _cube(17)  # three levels, level 1 inside the cluster
        out = _vcycle(plan, _hessian(plan, q), _rhs(len(V), pinned).float())
        plan.close()
        return out

    four = z(BARTELS_MG_DEGC="4", BARTELS_MG_DEGCL="4")
    assert np.array_equal(z(BARTELS_MG_DEGC="4"), four)
    assert not np.array_equal(z(), four)
    assert np.array_equal(z(), z(BARTELS_MG_DEGCL="2"))
