"""Small block-Jacobi solves as one cluster launch per inner solve.

Sizes around the split of the rows over the cluster (16 CTAs of whole groups of
96 rows), counts that are not whole 3x3 blocks, rows longer than what shared
memory stages, one row that holds the whole system, the largest size that takes
this path and the first that does not, and right-hand sides whose squares leave
the float range (which take the general path)."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu

REL = 1e-10  # the solver's own criterion: |b - A x| <= REL |b|, evaluated here in FP64


def _spd(n, band, seed, hub=False):
    rng = np.random.default_rng(seed)
    offs = np.unique(rng.integers(1, max(2, min(n, 3 * band)), band)) if n > 1 else []
    d = [rng.uniform(-1, 1, max(n - o, 0)) for o in offs if o < n]
    A = sp.diags(d, [o for o in offs if o < n], shape=(n, n)) if d else sp.csr_matrix((n, n))
    if hub and n > 2:
        r = sp.csr_matrix((rng.uniform(-1, 1, n - 1), (np.zeros(n - 1, int), np.arange(1, n))), shape=(n, n))
        A = A + r
    A = A + A.T
    A = A + sp.diags(np.asarray(abs(A).sum(axis=1)).ravel() + rng.uniform(0.1, 1.0, n))
    A = A.tocsr()
    A.sort_indices()
    return A


@pytest.mark.parametrize("n,band,hub", [(1, 0, False), (2, 1, False), (4, 2, False), (95, 6, True), (1535, 9, False),
                                        (1536, 9, False), (1537, 9, True), (3001, 120, False), (10080, 40, False),
                                        (24575, 20, False), (24576, 60, False), (24577, 20, False)])
@pytest.mark.parametrize("scale", [1.0, 1e18])
def test_search_direction_meets_its_residual(n, band, hub, scale):
    import bartels_gb300 as bg
    A = _spd(n, band, n, hub)
    g = scale * np.random.default_rng(n + 1).standard_normal(n)
    d, ok, rep = bg.search_direction_newton_sparse(g, A, rel_tol=REL)
    assert ok and rep.converged
    r = np.linalg.norm(-g - A @ d)
    assert r <= 1.001 * REL * np.linalg.norm(g)


def test_an_iteration_cap_is_reported():
    import bartels_gb300 as bg
    A = _spd(3000, 20, 5)
    g = np.random.default_rng(1).standard_normal(3000)
    d, ok, rep = bg.search_direction_newton_sparse(g, A, rel_tol=REL, max_iters=3)
    assert not ok and rep.iterations <= 3 and np.isfinite(d).all()
