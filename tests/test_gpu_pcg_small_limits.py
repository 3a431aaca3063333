"""Where the small solve's cluster cannot or must not be used: a device that cannot
host it, sums that leave the range of its float pairs; and what its size leaves
empty (CTAs without rows, pinned vertices)."""
import numpy as np
import pytest

from test_gpu_pcg_small import REL, _spd

pytestmark = pytest.mark.gpu


def _direction(A, g, **kw):
    import bartels_gb300 as bg
    d, ok, rep = bg.search_direction_newton_sparse(g, A, rel_tol=REL, **kw)
    assert ok and rep.converged
    assert np.linalg.norm(-g - A @ d) <= 1.001 * REL * np.linalg.norm(g)
    return d, rep


@pytest.fixture
def general(monkeypatch):
    """A default context on which the cluster counts as not hosted."""
    from bartels_gb300.api import Context
    monkeypatch.setenv("BARTELS_PCG_SMALL", "0")
    ctx = Context(0)
    monkeypatch.setattr(Context, "_default", ctx)
    yield ctx
    ctx.close()


@pytest.mark.parametrize("n,band,hub", [(1, 0, False), (4, 2, False), (1537, 9, True), (10080, 40, False)])
def test_the_general_loop_takes_over(n, band, hub, general):
    A = _spd(n, band, n, hub)
    before = general.kernel_launches
    _, rep = _direction(A, np.random.default_rng(n + 1).standard_normal(n))
    assert general.kernel_launches - before >= 3 * rep.iterations


def test_ctas_without_rows_many_times():
    """Up to 96 unknowns belong to the first CTA: the other fifteen only take part in the sums."""
    for n in (1, 3, 31, 96, 97):
        A = _spd(n, 4 if n > 1 else 0, n)
        g = np.random.default_rng(n).standard_normal(n)
        d0, rep0 = _direction(A, g)
        for _ in range(50):
            d, rep = _direction(A, g)
            assert np.array_equal(d, d0) and rep.iterations == rep0.iterations


@pytest.mark.parametrize("n", [1, 3, 13])
def test_pinned_plan(n):
    from test_gpu_multigrid import SOL_TOL, _cube, _direct, _hessian, _rhs, _solve
    plan, V, q, pinned = _cube(n)
    vals = _hessian(plan, q)
    b = _rhs(len(V), pinned)
    x, rep = _solve(plan, vals, b, "jacobi")
    ref = _direct(plan, vals, b, pinned)
    assert rep.converged and np.all(x[np.repeat(pinned, 3)] == 0.0)
    assert np.linalg.norm(x - ref) <= SOL_TOL * np.linalg.norm(ref)
    plan.close()


# r.z and p.Ap scale with 1 / A and A where b alone is of ordinary size. What the general loop takes has to be
# taken, and what it refuses (a warp's FP32 sum of r.z, ~96 b^2 / (18 a), leaves the range in the first case) is
# refused: sums of the whole system past the largest float while every warp's fits, sums near the smallest, ordinary
@pytest.mark.parametrize("n,a,b", [(10080, 1e-36, 10.0), (24576, 1e-36, 3.0), (10080, 1e-36, 1.0), (10080, 1e-30, 1.0),
                                   (10080, 1e15, 1.0), (3001, 1.0, 1e-4)])
def test_matrices_far_from_unit_scale(n, a, b, general, monkeypatch):
    import bartels_gb300 as bg
    from bartels_gb300.api import Context
    A = a * _spd(n, 20, n)
    g = b * np.random.default_rng(n).standard_normal(n)
    try:
        _direction(A, g)
        taken = True
    except bg.BartelsError:
        taken = False
    monkeypatch.setattr(Context, "_default", None)
    monkeypatch.delenv("BARTELS_PCG_SMALL")
    if taken:
        _direction(A, g)
    else:
        with pytest.raises(bg.BartelsError):
            _direction(A, g)
    Context.default().close()
    assert taken == (96 * b * b / (18 * a) < 3.4e38)
