"""How far past the tolerance a solve goes: the error of lapGJinv X follows the
residual at which the iteration stops, so that is held at 0.4 of the tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('K', [1, 9])
@pytest.mark.parametrize('n', [700, 2001])
def test_residual_at_the_stop(n, K):
    from betse_gb300.dense import LapGJ
    from test_gpu_graph_solver import _grid
    e, tri, vor, area = _grid(n)
    X = np.random.default_rng(n).standard_normal((n, K))
    with LapGJ(e, tri, vor, area, max_rhs=K) as op:
        for tol in 10.0 ** -np.arange(4, 13):
            for fn in (op.solve, op.apply):
                fn(X, tol=tol)
                assert op.last_rel_res <= 0.4 * tol, (fn.__name__, tol)
