"""k_graph_cg where it can go wrong: node counts around the dense level's limit
and not a multiple of an aggregate, block widths around every split of the
columns (lanes, slabs of 32, column groups), several components, a zero
right-hand side, and a solve that runs out of iterations.

Against the dense pseudo-inverse.  Solves run to 1e-13 relative residual; the
error of an iterate is bounded by that times the condition number of L, at
most 2e4 for these grids, so 2e-9 of the largest value."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL, BOUND = 1e-13, 2e-9


def _grid(n, width=23, seed=0, parts=1):
    """A triangulated strip of n nodes (numbered along it), cut into parts."""
    rng = np.random.default_rng(seed)
    e = []
    for i in range(n):
        for j in ([i + 1] if (i + 1) % width else []) + [i + width] + ([i + width + 1] if (i + 1) % width else []):
            if j < n and i * parts // n == j * parts // n:
                e.append((i, j))
    e = np.array(e)
    return e, rng.uniform(0.5, 2.0, len(e)), rng.uniform(0.5, 2.0, len(e)), rng.uniform(0.5, 2.0, n)


def _pinv(e, n, parts=1):
    """(L+, D): with J the projector on the components' constants, L+ =
    (L + J)^-1 - J (numpy's pinv cuts the null space at 1e-15 of the largest
    singular value, which some of these matrices exceed)."""
    D = np.zeros((len(e), n))
    D[np.arange(len(e)), e[:, 0]] = -1.0
    D[np.arange(len(e)), e[:, 1]] = 1.0
    part = np.arange(n) * parts // n
    J = (part[:, None] == part[None, :]) / np.bincount(part)[part]
    return np.linalg.inv(D.T @ D + J) - J, D


@pytest.mark.parametrize('n', [2, 5, 64, 65, 511, 512, 513, 1001])
def test_solve_and_apply_match_the_pseudo_inverse(n):
    from betse_gb300.dense import LapGJ
    e, tri, vor, area = _grid(n)
    Lp, D = _pinv(e, n)
    X = np.random.default_rng(n).standard_normal((n, 9))
    with LapGJ(e, tri, vor, area, max_rhs=9) as op:
        for K in (1, 9):
            ref = Lp @ X[:, :K]
            assert np.max(np.abs(op.solve(X[:, :K], tol=TOL) - ref)) <= BOUND * np.max(np.abs(ref))
        A = -Lp @ (D.T @ np.diag(tri / vor) @ D) @ Lp @ np.diag(area)
        ref = A @ X
        assert np.max(np.abs(op.apply(X, tol=TOL) - ref)) <= BOUND * np.max(np.abs(ref))


@pytest.mark.parametrize('K', [1, 2, 3, 4, 5, 8, 17, 32, 33, 64, 65, 130, 257])
def test_block_widths_match_the_pseudo_inverse(K):
    from betse_gb300.dense import LapGJ
    n = 777
    e, tri, vor, area = _grid(n)
    Lp, _ = _pinv(e, n)
    X = np.random.default_rng(K).standard_normal((n, K))
    X[:, K // 2] = 0.0                                    # a column with nothing to solve
    ref = Lp @ X
    with LapGJ(e, tri, vor, area, max_rhs=K) as op:
        Y = op.solve(X, tol=TOL)
    assert np.max(np.abs(Y - ref)) <= BOUND * max(np.max(np.abs(ref)), 1e-300)
    assert np.all(Y[:, K // 2] == 0.0)


def test_components_are_solved_apart():
    from betse_gb300.dense import LapGJ
    n = 1200
    e, tri, vor, area = _grid(n, parts=3)
    Lp, _ = _pinv(e, n, 3)
    X = np.random.default_rng(4).standard_normal((n, 3))
    for p in range(3):
        X[p * 400:(p + 1) * 400] -= X[p * 400:(p + 1) * 400].mean(0)      # in the range of L
    ref = Lp @ X
    with LapGJ(e, tri, vor, area, max_rhs=3) as op:
        Y = op.solve(X, tol=TOL)
    for p in range(3):                                    # the solver projects on the whole graph's constants only
        s = slice(p * 400, (p + 1) * 400)
        d = Y[s] - ref[s]
        assert np.max(np.abs(d - d.mean(0))) <= BOUND * np.max(np.abs(ref))


def test_running_out_of_iterations_is_reported():
    from betse_gb300.dense import LapGJ
    e, tri, vor, area = _grid(2000)
    X = np.random.default_rng(1).standard_normal((2000, 2))
    with LapGJ(e, tri, vor, area, max_rhs=2) as op:
        with pytest.raises(RuntimeError, match='did not reach'):
            op.solve(X, tol=1e-13, max_iter=5)
        assert op.last_iters == 5 and op.last_rel_res > 1e-13
        op.solve(X, tol=1e-10)                            # the handle is fine
