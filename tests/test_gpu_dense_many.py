"""More dense operators alive than one page of error words holds (1024), made and
released from two threads, and words handed on: every operator reports no timeout
and applies its own matrix.

Against NumPy at the operator's accuracy (BF16 pairs: 2^-16 of the terms)."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(op, A, x):
    y = op.apply(x)                                        # raises on a reported timeout
    assert np.max(np.abs(y - A @ x)) <= 2.0 ** -15 * np.max(np.abs(A) @ np.abs(x))


def test_more_operators_than_a_page():
    from betse_gb300.dense import DenseOperator
    rng = np.random.default_rng(4)
    A = [rng.standard_normal((5, 5)) for _ in range(1030)]
    x = rng.standard_normal((5, 3))
    ops = [DenseOperator(a) for a in A]
    for i in (0, 1, 1022, 1023, 1024, 1025, 1029):
        _check(ops[i], A[i], x)
    for i in (3, 1023, 1024, 1027):
        ops[i].close()
        ops[i] = DenseOperator(A[i])
        _check(ops[i], A[i], x)
    bad = []

    def work(k):
        try:
            for i in range(k, 40, 2):
                op = DenseOperator(A[i])
                _check(op, A[i], x)
                op.close()
        except BaseException as e:                         # pragma: no cover - reported below
            bad.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad
    for op in ops:
        op.close()
