"""The tensor-core product at every width of its output tiles (16 to 128
columns, chosen from the sizes): one column short of a tile, a whole one and
one more, one and several packed 128-column tiles, rows short of 128.

Against FP64 at the tolerance of test_gpu_dense_op.py (1e-4 of the largest),
and a column must be the same bits whichever block of columns it is part of:
the widths differ only in which columns a CTA holds."""
import numpy as np
import pytest

import golden_io as gi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('n,counts', [(65, (1, 15, 16, 17, 33, 129)), (700, (1, 31, 32, 64, 96, 130, 257)),
                                      (3001, (1, 16, 96, 100, 250))])
def test_a_column_does_not_depend_on_its_block(n, counts):
    from betse_gb300.dense import DenseOperator
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n))
    X = rng.standard_normal((n, max(counts)))
    with DenseOperator(A) as op:
        Y = [op.apply(np.ascontiguousarray(X[:, :k])) for k in counts]
    ref = A @ X
    for k, y in zip(counts, Y):
        assert gi.rel_err(y, ref[:, :k]) < 1e-4, k
        assert np.array_equal(y, Y[-1][:, :k]), k
