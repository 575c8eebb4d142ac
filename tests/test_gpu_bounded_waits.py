"""Failure detection without a fault: the grid barriers of the resident plain step
and of the graph solver start from a count that they cannot reach, so that every
CTA's bounded wait runs out; the timeout is reported, nothing is written back, and
the handle goes on as if nothing had happened."""
import numpy as np
import pytest

import golden_io as gi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('name', ['noecm_r80_s1', 'noecm_r20_s2'])
def test_resident_plain_step(name):
    from betse_gb300.engine import ClusterEngine
    cg, sp, Dm, st, _ = gi.engine_inputs(gi.load(name))
    got = []
    for check in (True, False):
        with ClusterEngine(cg, sp, 'fp64') as e:
            e.set_membrane_diffusivity(Dm)
            e.upload(**st)
            for n in (11, 12):
                e.step(n)
                if check:
                    before = e.download()
                    assert e.resident_barrier_check(0.05) is True
                    after = e.download()
                    for k in before:
                        assert np.array_equal(before[k], after[k]), k
            e.check_stable()
            got.append(e.download())
    for k in got[1]:
        assert np.array_equal(got[0][k], got[1][k]), k


def test_gated_plain_step_has_no_check():
    from betse_gb300._lib import BxLibraryError
    from betse_gb300.engine import ClusterEngine
    cg, sp, Dm, st, _ = gi.engine_inputs(gi.load('noecm_r50_s9_vgj'))
    with ClusterEngine(cg, sp, 'fp64') as e:
        e.set_membrane_diffusivity(Dm)
        e.upload(**st)
        with pytest.raises(BxLibraryError):
            e.resident_barrier_check(0.05)


@pytest.mark.parametrize('n', [200, 3000])
def test_graph_solver(n):
    from betse_gb300.dense import LapGJ
    from test_gpu_graph_solver import _grid
    X = np.random.default_rng(n).standard_normal((n, 3))
    with LapGJ(*_grid(n), max_rhs=3) as op:
        ref = op.apply(X)
        assert op.barrier_check() is True
        assert np.array_equal(op.apply(X), ref)
