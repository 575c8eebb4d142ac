"""The factored plain step at voltages far outside a cell's range, as a run
that diverges reaches them: up to 17 V of either sign and as much between
neighbours, where expm1 of the reduced voltage reaches 1e276 and is still
finite.  Monovalent ions only: exp(2 F V / (R T)) overflows in the formula
itself from 9.5 V on.  The pump is off: its quotient overflows too, and so do
the gates' rates between neighbours a few volts apart.

One step against the NumPy oracle at the tolerance of the other FP64 tests:
1e-10 of each ion's largest concentration."""
import numpy as np
import pytest

import golden_io as gi
import oracle
import synthetic

pytestmark = pytest.mark.gpu


RANGES = [(-17.0, -8.0), (-8.5, 8.5), (8.0, 17.0), (-9.6, -9.0)]


@pytest.mark.parametrize('name,low,high', [(n, *r) for n in (None, 'ecm_r50_s3') for r in RANGES] +
                         [('noecm_r50_s9_vgj', -9.6, -9.0)])
def test_one_step_from_large_voltages(name, low, high):
    from betse_gb300.engine import ClusterEngine
    d = gi.load(name) if name else synthetic.ragged_fixture(n_cells=80)
    d['par_zs'] = np.where(np.abs(d['par_zs']) == 2.0, np.sign(d['par_zs']), d['par_zs'])
    d['par_alpha_NaK'] = np.float64(0.0)
    m2c = np.asarray(d['geom_mem_to_cells'])
    d['init_vm'] = np.random.default_rng(1).uniform(low, high, m2c.max() + 1)[m2c]
    g, p, s = gi.geometry(d), gi.params(d), gi.state(d)
    cg, sp, Dm, st, D_env = gi.engine_inputs(d)
    before = s.cc_cells.copy()
    oracle.run(g, p, s, 1)
    assert np.isfinite(s.cc_cells).all() and gi.rel_err(s.cc_cells, before) > 1e-6    # the fluxes count
    with ClusterEngine(cg, sp, 'fp64') as e:
        e.set_membrane_diffusivity(Dm)
        if p.is_ecm:
            e.set_env_diffusivity(D_env)
        e.upload(**st)
        e.step(1)
        got = e.download()
    for i in range(len(s.cc_cells)):
        assert np.abs(got['cc_cells'][i] - s.cc_cells[i]).max() <= 1e-10 * np.abs(s.cc_cells[i]).max(), i
