"""The factored plain step's own exponentials over the whole range of Vmem:
steps from voltages of every magnitude (1e-12 V to 0.3 V, both signs, equal
neighbours, zero) against the NumPy oracle, whose expm1 and exp are the C
library's, at the tolerance of the other FP64 tests: 1e-10 of each ion's
largest concentration."""
import numpy as np
import pytest

import golden_io as gi
import oracle
import synthetic

pytestmark = pytest.mark.gpu

N = 2


@pytest.mark.parametrize('name', [None, 'noecm_r50_s9_vgj'])
@pytest.mark.parametrize('scale', [1e-12, 1e-6, 1e-3, 0.03, 0.1, 0.3])
def test_steps_from_any_voltage(scale, name):
    from betse_gb300.engine import ClusterEngine
    d = gi.load(name) if name else synthetic.ragged_fixture(n_cells=80)
    m2c = np.asarray(d['geom_mem_to_cells'])
    rng = np.random.default_rng(1)
    v = rng.uniform(-scale, scale, m2c.max() + 1)
    v[::7] = v[0]                                   # some neighbours at one voltage
    v[3] = 0.0
    d['init_vm'] = v[m2c]
    g, p, s = gi.geometry(d), gi.params(d), gi.state(d)
    oracle.run(g, p, s, N)
    cg, sp, Dm, st, _ = gi.engine_inputs(d)
    with ClusterEngine(cg, sp, 'fp64') as e:
        e.set_membrane_diffusivity(Dm)
        e.upload(**st)
        e.step(N)
        got = e.download()
    for i in range(len(s.cc_cells)):
        assert np.abs(got['cc_cells'][i] - s.cc_cells[i]).max() <= 1e-10 * np.abs(s.cc_cells[i]).max(), i
    ok, err, bound = gi.vm_err_ok(d, got['vm'], s.vm, s.cc_cells)
    assert ok, (err, bound)
