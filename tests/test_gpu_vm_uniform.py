"""A Vmem that differs within a cell while the handle could take it for one
value per cell, which the factored plain step reads: a state uploaded under a
boundary potential that makes vm + Phi_b uniform, or steps replayed from a
captured graph under a potential, and the potential then cleared.

Against the NumPy oracle, which keeps Vmem per membrane, at 1e-10 relative
(Vmem plus the cancellation floor of the charge sum)."""
import numpy as np
import pytest

import golden_io as gi
import oracle

pytestmark = pytest.mark.gpu

N = 3


def _check(d, got, s):
    ok, err, bound = gi.vm_err_ok(d, got['vm'], s.vm, s.cc_cells)
    assert ok, (err, bound)
    for k in ('cc_cells', 'cc_at_mem'):
        assert gi.rel_err(got[k], getattr(s, k)) < 1e-10, k


@pytest.mark.parametrize('name', ['noecm_r50_s7', 'ecm_r50_s3'])
def test_state_uploaded_under_a_potential_that_is_cleared(name):
    from betse_gb300.engine import ClusterEngine
    d = gi.load(name)
    g, p, s = gi.geometry(d), gi.params(d), gi.state(d)
    G = int(np.prod(g.grid_shape))
    m2c = np.asarray(g.mem_to_cells)
    phib = np.random.default_rng(1).integers(-8, 9, G) / 1024.0       # sums below are exact
    cell = np.random.default_rng(2).integers(-64, -32, m2c.max() + 1) / 1024.0
    s.vm = cell[m2c] - phib[g.map_mem2ecm]
    cg, sp, Dm, st, D_env = gi.engine_inputs(d)
    st = dict(st, vm=s.vm.copy())
    if p.is_ecm:
        st.update(E_env_x=s.E_env_x.copy(), E_env_y=s.E_env_y.copy())
    with ClusterEngine(cg, sp, 'fp64') as e:
        e.set_membrane_diffusivity(Dm)
        if p.is_ecm:
            e.set_env_diffusivity(D_env)
        e.set_boundary_potential(phib)
        e.upload(**st)
        e.set_boundary_potential(None)
        e.step(N)
        got = e.download()
    oracle.run(g, p, s, N)
    _check(d, got, s)


def test_graph_steps_under_a_potential_that_is_cleared():
    """64 captured steps with the potential on from a Vmem that is one value per
    cell, after a call that captured them."""
    from betse_gb300.engine import ClusterEngine
    d = gi.load('noecm_r50_s7')
    g, p, s = gi.geometry(d), gi.params(d), gi.state(d)
    ny, nx = (int(x) for x in g.grid_shape)
    yy, xx = np.mgrid[0:ny, 0:nx]
    phib = (3e-3 * np.sin(np.pi * xx / (nx - 1)) * np.cos(np.pi * yy / (ny - 1))).ravel()
    cg, sp, Dm, st, _ = gi.engine_inputs(d)
    with ClusterEngine(cg, sp, 'fp64') as e:
        e.set_membrane_diffusivity(Dm)
        e.set_boundary_potential(phib)
        for _ in range(2):
            e.upload(**st)
            e.step(64)
        e.set_boundary_potential(None)
        e.step(N)
        got = e.download()
    s.Phi_b = phib
    oracle.run(g, p, s, 64)
    s.Phi_b = np.zeros_like(phib)
    oracle.run(g, p, s, N)
    _check(d, got, s)
