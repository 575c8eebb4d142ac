"""Networks stepped with the ions where Vmem is not one value per cell: cell
polarizability, a boundary potential, an uploaded Vmem that differs within a
cell; two calls in a row of more than 32 steps each, so that captured steps
follow steps of their own from either parity of the state's two buffers.

Against as many single steps bit for bit (the same kernels in the same order),
and against the NumPy oracle at the tolerance of test_gpu_network.py: 1e-10
relative (Vmem plus the cancellation floor of the charge sum)."""
import numpy as np
import pytest

import golden_io as gi
from oracle.network import Network as OracleNetwork, NetworkState, run_with_ions
from test_oracle_network import network_inputs

pytestmark = pytest.mark.gpu

RTOL = 1e-10


def _case(kind):
    """(fixture, boundary potential or None)"""
    d = gi.load('net_r50_s21')
    phib = None
    if kind == 'uneven':
        d['init_vm'] = d['init_vm'] + np.random.default_rng(2).uniform(-5e-3, 5e-3, len(d['init_vm']))
    elif kind == 'polar':
        d['par_cell_polarizability'] = np.float64(1e-4)
    elif kind == 'phib':
        ny, nx = (int(x) for x in d['geom_grid_shape'])
        yy, xx = np.mgrid[0:ny, 0:nx]
        phib = (3e-3 * np.sin(np.pi * xx / (nx - 1)) * np.cos(np.pi * yy / (ny - 1))).ravel()
    return d, phib


def _gpu(d, phib, calls):
    from betse_gb300.engine import ClusterEngine
    from betse_gb300.network import Network, NetworkSpec
    cfg, names, targets, mods = network_inputs(d)
    cg, sp, Dm, st, _ = gi.engine_inputs(d)
    g = gi.geometry(d)
    spec = NetworkSpec.from_config(cfg['substances'], cfg['reactions'], cfg['time_dilation'], n_cells=len(g.cell_vol),
                                   profiles={'spot': targets['B']}, growth_mod=mods,
                                   ion_names=[str(x) for x in d['par_ion_names']], mem_vol=d['net_mem_vol'],
                                   R_rads=g.R_rads)
    with ClusterEngine(cg, sp, 'fp64') as eng, Network(eng, spec) as net:
        eng.set_membrane_diffusivity(Dm)
        if phib is not None:
            eng.set_boundary_potential(phib)
        eng.upload(**st)
        net.upload(d['init_net_c_cells'], d['init_net_cc_at_mem'], d['init_net_c_env'])
        for n in calls:
            net.step(n, with_ions=True)
        net.check_stable()
        eng.check_stable()
        return dict(eng.download(), **{'net_' + k: v for k, v in net.download().items()})


@pytest.mark.parametrize('kind', ['even', 'uneven', 'polar', 'phib'])
@pytest.mark.parametrize('calls', [(33, 45), (50, 45), (1, 32, 40), (1, 34, 64), (2, 100)])
def test_calls_of_many_steps_equal_single_steps(kind, calls):
    d, phib = _case(kind)
    got = _gpu(d, phib, calls)
    ref = _gpu(d, phib, (1,) * sum(calls))
    for k in ref:
        assert np.array_equal(got[k], ref[k]), k


@pytest.mark.parametrize('kind', ['uneven', 'polar', 'phib'])
def test_calls_of_many_steps_match_the_oracle(kind):
    d, phib = _case(kind)
    calls = (50, 45)
    got = _gpu(d, phib, calls)
    g, p, s = gi.geometry(d), gi.params(d), gi.state(d)
    if phib is not None:
        s.Phi_b = phib
    cfg, names, targets, mods = network_inputs(d)
    onet = OracleNetwork(cfg['substances'], cfg['reactions'], g, p, d['net_mem_vol'], cfg['time_dilation'], targets, mods)
    st = NetworkState(d['init_net_c_cells'], d['init_net_cc_at_mem'], d['init_net_c_env'][:, 0])
    run_with_ions(onet, st, g, p, s, sum(calls))
    assert st.unstable == 0
    ok, err, bound = gi.vm_err_ok(d, got['vm'], s.vm, s.cc_cells)
    assert ok, (err, bound)
    assert gi.rel_err(got['cc_cells'], s.cc_cells) < RTOL
    for k in ('c_cells', 'cc_at_mem'):
        assert gi.rel_err(got['net_' + k], getattr(st, k)) < RTOL, k
    np.testing.assert_allclose(got['net_c_env'], st.c_env, rtol=RTOL, atol=0)
