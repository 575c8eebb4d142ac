"""The factored plain FP64 step with extracellular spaces (k_plain_step's ECM
form): cells of 1 to 20 membranes over tile edges, junctions that are not
mutual, a fast pump, voltage-gated junctions, a trivalent ion, grid cells
without potassium or without sodium (the pump's quotient vanishes), and an
electric field with smoothing and without.

Against k_cell_step, which a step that is asked for its outputs runs and which
matches the NumPy oracle elsewhere, at the tolerances of the other FP64 tests:
1e-10 relative, Vmem plus the cancellation floor of the charge sum.  Every tile
size must give the same bits: each cell, membrane and grid value is formed by
the same operations in the same order."""
import numpy as np
import pytest

import golden_io as gi
import synthetic
from test_gpu_plain_factored import _odd_charge, _odd_junctions

pytestmark = pytest.mark.gpu

N = 12


def _fixture(template, cells):
    """Ragged cells on a golden fixture's grid."""
    t = gi.load(template)
    d = synthetic.ragged_fixture(seed=cells, n_cells=cells, template=template)
    d['init_cc_env'] = t['init_cc_env'].copy()
    for k in t:
        if k.startswith('init_') and k not in d:
            d[k] = t[k]
    for k in t:
        if k.startswith('geom_') and k not in d:
            d[k] = t[k]
    return d


def _bare_spots(d):
    """No K in some grid cells, no Na in others, neither in a few."""
    names = [str(x) for x in d['par_ion_names']]
    env = d['init_cc_env'].copy()
    sites = np.unique(d['geom_map_mem2ecm'])
    env[names.index('K'), sites[0:20]] = 0.0
    env[names.index('Na'), sites[15:30]] = 0.0
    d['init_cc_env'] = env
    return d


def _engine(d, **params):
    from betse_gb300.engine import ClusterEngine
    cg, sp, Dm, st, D_env = gi.engine_inputs(d)
    eng = ClusterEngine(cg, sp.replace(**params), 'fp64')
    eng.set_membrane_diffusivity(Dm)
    eng.set_env_diffusivity(D_env)
    eng.upload(**st)
    return eng


def _check(d, n=N, **params):
    with _engine(d, **params) as e:
        for _ in range(n):
            e.step(1, outputs=True)
        ref = e.download()
    assert all(np.isfinite(v).all() for v in ref.values())
    first = None
    for tpb in (None, 32, 64, 128, 256):
        with _engine(d, **params) as e:
            if tpb:
                e.set_launch_config(tpb, 0)
            e.step(n)
            got = e.download()
        first = first or got
        for k in ref:
            assert np.array_equal(got[k], first[k]), (tpb, k)
    ok, err, bound = gi.vm_err_ok(d, first['vm'], ref['vm'], ref['cc_cells'])
    assert ok, (err, bound)
    for k in ('cc_cells', 'cc_at_mem', 'cc_env', 'gjopen'):
        if k in ref:
            assert gi.rel_err(first[k], ref[k]) < 1e-10, k


@pytest.mark.parametrize('template', ['ecm_r50_s3', 'ecm_r40_s5_sharp'])
@pytest.mark.parametrize('cells', [6, 63, 65, 129])
def test_tile_edges(template, cells):
    _check(_fixture(template, cells))


@pytest.mark.parametrize('change', [_odd_junctions, _odd_charge, _bare_spots])
def test_odd_junctions_charges_and_bare_grid_cells(change):
    _check(change(_fixture('ecm_r50_s3', 80)))


def test_gated_junctions():
    _check(_odd_junctions(_fixture('ecm_r50_s3', 90)), v_sensitive_gj=True, gj_vthresh=15.0, gj_min=0.1)


def test_vmem_that_differs_within_a_cell():
    d = _fixture('ecm_r50_s3', 70)
    d['init_vm'] = d['init_vm'] + np.random.default_rng(2).uniform(-5e-3, 5e-3, len(d['init_vm']))
    for n in (1, 2, 45):
        _check(d, n)
