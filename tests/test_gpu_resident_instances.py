"""The split form's resident kernel on both sides of each change of its instance:
22, 23, 28, 29, 33 tiles a CTA, on chains of cells with two membranes each (so
few junctions that as many tiles fit the shared memory of an SM).

Against the streaming factored kernel with test_gpu_factored.py's tolerances: the
same per-cell arithmetic, the environment summed in another order."""
import numpy as np
import pytest

import golden_io as gi

pytestmark = pytest.mark.gpu


def _chain(C):
    from betse_gb300.cluster import ClusterGeometry
    rng = np.random.default_rng(C)
    M = 2 * C
    nn = np.arange(M) + np.where(np.arange(M) % 2, 1, -1)        # right of c with left of c + 1
    nn[0], nn[-1] = 0, M - 1
    sa = np.repeat(rng.uniform(3e-11, 1.4e-10, C), 2)
    cell_sa = 2 * sa[::2]
    vol = cell_sa * rng.uniform(6e-7, 1.2e-6, C)
    w = rng.uniform(0.5, 1.0, M)
    d = gi.load('noecm_r50_s7')
    shape = tuple(int(x) for x in d['geom_grid_shape'])
    return ClusterGeometry.from_arrays(
        mem_to_cells=np.arange(M) // 2, nn_i=nn, bflags_mems=[0, M - 1], map_mem2ecm=np.zeros(M), mem_sa=sa,
        mem_nx=np.ones(M), mem_ny=np.zeros(M), gj_weight=np.minimum(w, w[nn]), cell_vol=vol, cell_sa=cell_sa,
        diviterm=vol / cell_sa, grid_shape=shape, delta=float(d['geom_delta']), gj_len=float(d['geom_gj_len']))


@pytest.mark.parametrize('tiles', [22, 23, 28, 29, 33])
def test_tiles_of_a_cta(tiles):
    import torch
    from betse_gb300.engine import ClusterEngine
    g = _chain(32 * tiles * torch.cuda.get_device_properties(0).multi_processor_count - 5)
    _, p, _, st0, _ = gi.engine_inputs(gi.load('noecm_r50_s7'))
    rng = np.random.default_rng(1)
    Dm = 10.0 ** rng.uniform(-19, -17, (p.n_ions, g.n_mems))
    cc = np.repeat(st0['cc_cells'][:, :1], g.n_cells, axis=1)
    rho = (p.zs * p.F) @ cc
    m2c = np.asarray(g.mem_to_cells)
    env = np.asarray(st0['cc_env']).reshape(p.n_ions, -1)[:, 0]
    res = {}
    for kernel in ('factored', 'resident'):
        with ClusterEngine(g, p, 'split') as e:
            e.set_membrane_diffusivity(Dm)
            e.upload(((1.0 / p.cm) * (rho * g.diviterm))[m2c], cc, cc[:, m2c].copy(), env)
            e.set_launch_config(256, kernel)
            if kernel == 'resident':
                info = e.resident_info()
                assert info['fits'] and info['threads'] == 32 * min(tiles, 32), info
            e.step(30)
            e.check_stable()
            res[kernel] = e.download()
    for k in ('cc_cells', 'cc_env'):
        assert gi.rel_err(res['resident'][k], res['factored'][k]) < 1e-9, k
    assert gi.rel_err(res['resident']['cc_at_mem'], res['factored']['cc_at_mem']) < 2.5e-7
    assert np.max(np.abs(res['resident']['vm'] - res['factored']['vm'])) < 2e-8
