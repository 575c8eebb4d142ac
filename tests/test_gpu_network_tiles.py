"""The network kernels where their tiles can go wrong: cells of 1 to 20
membranes, 6 cells, one short of a tile, a whole tile, one more, two and a bit;
a Vmem that differs from membrane to membrane (the flux is then formed per
membrane, not per cell) and one that does not; and sixteen substances on cells
of some 25 membranes, where a tile has fewer than 32 cells.

The network alone on a frozen Vmem against the NumPy oracle, at the tolerance
of test_gpu_network.py: 1e-10 relative."""
import copy

import numpy as np
import pytest

import golden_io as gi
import synthetic
from oracle.network import Network as OracleNetwork
from test_oracle_network import network_inputs

pytestmark = pytest.mark.gpu

RTOL = 1e-10
N = 20


def _merge(d, k):
    """Every k neighbouring cells made one."""
    C = len(d['geom_num_mems']) // k
    cells = C * k
    M = int(d['geom_num_mems'][:cells].sum())
    keep = lambda a: np.asarray(a)[..., :M]          # noqa: E731
    nn = d['geom_nn_i'][:M].copy()
    own = nn >= M
    nn[own] = np.nonzero(own)[0]
    d['geom_nn_i'] = nn
    d['geom_bflags_mems'] = np.nonzero(nn == np.arange(M))[0].astype(np.int64)
    d['geom_mem_to_cells'] = d['geom_mem_to_cells'][:M] // k
    for n in ('mem_sa', 'R_rads', 'map_mem2ecm', 'gj_default_weights'):
        d['geom_' + n] = keep(d['geom_' + n])
    d['geom_mem_vects_flat'] = d['geom_mem_vects_flat'][:M]
    for n in ('par_smooth_weight_mem', 'par_smooth_weight_o', 'par_Dm_cells', 'init_cc_at_mem', 'init_cc_env',
              'init_vm'):
        d[n] = keep(d[n])
    for n in ('num_mems', 'cell_vol', 'cell_sa'):
        d['geom_' + n] = d['geom_' + n][:cells].reshape(C, k).sum(1)
    d['geom_diviterm'] = d['geom_cell_vol'] / d['geom_cell_sa']
    d['init_cc_cells'] = d['init_cc_cells'][:, :C]
    return d


def _check(d, per_membrane, copies=1):
    from betse_gb300.engine import ClusterEngine
    from betse_gb300.network import Network, NetworkSpec
    cfg, _, _, _ = network_inputs(gi.load('net_r50_s21'))
    subs = list(cfg['substances'])
    for k in range(1, copies):
        for s in cfg['substances']:
            s = copy.deepcopy(s)
            s['name'] = f"{s['name']}_{k}"
            subs.append(s)
    subs = subs[:16]
    rng = np.random.default_rng(3)
    if per_membrane:
        d['init_vm'] = d['init_vm'] + rng.uniform(-5e-3, 5e-3, len(d['init_vm']))
    g, p, s = gi.geometry(d), gi.params(d), gi.state(d)
    C, m2c = len(g.cell_vol), np.asarray(g.mem_to_cells)
    spot = np.sort(rng.choice(C, size=max(1, C // 3), replace=False))
    gmod = rng.uniform(0.2, 1.2, size=C)
    spots = {s['name']: spot for s in subs if s['name'][0] == 'B'}
    gmods = {s['name']: gmod for s in subs if s['name'][0] == 'A'}
    mem_vol = 0.5 * np.asarray(g.R_rads) * np.asarray(g.mem_sa)
    onet = OracleNetwork(subs, cfg['reactions'], g, p, mem_vol, cfg['time_dilation'], spots, gmods)
    st = onet.initial_state()
    st.c_cells *= rng.uniform(0.8, 1.2, st.c_cells.shape)
    st.cc_at_mem = st.c_cells[:, m2c] * rng.uniform(0.95, 1.05, (len(subs), len(m2c)))
    c0 = st.c_cells.copy(), st.cc_at_mem.copy(), st.c_env.copy()
    vm = s.vm
    for _ in range(N):
        onet.step(st, vm, vm[g.nn_i] - vm, p.gj_block * g.gj_weight, p.gj_block)
    assert st.unstable == 0
    cg, sp, Dm, state, _ = gi.engine_inputs(d)
    with ClusterEngine(cg, sp, 'fp64') as eng:
        eng.set_membrane_diffusivity(Dm)
        eng.upload(**state)
        spec = NetworkSpec.from_config(subs, cfg['reactions'], cfg['time_dilation'], n_cells=C,
                                       profiles={'spot': spot}, growth_mod=gmods,
                                       ion_names=[str(x) for x in d['par_ion_names']], mem_vol=mem_vol,
                                       R_rads=g.R_rads)
        with Network(eng, spec) as net:
            net.upload(*c0)
            net.step(N, with_ions=False)
            net.check_stable()
            got = net.download()
    for k in ('c_cells', 'cc_at_mem'):
        ref = getattr(st, k)
        assert np.max(np.abs(got[k] - ref)) < RTOL * np.max(np.abs(ref)), k
    np.testing.assert_allclose(got['c_env'], st.c_env, rtol=RTOL, atol=0)


@pytest.mark.parametrize('per_membrane', [False, True])
@pytest.mark.parametrize('cells', [6, 31, 32, 33, 70])
def test_tile_edges(cells, per_membrane):
    _check(synthetic.ragged_fixture(seed=cells, n_cells=cells), per_membrane)


def test_sixteen_substances_on_cells_of_many_membranes():
    _check(_merge(synthetic.ragged_fixture(seed=5, n_cells=300), 6), True, copies=5)
