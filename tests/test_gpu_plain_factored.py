"""The factored plain FP64 step (k_plain_step) where it can go wrong: tile
edges (63, 64, 65, 129 cells and every pinned tile size), cells of 1 to 20
membranes, junctions that are not mutual, partners that are the own cell, a
boundary flag on one side only, zero weights, charges without a fast path, and
a Vmem that differs within a cell (one step of the per-membrane kernel first).

Against the NumPy oracle at the tolerances of the other FP64 tests: 1e-10
relative, Vmem plus the cancellation floor of the charge sum.  The resident
form, the streaming form and every tile size must agree bit for bit: the same
arithmetic per cell and junction, and an environment sum over one tree."""
import numpy as np
import pytest

import golden_io as gi
import oracle
import synthetic

pytestmark = pytest.mark.gpu

N = 12


def _engine(d, **params):
    from betse_gb300.engine import ClusterEngine
    cg, sp, Dm, st, _ = gi.engine_inputs(d)
    eng = ClusterEngine(cg, sp.replace(**params), 'fp64')
    eng.set_membrane_diffusivity(Dm)
    eng.upload(**st)
    return eng


def _odd_junctions(d, seed=5):
    """Junctions no Voronoi cluster has: a partner that points elsewhere, a
    self partner that is not a boundary, a flag on one side, a closed one."""
    rng = np.random.default_rng(seed)
    nn = d['geom_nn_i'].copy()
    M = len(nn)
    pick = rng.choice(M, size=12, replace=False)
    nn[pick[:4]] = rng.integers(0, M, size=4)             # not mutual
    nn[pick[4:6]] = pick[4:6]                             # itself
    d['geom_nn_i'] = nn
    d['geom_bflags_mems'] = np.union1d(d['geom_bflags_mems'], pick[6:9]).astype(np.int64)   # one side only
    w = d['geom_gj_default_weights'].copy()
    w[pick[9:]] = 0.0
    d['geom_gj_default_weights'] = w
    return d


def _odd_charge(d):
    """P as a trivalent anion of a third of the concentration: the same charge."""
    i = [str(x) for x in d['par_ion_names']].index('P')
    z = np.array(d['par_zs'], np.float64)
    z[i] = -3.0
    d['par_zs'] = z
    for k in ('init_cc_cells', 'init_cc_at_mem', 'init_cc_env'):
        a = d[k].copy()
        a[i] /= 3.0
        d[k] = a
    return d


def _check(d, n=N):
    g, p, s = gi.geometry(d), gi.params(d), gi.state(d)
    oracle.run(g, p, s, n)
    with _engine(d) as e:
        e.step(n)
        e.check_stable()
        got = e.download()
    ok, err, bound = gi.vm_err_ok(d, got['vm'], s.vm, s.cc_cells)
    assert ok, (err, bound)
    for k in ('cc_cells', 'cc_at_mem'):
        assert gi.rel_err(got[k], getattr(s, k)) < 1e-10, k
    assert gi.rel_err(got['cc_env'], s.cc_env[:, 0]) < 1e-10


@pytest.mark.parametrize('cells', [6, 63, 64, 65, 129])
def test_tile_edges_match_oracle(cells):
    _check(synthetic.ragged_fixture(seed=cells, n_cells=cells))


@pytest.mark.parametrize('change', [_odd_junctions, _odd_charge, lambda d: _odd_junctions(_odd_charge(d))])
def test_odd_junctions_and_charges_match_oracle(change):
    _check(change(synthetic.ragged_fixture(n_cells=80)))


def test_vmem_that_differs_within_a_cell_matches_oracle():
    d = synthetic.ragged_fixture(n_cells=70)
    d['init_vm'] = d['init_vm'] + np.random.default_rng(2).uniform(-5e-3, 5e-3, len(d['init_vm']))
    for n in (1, 2, N, 45):
        _check(d, n)


@pytest.mark.parametrize('name', ['noecm_r80_s1', 'noecm_r50_s9_vgj', 'noecm_r50_s11_ca'])
def test_resident_streaming_and_tile_sizes_agree_bit_for_bit(name):
    d = gi.load(name)
    with _engine(d) as e:
        for _ in range(40):
            e.step(1)                       # single steps: the streaming form
        ref = e.download()
    for tpb in (None, 32, 64, 128, 256):
        with _engine(d) as e:
            if tpb:
                e.set_launch_config(tpb, 0)
            e.step(40)                      # one cooperative launch where the tiles fit
            got = e.download()
        for k in ref:
            assert np.array_equal(got[k], ref[k]), (tpb, k)


def test_gated_odd_junctions_against_the_per_membrane_kernel():
    """Voltage-gated junctions without symmetry, against k_cell_step, which a
    step that is asked for its outputs runs."""
    d = _odd_junctions(synthetic.ragged_fixture(n_cells=90))
    gate = dict(v_sensitive_gj=True, gj_vthresh=15.0, gj_min=0.1)
    with _engine(d, **gate) as a, _engine(d, **gate) as b:
        a.step(N)
        for _ in range(N):
            b.step(1, outputs=True)
        sa, sb = a.download(), b.download()
    ok, err, bound = gi.vm_err_ok(d, sa['vm'], sb['vm'], sb['cc_cells'])
    assert ok, (err, bound)
    for k in ('cc_cells', 'cc_at_mem', 'cc_env', 'gjopen'):
        assert gi.rel_err(sa[k], sb[k]) < 1e-10, k
