"""The work that is measured: what a user of this package has it do.

Each case is one pass through the public entry points, over the sizes that the
tests, the benchmark and the drop-in loop use:

  plain    the FP64 step (the drop-in's default form and launch), one interval
           between two of BETSE's sampled steps: state in, 100 steps, state out
  ecm      the same with extracellular spaces, FP64 or split form
  split    the FP32/FP64-split step on the resident kernel (what the autotuner
           picks for one large cluster)
  sweep    a batch of uneven clusters on the factored kernel (what the
           autotuner picks for a parameter sweep)
  sampled  one sampled step: a step with outputs, the outputs, the environment
           fields and the state, as the drop-in mirrors them
  network  a gene network stepping with the ions
  lapgj    cells.lapGJinv applied to right-hand sides (physics/pressures.py:59)
  dense    the tensor-core product with a dense inverse Laplacian
  train    one training step of the warm-start network

States are a fresh init phase (uniform concentrations) or a resumed run
(every cell its own concentrations and Vmem).
"""
import copy
import functools
import math

import numpy as np
import torch

from betse_gb300 import generator as gen
from betse_gb300 import torch_ops as tops
from betse_gb300.dense import DenseOperator, LapGJ, lap_gj_inputs
from betse_gb300.engine import BatchEngine, ClusterEngine
from betse_gb300.gnn import GraphNet, init_params
from betse_gb300.network import Network, NetworkSpec

NONCE = 1e-25
DM_P = gen.ION_NAMES.index('P')
I_NA, I_K, I_CA, I_M = (gen.ION_NAMES.index(n) for n in ('Na', 'K', 'Ca', 'M'))
N_IN, N_OUT, LR = 10, 6, 1e-3          # the warm-start network's features, targets, learning rate


def listed():
    return [
        # BETSE's own cluster size and form: the smallest call, where launches and latency count
        dict(name='plain_240', kind='plain', cells=240, steps=100, gated=False, resumed=False),
        # BETSE's default options (voltage-gated gap junctions, Ca-ATPase), a resumed run of a few thousand cells
        dict(name='plain_gated_3k', kind='plain', cells=3000, steps=100, gated=True, resumed=True),
        # the largest cluster of the benchmark in the plain form
        dict(name='plain_100k', kind='plain', cells=95800, steps=100, gated=False, resumed=True),
        # extracellular spaces on the benchmark's 20k-cell cluster, in both forms
        dict(name='ecm_fp64_20k', kind='ecm', form='fp64', cells=19900, grid=200, steps=100),
        dict(name='ecm_split_20k', kind='ecm', form='split', cells=19900, grid=200, steps=100),
        # the headline form on the largest cluster
        dict(name='split_100k', kind='split', cells=95800, steps=400, resumed=False),
        # a parameter sweep: uneven clusters with their own pump and Na/K diffusivities
        dict(name='sweep_64', kind='sweep', clusters=64, steps=400),
        # a sampled step of a cluster of a few thousand cells on a 50 x 50 environment grid
        dict(name='sampled_5k', kind='sampled', cells=5000, grid=51),
        # a gene network with the ions
        dict(name='network_20k', kind='network', cells=19900, steps=50),
        # the pressure solve of one time step: one right-hand side
        dict(name='lapgj_100k', kind='lapgj', cells=95800, rhs=1),
        # an operator of BETSE's own size range applied to a block of right-hand sides
        dict(name='dense_3k', kind='dense', n=3001, rhs=96),
        # a training batch of the warm start: some thirty clusters' worth of cells
        dict(name='train_30k', kind='train', nodes=30000),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(['plain', 'plain', 'plain', 'ecm', 'split', 'sweep', 'sampled', 'network', 'lapgj', 'dense',
                       'train'])
    if kind == 'plain':
        return dict(kind=kind, cells=log_int(200, 95000), steps=rng.randint(60, 100), gated=rng.random() < 0.4,
                    resumed=rng.random() < 0.5)
    if kind == 'ecm':
        cells = log_int(400, 19000)
        grid = int(min(199, max(24, math.sqrt(2 * cells)))) + rng.randint(0, 1)
        return dict(kind=kind, form=rng.choice(['fp64', 'split']), cells=cells, grid=grid, steps=rng.randint(60, 100))
    if kind == 'split':
        return dict(kind=kind, cells=log_int(2000, 95000), steps=rng.randint(200, 400), resumed=rng.random() < 0.5)
    if kind == 'sweep':
        return dict(kind=kind, clusters=rng.randint(8, 64), steps=rng.randint(200, 400))
    if kind == 'sampled':
        return dict(kind=kind, cells=log_int(500, 5000), grid=rng.randint(25, 51))
    if kind == 'network':
        return dict(kind=kind, cells=log_int(300, 19000), steps=rng.randint(30, 50))
    if kind == 'lapgj':
        cells = log_int(500, 95000)
        return dict(kind=kind, cells=cells, rhs=rng.choice([1, 2, 3, 7]) if cells > 10000 else rng.randint(1, 20))
    if kind == 'dense':
        return dict(kind=kind, n=rng.randint(300, 3500), rhs=log_int(2, 250))
    return dict(kind=kind, nodes=log_int(1500, 30000))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=24)
def _lattice(cells, grid, lattice_seed):
    radius = math.sqrt(cells / 0.0456) * 1e-6          # cells ~ 0.0456 (R / 1 um)^2 for this lattice
    return radius, gen.make_cluster(radius, lattice_seed, grid_size=grid)


def _workload(case, seed, **kw):
    """Geometry, parameters, Dm and initial state of one cluster: the
    generator's seeded workload on one lattice a size, its diffusivities and
    junction weights from the seed; a resumed state on request."""
    ecm = case['kind'] == 'ecm'
    radius, gc = _lattice(case['cells'], case.get('grid', 20), 3)
    gc = copy.copy(gc)
    gc.geom = copy.copy(gc.geom)
    gc.geom.extra = {}
    g, p, Dm, st, D_env = gen.workload(radius, seed, is_ecm=ecm, dt=5e-3 if ecm else 1e-2, cluster=gc, **kw)
    if case.get('gated'):
        p = p.replace(v_sensitive_gj=True, iCa=I_CA, alpha_Ca=5e-8)
    if case.get('resumed'):
        _resume(g, p, st, np.random.default_rng(seed + 77))
    return g, p, Dm, st, D_env


def _resume(g, p, st, rng):
    """Every cell its own concentrations, charged to its own Vmem (M balances)."""
    cc = st['cc_cells']
    for i in range(len(cc)):
        if i not in (I_M, DM_P):
            cc[i] *= rng.uniform(0.9, 1.1, cc.shape[1])
    v = rng.uniform(-0.06, 0.01, cc.shape[1])
    q = np.dot(p.zs, cc) - p.zs[I_M] * cc[I_M]
    cc[I_M] = (v * p.cm / (p.F * g.diviterm) - q) / p.zs[I_M]
    rho = np.dot(p.zs * p.F, cc)
    m2c = np.asarray(g.mem_to_cells)
    st['vm'] = (1 / p.cm) * (rho * g.diviterm)[m2c]
    st['cc_at_mem'] = cc[:, m2c].copy()


@functools.lru_cache(maxsize=4)
def _sweep_sizes(clusters):
    """Cell counts log-uniform in [200, 5000] (sixteen lattices, reused)."""
    rng = np.random.default_rng(7)
    pool = np.exp(rng.uniform(np.log(200), np.log(5000), 16)).astype(int)
    return [int(pool[k % 16]) for k in range(clusters)]


def _sweep(case, seed):
    rng = np.random.default_rng(seed)
    out = ([], [], [], [])
    for k, cells in enumerate(_sweep_sizes(case['clusters'])):
        dm, pump = np.exp(rng.uniform(np.log(0.1), np.log(3.0), 2))
        w = _workload(dict(kind='sweep', cells=cells), seed * 100 + k, na_k_dm_mult=float(dm), pump_mult=float(pump))
        for lst, v in zip(out, w):
            lst.append(v)
    return out


def _pinned(a):
    """A page-locked copy of a float64 array, as a NumPy view."""
    t = torch.empty(np.shape(a), dtype=torch.float64, pin_memory=True)
    t.numpy()[...] = a
    return t.numpy()


def _gpu(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device='cuda')


SPOT_DIV, KEQ_DG = 3, -5000.0


def _network_config(g, seed):
    """Four substances in BETSE's configuration form: Hill activation and
    inhibition, growth modulation and targets, a charged substance crossing
    membranes and junctions, one with intracellular transport, two reactions."""
    def sub(name, z, Dm, Dgj, env, cell, prod, decay, acts=None, inhs=None, ui=False, imp=False, where='all',
            mod='None'):
        a, i = acts or ([], [], []), inhs or ([], [], [])
        gad = {'production rate': prod, 'decay rate': decay, 'apply to': where, 'modulator function': mod,
               'activators': a[0] or 'None', 'Km activators': a[1] or 'None', 'n activators': a[2] or 'None',
               'inhibitors': i[0] or 'None', 'Km inhibitors': i[1] or 'None', 'n inhibitors': i[2] or 'None'}
        return {'name': name, 'Dm': Dm, 'Do': 1.0e-11, 'Dgj': Dgj, 'z': z, 'env conc': env, 'cell conc': cell,
                'update intracellular': ui, 'use time dilation': False, 'TJ permeable': False, 'GJ impermeable': imp,
                'TJ factor': 1.0, 'growth and decay': gad, 'plotting': {'plot 2D': False, 'animate': False}}

    subs = [sub('g1', 0, 0.0, 1e-15, 0.0, 0.1, 0.5, 0.2, inhs=(['g3'], [0.3], [2.0]), mod='gradient_x'),
            sub('g2', 0, 0.0, 1e-15, 0.0, 0.05, 1.0, 0.5, acts=(['g1', 'g3!'], [0.2, 0.5], [2.0, 1.0]), imp=True,
                where=['spot']),
            sub('g3', -1, 1e-18, 1e-14, 0.5, 0.2, 0.2, 0.1, acts=(['g2'], [0.1], [1.0])),
            sub('g4', 0, 5e-19, 1e-15, 1.0, 0.1, 0.05, 0.05, inhs=(['g3'], [0.4], [1.0]), ui=True)]
    react = [{'name': 'r1', 'reaction zone': 'cell', 'reactants': ['g1', 'g3'], 'reactant multipliers': [1, 1],
              'Km reactants': [0.1, 0.2], 'products': ['g4'], 'product multipliers': [1], 'Km products': [0.5],
              'max rate': 0.01, 'standard free energy': 'None', 'reaction activators': ['g2'], 'activator Km': [0.1],
              'activator n': [2.0]},
             {'name': 'r2', 'reaction zone': 'cell', 'reactants': ['g4'], 'reactant multipliers': [1],
              'Km reactants': [0.3], 'products': ['g2'], 'product multipliers': [2], 'Km products': [0.4],
              'max rate': 0.02, 'standard free energy': KEQ_DG}]
    rng = np.random.default_rng(seed + 5)
    C = g.n_cells
    spot = np.sort(rng.choice(C, size=C // SPOT_DIV, replace=False))
    gmod = rng.uniform(0.2, 1.2, size=C)
    c0 = np.array([[0.1], [0.05], [0.2], [0.1]]) * rng.uniform(0.8, 1.2, (4, C))
    return subs, react, spot, gmod, c0, np.array([0.0, 0.0, 0.5, 1.0])


def _train_inputs(case, seed):
    _, gc = _lattice(case['nodes'], 20, 3)
    ptr, nbr = np.asarray(gc.geom.cell_nn_ptr), np.asarray(gc.geom.cell_nn)
    t = torch.Generator('cuda').manual_seed(seed)
    x = torch.randn(len(ptr) - 1, N_IN, device='cuda', generator=t)
    mix = torch.randn(N_IN, N_OUT, device='cuda', generator=t) / math.sqrt(N_IN)
    return ptr, nbr, x, torch.tanh(x @ mix).contiguous(), init_params(N_IN, N_OUT, seed)


def prepare(case, seed):
    kind = case['kind']
    s = {'case': case}
    if kind in ('plain', 'split') and not case.get('gated'):
        # the state in CUDA tensors, stepped through the PyTorch operators
        g, p, Dm, st, _ = _workload(case, seed)
        s['h'] = _Handle(tops.create(g, p, 'fp64' if kind == 'plain' else 'split'), g, p)
        torch.ops.bx.set_membrane_diffusivity(s['h'].h, torch.as_tensor(Dm))
        s['state'] = [_gpu(st[k]) for k in ('vm', 'cc_cells', 'cc_at_mem', 'cc_env')]
        if kind == 'split':
            s['h'].pin_resident()
    elif kind in ('plain', 'ecm'):
        # BETSE's arrays on the host, as the drop-in loop holds them
        g, p, Dm, st, D_env = _workload(case, seed)
        e = s['eng'] = ClusterEngine(g, p, case.get('form', 'fp64'))
        e.set_membrane_diffusivity(Dm)
        if kind == 'ecm':
            e.set_env_diffusivity(D_env)
        s['state'] = {k: _pinned(v) for k, v in st.items()}
        e.upload(**s['state'])
        s['out'] = {k: _pinned(v) for k, v in e.download().items()}
    elif kind == 'sweep':
        gs, ps, Dms, sts = _sweep(case, seed)
        e = s['eng'] = BatchEngine(gs, ps, 'split')
        e.set_membrane_diffusivity(Dms)
        e.set_launch_config(256, 'factored', 12)
        cat = {k: np.concatenate([x[k] for x in sts], axis=a)
               for k, a in (('vm', 0), ('cc_cells', 1), ('cc_at_mem', 1))}
        cat['cc_env'] = np.stack([x['cc_env'] for x in sts])
        s['state'] = {k: _pinned(v) for k, v in cat.items()}
        s['out'] = {k: _pinned(v) for k, v in cat.items()}
    elif kind == 'sampled':
        g, p, Dm, st, _ = _workload(dict(case, resumed=True), seed)
        s['h'] = _Handle(tops.create(g, p, 'fp64'), g, p)
        torch.ops.bx.set_membrane_diffusivity(s['h'].h, torch.as_tensor(Dm))
        torch.ops.bx.set_lap_env_inv(s['h'].h, torch.linalg.inv(_laplacian(g)).cpu())
        s['state'] = [_gpu(st[k]) for k in ('vm', 'cc_cells', 'cc_at_mem', 'cc_env')]
        s['weight'] = _gpu(g.D_env_weight)
    elif kind == 'network':
        g, p, Dm, st, _ = _workload(case, seed)
        subs, react, spot, gmod, c0, env0 = _network_config(g, seed)
        e = s['eng'] = ClusterEngine(g, p, 'fp64')
        e.set_membrane_diffusivity(Dm)
        s['state'] = {k: _pinned(v) for k, v in st.items()}
        s['out'] = {k: _pinned(v) for k, v in st.items()}
        R = np.asarray(g.R_rads)
        spec = NetworkSpec.from_config(subs, react, 1.0, n_cells=g.n_cells, profiles={'spot': spot},
                                       growth_mod={'g1': gmod}, ion_names=p.ion_names,
                                       mem_vol=0.5 * R * np.asarray(g.mem_sa), R_rads=R)
        s['net'] = Network(e, spec)
        s['sub'] = (c0, c0[:, np.asarray(g.mem_to_cells)].copy(), env0)
    elif kind == 'lapgj':
        g, inputs, X = _lapgj_inputs(case, seed)
        s['op'], s['X'] = LapGJ(*inputs, max_rhs=max(1, case['rhs'])), X
    elif kind == 'dense':
        A, X = _dense_inputs(case, seed)
        s['op'], s['X'] = DenseOperator(A.cpu().numpy()), X
    else:
        ptr, nbr, x, y, w = _train_inputs(case, seed)
        net = s['net'] = GraphNet(w)
        net.set_graph(ptr, nbr)
        s['x'], s['y'] = x, y
    return s


class _Handle:
    """A cluster handle of the PyTorch operators, released with its owner."""

    def __init__(self, h, g, p):
        self.h, self.geom, self.params = h, g, p

    def pin_resident(self):
        """The resident kernel, which the autotuner picks for one large cluster."""
        from betse_gb300 import _lib
        from betse_gb300.engine import KERNELS
        _lib.check(_lib.load().bx_set_launch_config(self.h, 256, KERNELS['resident']), 'bx_set_launch_config')

    def __del__(self):
        try:
            tops.release(self.h)
        except Exception:
            pass


def _lapgj_inputs(case, seed):
    _, gc = _lattice(case['cells'], 20, 3)
    t = torch.Generator('cuda').manual_seed(seed)
    X = torch.randn(gc.geom.n_cells, case['rhs'], dtype=torch.float64, device='cuda', generator=t)
    return gc.geom, lap_gj_inputs(gc.geom, gc.cell_centres), X


def _dense_inputs(case, seed):
    """An operator with the decay of an inverse Laplacian along the Z curve."""
    n = case['n']
    t = torch.Generator('cuda').manual_seed(seed)
    k = torch.arange(n, dtype=torch.float64, device='cuda')
    A = -1.0 / (1.0 + (k[:, None] - k[None, :]).abs().sqrt())
    A *= 1.0 + 0.2 * torch.rand(n, n, dtype=torch.float64, device='cuda', generator=t)
    return A, torch.randn(n, case['rhs'], dtype=torch.float64, device='cuda', generator=t)


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    case = s['case']
    kind = case['kind']
    if kind in ('plain', 'split') and 'h' in s:
        h = s['h'].h
        torch.ops.bx.state_upload(h, *s['state'])
        torch.ops.bx.step(h, case['steps'], False)
        tops.check_stable(h)
        return dict(zip(('vm', 'cc_cells', 'cc_at_mem', 'cc_env'), torch.ops.bx.state_download(h)))
    if kind in ('plain', 'ecm'):
        e = s['eng']
        e.upload(**s['state'])
        e.step(case['steps'])
        e.check_stable()
        return e.download(out=s['out'])
    if kind == 'sweep':
        e = s['eng']
        e.upload_concat(**s['state'])
        e.step(case['steps'])
        e.check_stable()
        return e.download_concat(out=s['out'])
    if kind == 'sampled':
        h = s['h'].h
        torch.ops.bx.state_upload(h, *s['state'])
        torch.ops.bx.step(h, 1, True)
        tops.check_stable(h)
        o = dict(zip(OUTPUTS, torch.ops.bx.outputs(h)))
        f = dict(zip(FIELDS, torch.ops.bx.env_fields(h, s['weight'])))     # without J_env and B_field (see FIELDS)
        st = dict(zip(('vm', 'cc_cells', 'cc_at_mem', 'cc_env'), torch.ops.bx.state_download(h)))
        return {'outputs': {k: v for k, v in o.items() if v.numel()}, 'fields': f, 'state': st}
    if kind == 'network':
        e, net = s['eng'], s['net']
        e.upload(**s['state'])
        net.upload(*s['sub'])
        net.step(case['steps'], with_ions=True)
        e.check_stable()
        net.check_stable()
        return {'ions': e.download(out=s['out']), 'substances': net.download()}
    if kind in ('lapgj', 'dense'):
        return s['op'].apply(s['X'])
    loss = s['net'].train_step(s['x'], s['y'], LR)
    return {'loss': loss, 'params': s['net'].params()}


OUTPUTS = ('fluxes_mem', 'fluxes_gj', 'rate_NaKATP', 'rho_cells', 'Jn', 'I_mem', 'J_cell_x', 'J_cell_y', 'Jc',
           'vm_ave', 'dvm', 'E_cell_x', 'E_cell_y', 'Emc', 'E_gj_x', 'E_gj_y', 'gjopen', 'sigma_cell',
           'fluxes_env_x', 'fluxes_env_y', 'rho_env', 'v_env')
# the next three that env_fields gives, J_env and B_field, are rounding residue without extracellular
# spaces (the field that is split is a gradient): no number to compare
FIELDS = ('v_env', 'E_env_x', 'E_env_y')


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Bytes: inputs once, outputs once.  Operations: per membrane and step two
    shared exponentials and, for each of six ions, two GHK fluxes and their
    sums; per cell the pump, the update and the charge."""
    kind = case['kind']
    I = 6
    if kind in ('plain', 'ecm', 'split', 'sweep', 'network', 'sampled'):
        C = sum(_sweep_sizes(case['clusters'])) if kind == 'sweep' else case['cells']
        M, G = 6 * C, case.get('grid', 0) ** 2
        bytes_ = M * (8 * I + 2 * 8 * (I + 1) + 21) + C * (2 * 8 * I + 28)
        flops = case.get('steps', 1) * (M * 180 + C * 200)
        if kind == 'ecm':
            bytes_ += G * 8 * (3 * I + 4)
            flops += case['steps'] * G * (I * 30 + 50)
        if kind == 'network':
            bytes_ += 4 * (2 * 8 * M + 2 * 8 * C) + M * 16
            flops += case['steps'] * (M * 90 + C * 200)
        if kind == 'sampled':
            bytes_ += M * 8 * (2 * I + 9) + C * 8 * 7 + 8 * G * G + 6 * 8 * G
            flops += M * 100 + 8 * G * G
        return {'bytes': bytes_, 'flops': flops}
    if kind == 'lapgj':
        # two solves by conjugate gradients with a multigrid cycle: some 60 iterations of some 70 operations a node
        n, K = case['cells'], case['rhs']
        return {'bytes': n * (16 * K + 7 * 12 * 2 + 8), 'flops': 2 * 60 * 70.0 * n * K}
    if kind == 'dense':
        n, K = case['n'], case['rhs']
        return {'bytes': 4 * n * n + 16 * n * K, 'flops': 3 * 2.0 * n * n * K}
    n = case['nodes']
    return {'bytes': n * (4 * (N_IN + N_OUT) + 4 * 7) + 3 * 4 * 33000, 'flops': 3 * 2.0 * n * 64 * 64 * 8}


# ---------------------------------------------------------------------------
# the same in plain torch, 64 bits (BETSE's formulas)
# ---------------------------------------------------------------------------
def _dev():
    return 'cuda' if torch.cuda.is_available() else 'cpu'


def _ghk(cA, cB, D, d, z, v, p):
    a = (z + NONCE) * (v + NONCE) * (p.F / (p.R * p.T))
    return -(D * a / d) * ((cB - cA * torch.exp(-a)) / -torch.expm1(-a))


class _Ref:
    """Clusters side by side: BETSE's time step on concatenated arrays."""

    def __init__(self, gs, ps, Dms, sts, D_env=None):
        d = _dev()
        self.p = p = ps[0]
        mo = np.cumsum([0] + [g.n_mems for g in gs])
        co = np.cumsum([0] + [g.n_cells for g in gs])
        ten = lambda a, t=torch.float64: torch.as_tensor(np.ascontiguousarray(a), dtype=t, device=d)  # noqa: E731
        cat = lambda f: np.concatenate([np.asarray(f(g)) for g in gs])  # noqa: E731
        off = lambda f, o: ten(np.concatenate([np.asarray(f(g)) + o[k] for k, g in enumerate(gs)]), torch.int64)  # noqa: E731
        self.m2c, self.nn = off(lambda g: g.mem_to_cells, co), off(lambda g: g.nn_i, mo)
        self.map = ten(cat(lambda g: g.map_mem2ecm), torch.int64)
        for n in ('mem_sa', 'mem_nx', 'mem_ny', 'gj_weight', 'cell_vol', 'cell_sa', 'diviterm', 'smooth_weight_mem',
                  'smooth_weight_o'):
            setattr(self, n, ten(cat(lambda g, n=n: getattr(g, n))))
        self.bnd = ten(cat(lambda g: g.bflag), torch.bool)
        self.cl = ten(np.repeat(np.arange(len(gs)), np.diff(mo)), torch.int64)
        self.alpha = ten([q.alpha_NaK * q.nakatp_block for q in ps])[self.cl]
        self.vol_env, self.n_mem = ten([q.vol_env for q in ps]), ten(np.diff(mo))
        self.z = ten(p.zs)[:, None]
        self.Dgj, self.Dfree = ten(p.D_gj)[:, None], ten(p.D_free)[:, None]
        self.gj_len, self.delta, self.shape = gs[0].gj_len, gs[0].delta, tuple(gs[0].grid_shape)
        self.C, self.M = int(co[-1]), int(mo[-1])
        self.Dm = ten(np.concatenate(Dms, axis=1))
        self.vm = ten(np.concatenate([s['vm'] for s in sts]))
        self.cc = ten(np.concatenate([s['cc_cells'] for s in sts], axis=1))
        self.cam = self.cc[:, self.m2c]
        self.go = self.gj_weight.clone() if p.v_sensitive_gj else p.gj_block * self.gj_weight
        self.ecm = bool(p.is_ecm)
        if self.ecm:
            self.env = ten(sts[0]['cc_env'])
            self.Ex, self.Ey = ten(sts[0]['E_env_x']), ten(sts[0]['E_env_y'])
            self.D_env, self.bound = ten(D_env), ten(p.c_env_bound)
            self.touched = torch.zeros(self.env.shape[1], dtype=torch.bool, device=d)
            self.touched[self.map] = True
            self.msa = float(np.asarray(gs[0].mem_sa_per_env)[np.asarray(gs[0].map_mem2ecm)].mean())
        else:
            self.env = ten(np.stack([s['cc_env'] for s in sts], axis=1))

    def seg(self, x):
        out = torch.zeros(*x.shape[:-1], self.C, dtype=x.dtype, device=x.device)
        return out.index_add_(-1, self.m2c, x)

    def gate(self, vgj):
        p, V = self.p, 1e3 * vgj.abs() - self.p.gj_vthresh
        a, b = 0.0013 * torch.exp(-0.077 * V), 0.0013 * torch.exp(0.14 * V)
        b = b / (1 + 50 * b)
        dt = 1e3 * p.dt
        self.go = p.gj_block * ((self.go + dt * (a + b * p.gj_min)) / (1 + a * dt + b * dt))

    def step(self):
        p, z = self.p, self.z
        RT = p.R * p.T
        env = self.env[:, self.map] if self.ecm else self.env[:, self.cl]
        cam, vm = self.cam, self.vm
        nai, nao, ki, ko = cam[I_NA], env[I_NA], cam[I_K], env[I_K]
        Q = (p.cADP * p.cPi * 1e-6 * (nao * 1e-3) ** 3 * (ki * 1e-3) ** 2) / (
            p.cATP * 1e-3 * (nai * 1e-3) ** 3 * (ko * 1e-3) ** 2)
        keq = torch.exp(-(p.deltaGATP / RT - p.F * vm / RT))
        xn, xk, xa = (nai / p.KmNK_Na) ** 3, (ko / p.KmNK_K) ** 2, p.cATP / p.KmNK_ATP
        self.fNa = -3 * self.alpha * (xn * xk * xa / ((1 + xn) * (1 + xk) * (1 + xa))) * (1 - Q / keq)
        f = _ghk(env, cam, self.Dm, p.tm, z, vm, p)
        f[I_NA] += self.fNa
        f[I_K] -= (2.0 / 3.0) * self.fNa
        self.vgj = vgj = vm[self.nn] - vm
        fg = torch.empty_like(f)
        for i in range(len(z)):
            if p.v_sensitive_gj:
                self.gate(vgj)
            fg[i] = _ghk(cam[i], cam[i][self.nn], self.Dgj[i] * p.gj_surface * self.go, self.gj_len, z[i], vgj, p)
        fg[:, self.bnd] = 0.0
        if self.ecm:
            self.env = self.np_update()
        if p.iCa >= 0 and p.alpha_Ca > 0:
            ci, co = self.cc[p.iCa][self.m2c].clamp(min=0), env[p.iCa].clamp(min=0)
            x = ci / p.KmCa_Ca
            xa = p.cATP / p.KmCa_ATP
            keq = torch.exp(-(p.deltaGATP / RT - 2 * p.F * vm / RT))
            f[p.iCa] -= p.alpha_Ca * (x * xa / ((1 + x) * (1 + xa))) * (1 - (p.cADP * p.cPi * co / (p.cATP * ci)) / keq)
        cc = self.cc + self.seg(f * self.mem_sa) / self.cell_vol * p.dt
        self.cam = cc[:, self.m2c]
        if self.ecm:
            out = torch.zeros_like(self.env).index_add_(1, self.map, -f * self.mem_sa)
            self.env = self.env + out / (p.cell_height * self.delta ** 2) * p.dt
        else:
            tot = torch.zeros_like(self.env).index_add_(1, self.cl, -f * self.mem_sa)
            self.env = self.env + tot * (p.dt / (self.vol_env * self.n_mem))
        self.cc = (cc + p.dt * self.seg(-fg * self.mem_sa) / self.cell_vol).clamp(min=0)
        self.rho = (z * p.F * self.cc).sum(0)
        self.vm_old = vm
        if self.ecm:
            self.field()
        self.vm = (1 / p.cm) * (self.rho * self.diviterm)[self.m2c]
        self.f, self.fg = f, fg

    # ---- the environment grid
    def grad(self, F):
        d, gx, gy = self.delta, torch.empty_like(F), torch.empty_like(F)
        gx[..., 1:-1] = (F[..., 2:] - F[..., :-2]) / (2 * d)
        gy[..., 1:-1, :] = (F[..., 2:, :] - F[..., :-2, :]) / (2 * d)
        gx[..., 0], gx[..., -1] = (F[..., 1] - F[..., 0]) / d, (F[..., -1] - F[..., -2]) / d
        gy[..., 0, :], gy[..., -1, :] = (F[..., 1, :] - F[..., 0, :]) / d, (F[..., -1, :] - F[..., -2, :]) / d
        return gx, gy

    def div(self, Fx, Fy):
        """The reference's divergence: one-sided edges with its signs."""
        d, x, y = self.delta, torch.empty_like(Fx), torch.empty_like(Fy)
        x[..., 1:-1] = (Fx[..., 2:] - Fx[..., :-2]) / (2 * d)
        y[..., 1:-1, :] = (Fy[..., 2:, :] - Fy[..., :-2, :]) / (2 * d)
        x[..., 0], x[..., -1] = (Fx[..., 0] - Fx[..., 1]) / d, (Fx[..., -2] - Fx[..., -1]) / d
        y[..., 0, :], y[..., -1, :] = (Fy[..., 0, :] - Fy[..., 1, :]) / d, (Fy[..., -2, :] - Fy[..., -1, :]) / d
        return x + y

    def gauss(self, a, reflect):
        w = torch.exp(-0.5 * torch.arange(-4, 5, dtype=torch.float64, device=a.device) ** 2)
        w = w / w.sum()
        for ax in (0, 1):
            n = a.shape[ax]
            k = torch.arange(-4, n + 4, device=a.device)
            src = torch.where(k < 0, -k - 1, torch.where(k >= n, 2 * n - 1 - k, k))
            pad = a.index_select(ax, src)
            if not reflect:
                inside = ((k >= 0) & (k < n)).double()
                pad = pad * (inside[:, None] if ax == 0 else inside[None, :])
            a = sum(w[q] * pad.narrow(ax, q, n) for q in range(9))
        return a

    def np_update(self):
        p = self.p
        c = self.env.view(-1, *self.shape).clone()
        b = self.bound[:, None]
        c[:, :, 0], c[:, :, -1] = b, b
        c[:, 0, :], c[:, -1, :] = b, b
        D = self.D_env.view_as(c)
        a = D * (self.z * p.q / (p.kb * p.T))[..., None]
        gx, gy = self.grad(c)
        fx, fy = -D * gx + a * self.Ex * c, -D * gy + a * self.Ey * c
        return (c + self.div(-fx, -fy) * p.dt).view_as(self.env)

    def field(self):
        p = self.p
        rho = (self.z * p.F * self.env).sum(0)
        src = torch.where(self.touched, rho * (p.cell_height * self.delta ** 2) / self.msa, torch.zeros_like(rho))
        v = self.gauss((src / (p.ko_env * p.eo * p.er)).view(self.shape), False)
        gx, gy = self.grad((2 / (p.ko_env * self.delta)) * (p.cell_radius / p.true_cell_size) * v)
        self.Ex, self.Ey = -gx, -gy

    def state(self):
        d = {'vm': self.vm, 'cc_cells': self.cc, 'cc_at_mem': self.cam, 'cc_env': self.env}
        if self.ecm:
            d.update(E_env_x=self.Ex.reshape(-1), E_env_y=self.Ey.reshape(-1))
        elif self.env.shape[1] == 1:
            d['cc_env'] = self.env[:, 0]
        else:
            d['cc_env'] = self.env.T
        if self.p.v_sensitive_gj:
            d['gjopen'] = self.go
        return d

    # ---- a sampled step's outputs and environment fields
    def outputs(self):
        p, zF, nx, ny = self.p, self.z * self.p.F, self.mem_nx, self.mem_ny
        J = -(zF * self.f).sum(0) + (zF * self.fg).sum(0)
        Jn = self.smooth_weight_mem * J + (self.seg(J * self.mem_sa) / self.cell_sa)[self.m2c] * self.smooth_weight_o
        jx, jy = (self.seg(Jn * n * self.mem_sa) / self.cell_sa for n in (nx, ny))
        sig = ((self.z ** 2) * p.F ** 2 * self.cc * self.Dfree * 0.1 / (p.R * p.T)).mean(0)
        ex, ey = jx / sig, jy / sig
        at = lambda a, b: a[self.m2c] * nx + b[self.m2c] * ny  # noqa: E731
        eg = -self.vgj / self.gj_len
        n = torch.zeros(self.C, dtype=torch.float64, device=J.device).index_add_(0, self.m2c, torch.ones_like(J))
        return dict(fluxes_mem=self.f.reshape(-1), fluxes_gj=self.fg.reshape(-1), rate_NaKATP=-self.fNa,
                    rho_cells=self.rho, Jn=Jn, I_mem=-Jn * self.mem_sa, J_cell_x=jx, J_cell_y=jy, Jc=at(jx, jy),
                    vm_ave=self.seg(self.vm) / n, dvm=(self.vm - self.vm_old) / p.dt, E_cell_x=ex, E_cell_y=ey,
                    Emc=at(ex, ey), E_gj_x=eg * nx, E_gj_y=eg * ny, gjopen=self.go, sigma_cell=sig)

    def fields(self, lap):
        vce = torch.zeros(self.shape, dtype=torch.float64, device=lap.device).view(-1)
        last = torch.full((vce.numel(),), -1, dtype=torch.int64, device=lap.device)
        last.scatter_reduce_(0, self.map, torch.arange(self.M, device=lap.device), 'amax')
        hit = last >= 0
        vce[hit] = (self.vm_old / 2)[self.m2c][last[hit]]      # the membrane vector, read at cell indices
        phi = self.gauss(-vce.view(self.shape), True)

        def inner(F):
            out = torch.zeros_like(F)
            out[1:-1, 1:-1] = F[1:-1, 1:-1]
            return out

        def decomp(Jx, Jy):
            AA = torch.linalg.solve(lap, -inner(self.div(-Jy, Jx)).reshape(-1)).view(self.shape)
            BB = torch.linalg.solve(lap, inner(self.div(Jx, Jy)).reshape(-1)).view(self.shape)
            ax, ay = self.grad(AA)
            return -ay, ax, *self.grad(BB)

        rx, ry, dx, dy = decomp(*self.grad(self.delta * phi))
        Ex, Ey = -(rx + dx), -(ry + dy)
        return {k: v.reshape(-1) for k, v in zip(FIELDS, (phi, Ex, Ey))}


def _laplacian(g):
    """FiniteDiffSolver.makeLaplacian: 5 points inside, identity on the edges."""
    ny, nx = g.grid_shape
    G = ny * nx
    k = torch.arange(G, device=_dev())
    i, j = k // nx, k % nx
    inside = (i > 0) & (i < ny - 1) & (j > 0) & (j < nx - 1)
    A = torch.zeros(G, G, dtype=torch.float64, device=_dev())
    ki, kb = k[inside], k[~inside]
    A[ki, ki], A[kb, kb] = -4.0, 1.0
    for o in (nx, -nx, 1, -1):
        A[ki, ki + o] = 1.0
    return A / g.delta ** 2


class _RefNetwork:
    """The four-substance network of _network_config beside a _Ref."""

    def __init__(self, ref, g, seed):
        _, _, spot, gmod, c0, env0 = _network_config(g, seed)
        ten = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=_dev())  # noqa: E731
        self.r, self.gmod, self.c, self.env = ref, ten(gmod), ten(c0), ten(env0)
        self.spot = torch.zeros(ref.C, dtype=torch.float64, device=_dev())
        self.spot[torch.as_tensor(spot, device=_dev())] = 1.0
        self.cm = self.c[:, ref.m2c]
        self.R = ten(g.R_rads)
        self.gamma = ref.mem_sa / (0.75 * 0.5 * self.R * ref.mem_sa)
        self.keq = math.exp(-KEQ_DG / (ref.p.R * ref.p.T))

    def step(self, vm, vgj):
        r, p, c = self.r, self.r.p, self.c
        hill = lambda x, km, n=1: (x / km) ** n / (1 + (x / km) ** n)  # noqa: E731
        kq = self.gamma * 1e-11 * p.dt / self.R
        cm = c[:, r.m2c]
        cm[3] = (kq * c[3][r.m2c] + self.cm[3]) / (1 + kq)
        r1 = 0.01 * hill(c[1], 0.1, 2) * hill(c[0], 0.1) * hill(c[2], 0.2)
        r2 = 0.02 * (1 - (1e-3 * c[1] ** 2) / (1e-3 * c[3]) / self.keq)
        rate = torch.stack([self.gmod * 0.5 * (1 / (1 + (c[2] / 0.3) ** 2)) - 0.2 * c[0] - r1,
                            self.spot * ((hill(c[0], 0.2, 2) + hill(c[2], 0.5)) - 0.5 * c[1]) + 2 * r2,
                            0.2 * hill(c[1], 0.1) - 0.1 * c[2] - r1,
                            0.05 / (1 + c[2] / 0.4) - 0.05 * c[3] + r1 - r2])
        c = c + rate * p.dt
        for k, (z, Dm, Dgj) in enumerate(((0, 0.0, 1e-15), (0, 0.0, None), (-1, 1e-18, 1e-14), (0, 5e-19, 1e-15))):
            if Dm:
                f = _ghk(self.env[k], cm[k], Dm, p.tm, z, vm, p)
                c[k] += r.seg(f * r.mem_sa) / r.cell_vol * p.dt
                cm[k] = cm[k] + f * self.gamma * p.dt if k == 3 else c[k][r.m2c]
                self.env[k] -= (f * r.mem_sa).sum() * p.dt / (p.vol_env * r.M)
            else:
                cm[k] = c[k][r.m2c]
            if Dgj is not None:
                f = _ghk(cm[k], cm[k][r.nn], Dgj * p.gj_block * r.go, r.gj_len, z, vgj, p)
                f[r.bnd] = 0.0
                c[k] += p.dt * r.seg(-f * r.mem_sa) / r.cell_vol
                cm[k] = cm[k] - f * self.gamma * p.dt if k == 3 else c[k][r.m2c]
        self.c, self.cm = c, cm


def _cg(apply, B):
    """Columns of L+ B by conjugate gradients on the mean-free space."""
    B = B - B.mean(0)
    X, R = torch.zeros_like(B), B.clone()
    P, rr, bb = R.clone(), (R * R).sum(0), (B * B).sum(0)
    for it in range(6000):
        Q = apply(P)
        a = torch.where(rr > 0, rr / (P * Q).sum(0).clamp(min=1e-300), torch.zeros_like(rr))
        X += a * P
        R -= a * Q
        new = (R * R).sum(0)
        if it % 50 == 0 and bool((new <= 1e-28 * bb).all()):
            break
        P = R + torch.where(rr > 0, new / rr.clamp(min=1e-300), torch.zeros_like(rr)) * P
        rr = new
    return X - X.mean(0)


def _exact_lapgj(case, seed):
    _, (edges, tri, vor, area), X = _lapgj_inputs(case, seed)
    n = len(area)
    e = torch.as_tensor(np.asarray(edges), device=X.device)
    w = torch.as_tensor(np.asarray(tri) / np.asarray(vor), device=X.device)

    def laplacian(weight):
        i = torch.cat([e[:, 0], e[:, 1], e[:, 0], e[:, 1]])
        j = torch.cat([e[:, 1], e[:, 0], e[:, 0], e[:, 1]])
        return torch.sparse_coo_tensor(torch.stack([i, j]), torch.cat([-weight, -weight, weight, weight]),
                                       (n, n)).coalesce().to_sparse_csr()

    L, Lw = laplacian(torch.ones_like(w)), laplacian(w)
    Y = _cg(lambda P: L @ P, torch.as_tensor(np.asarray(area), device=X.device)[:, None] * X)
    return -_cg(lambda P: L @ P, Lw @ Y)


def _exact_train(case, seed):
    ptr, nbr, x, y, w = _train_inputs(case, seed)
    d, W = x.device, 64
    p = torch.as_tensor(w, device=d).double().requires_grad_(True)
    deg = torch.as_tensor(np.diff(ptr), device=d).double()
    row = torch.as_tensor(np.repeat(np.arange(len(ptr) - 1), np.diff(ptr)), device=d)
    col = torch.as_tensor(np.asarray(nbr, np.int64), device=d)
    at = 0

    def take(*shape):
        nonlocal at
        n = math.prod(shape)
        at += n
        return p[at - n:at].view(*shape)

    X = torch.zeros(len(x), W, dtype=torch.float64, device=d)
    X[:, :N_IN] = x.double()
    H = torch.relu(X @ take(W, W).T + take(W))
    for _ in range(3):
        Ws, Wn, b = take(W, W), take(W, W), take(W)
        A = torch.zeros_like(H).index_add(0, row, H[col]) / deg.clamp(min=1)[:, None]
        H = H + torch.relu(H @ Ws.T + A @ Wn.T + b)
    out = (H @ take(W, W).T + take(W))[:, :N_OUT]
    loss = ((out - y.double()) ** 2).mean()
    loss.backward()
    g = p.grad
    new = p.detach() - LR * g / (g.abs() + 1e-8)              # Adam's first step
    return {'loss': float(loss), 'params': new.cpu().numpy()}


def exact(case, seed):
    kind = case['kind']
    if kind == 'lapgj':
        return _exact_lapgj(case, seed)
    if kind == 'dense':
        A, X = _dense_inputs(case, seed)
        return A @ X
    if kind == 'train':
        return _exact_train(case, seed)
    if kind == 'sweep':
        ref = _Ref(*_sweep(case, seed))
    else:
        g, p, Dm, st, D_env = _workload(dict(case, resumed=True) if kind == 'sampled' else case, seed)
        ref = _Ref([g], [p], [Dm], [st], D_env)
    if kind == 'network':
        net = _RefNetwork(ref, g, seed)
        for _ in range(case['steps']):
            vm = ref.vm
            ref.step()
            net.step(vm, ref.vgj)
        return {'ions': ref.state(), 'substances': {'c_cells': net.c, 'cc_at_mem': net.cm, 'c_env': net.env}}
    for _ in range(case.get('steps', 1)):
        ref.step()
    if kind == 'sampled':
        return {'outputs': ref.outputs(), 'fields': ref.fields(_laplacian(g)), 'state': ref.state()}
    return ref.state()
