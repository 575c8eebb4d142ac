"""State and outputs by one gathered copy where both sides are on the device,
by separate copies where one is not: CUDA tensors, pinned and pageable host
arrays must give the same bits, also through views that start at an odd
element (8-byte alignment only), and a state that fails its check still leaves
the handle without one."""
import ctypes as ct

import numpy as np
import pytest

import golden_io as gi

pytestmark = pytest.mark.gpu

KEYS = ('vm', 'cc_cells', 'cc_at_mem', 'cc_env', 'gjopen', 'E_env_x', 'E_env_y')


def _arrays(st, where):
    import torch
    out = {}
    for k, v in st.items():
        v = np.ascontiguousarray(v, np.float64)
        if where == 'device':
            t = torch.empty(v.size + 1, dtype=torch.float64, device='cuda')[1:]
            t.copy_(torch.as_tensor(v.ravel()))
        else:
            t = torch.empty(v.size + 1, dtype=torch.float64, pin_memory=where == 'pinned')[1:]
            t.numpy()[:] = v.ravel()
        out[k] = t
    torch.cuda.synchronize()
    return out


def _struct(cls, arrays):
    from betse_gb300 import _lib
    s = cls()
    for k, t in arrays.items():
        setattr(s, k, ct.cast(ct.c_void_p(t.data_ptr()), _lib._dp))
    return s


@pytest.mark.parametrize('name,precision', [('noecm_r50_s9_vgj', 'fp64'), ('noecm_r50_s7', 'split'),
                                            ('ecm_r50_s3', 'fp64'), ('ecm_r50_s3', 'split')])
def test_device_and_host_arrays_give_the_same_bits(name, precision):
    from betse_gb300 import _lib
    from betse_gb300.engine import ClusterEngine
    lib = _lib.load()
    d = gi.load(name)
    cg, sp, Dm, st, D_env = gi.engine_inputs(d)
    if sp.is_ecm:
        st['cc_env'] = np.asarray(st['cc_env'])
    else:
        st['cc_env'] = np.asarray(st['cc_env'])[:, 0] if np.ndim(st['cc_env']) == 2 else st['cc_env']
    got = {}
    for where in ('device', 'pinned', 'pageable'):
        with ClusterEngine(cg, sp, precision) as e:
            e.set_membrane_diffusivity(Dm)
            if sp.is_ecm:
                e.set_env_diffusivity(D_env)
            a = _arrays(st, where)
            _lib.check(lib.bx_state_upload(e.h, ct.byref(_struct(_lib.BxState, a))), 'bx_state_upload')
            e.step(5, outputs=True)
            out = _arrays({k: np.zeros(v.shape) for k, v in st.items()}, where)
            s = _struct(_lib.BxState, out)
            _lib.check(lib.bx_state_download(e.h, ct.byref(s)), 'bx_state_download')
            got[where] = {k: v.cpu().numpy().copy() for k, v in out.items()}
            if where == 'pageable':
                got[where + '_out'] = {k: np.asarray(v).copy() for k, v in e.outputs().items()}
            ref = e.download()
            for k in ref:
                assert np.array_equal(np.ravel(ref[k]), got[where][k]), (where, k)
            a['cc_at_mem'][0] += 1.0                                # no longer one value per cell
            rc = lib.bx_state_upload(e.h, ct.byref(_struct(_lib.BxState, a)))
            assert rc != 0 and lib.bx_state_download(e.h, ct.byref(s)) != 0
    for where in ('pinned', 'pageable'):
        for k in got['device']:
            assert np.array_equal(got[where][k], got['device'][k]), (where, k)


def test_outputs_into_device_and_host_arrays():
    import torch
    from betse_gb300 import torch_ops as tops
    from betse_gb300 import _lib
    from betse_gb300.engine import ClusterEngine
    d = gi.load('noecm_r80_s1')
    cg, sp, Dm, st, _ = gi.engine_inputs(d)
    with ClusterEngine(cg, sp, 'fp64') as e:
        e.set_membrane_diffusivity(Dm)
        e.upload(**st)
        e.step(3, outputs=True)
        host = e.outputs()
    h = tops.create(cg, sp, 'fp64')
    torch.ops.bx.set_membrane_diffusivity(h, torch.as_tensor(Dm))
    env = np.asarray(st['cc_env'])
    env = env[:, 0] if env.ndim == 2 else env
    torch.ops.bx.state_upload(h, *(torch.as_tensor(np.ascontiguousarray(st[k]), device='cuda')
                                   for k in ('vm', 'cc_cells', 'cc_at_mem')),
                              torch.as_tensor(np.ascontiguousarray(env), device='cuda'))
    torch.ops.bx.step(h, 3, True)
    dev = dict(zip(_lib.OUTPUT_FIELDS, torch.ops.bx.outputs(h)))
    tops.release(h)
    for k, v in host.items():
        if k in dev and dev[k].numel():
            assert np.array_equal(np.ravel(v), dev[k].cpu().numpy()), k
