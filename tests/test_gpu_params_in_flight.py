"""bx_set_params and bx_batch_set_params right after bx_step, which returns while
its steps run: the steps in flight keep the parameters they were called with.

Against the same calls with a wait between them, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS = 300                      # some ten times the host time of the call that follows


@pytest.mark.parametrize('precision,kernel,ecm', [('fp64', 'tile', False), ('fp64', 'tile', True),
                                                  ('split', 'tile', False), ('split', 'factored', False),
                                                  ('split', 'tile', True)])
def test_parameters_of_one_cluster(precision, kernel, ecm):
    import torch
    from betse_gb300 import generator as gen
    from betse_gb300.engine import ClusterEngine
    g, p, Dm, st, D_env = gen.workload(662e-6, 11, is_ecm=ecm, dt=1e-3, grid_size=60 if ecm else 20)
    q = p.replace(alpha_NaK=0.0, vol_env=p.vol_env * 3)
    got = []
    for wait in (False, True):
        with ClusterEngine(g, p, precision) as e:
            e.set_membrane_diffusivity(Dm)
            if ecm:
                e.set_env_diffusivity(D_env)
            e.upload(**st)
            e.set_launch_config(256, kernel)
            e.step(STEPS)                                # builds what a first call builds
            e.set_params(q)
            e.upload(**st)
            e.step(STEPS)
            if wait:
                torch.cuda.synchronize()
            e.set_params(p)
            e.check_stable()
            got.append(e.download())
    for k in got[1]:
        assert np.array_equal(got[0][k], got[1][k]), k


@pytest.mark.parametrize('precision', ['fp64', 'split'])
def test_parameters_of_a_batch(precision):
    import ctypes as ct

    import torch
    from betse_gb300 import _lib, generator as gen
    from betse_gb300.engine import BatchEngine
    wl = [gen.workload(300e-6, s, dt=1e-3) for s in (3, 5, 7, 11)]
    gs, ps, Dms, sts = ([w[i] for w in wl] for i in range(4))
    qs = [p.replace(alpha_NaK=0.0, vol_env=p.vol_env * 3) for p in ps]
    got = []
    for wait in (False, True):
        with BatchEngine(gs, ps, precision) as e:
            def params(x):
                c = (_lib.BxParams * len(x))(*[p.to_c() for p in x])
                _lib.check(e.lib.bx_batch_set_params(e.h, c), 'bx_batch_set_params')
            e.set_membrane_diffusivity(Dms)
            e.upload_states(sts)
            e.step(STEPS)
            params(qs)
            e.upload_states(sts)
            e.step(STEPS)
            if wait:
                torch.cuda.synchronize()
            params(ps)
            e.check_stable()
            got.append(e.download_states())
    for a, b in zip(*got):
        for k in b:
            assert np.array_equal(a[k], b[k]), k
