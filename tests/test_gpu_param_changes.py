"""bx_set_params after create with other ions: charges BETSE's six-ion set does
not have, and back.  Each of the two runs kernels of its own, so what was laid
out for one at create (tables, shared memory, the co-resident launch) has to
follow.

Against a handle created with the new parameters, bit for bit."""
import numpy as np
import pytest

import golden_io as gi
import synthetic

pytestmark = pytest.mark.gpu


def _other_ions(d):
    """P as a trivalent anion of a third of the concentration: the same charge."""
    d = dict(d)
    i = [str(x) for x in d['par_ion_names']].index('P')
    z = np.array(d['par_zs'], np.float64)
    z[i] = -3.0
    d['par_zs'] = z
    for k in ('init_cc_cells', 'init_cc_at_mem', 'init_cc_env'):
        d[k] = np.array(d[k])
        d[k][i] /= 3.0
    return d


@pytest.mark.parametrize('back', [False, True])
@pytest.mark.parametrize('name,precision,tpb,kernel', [
    ('noecm_r80_s1', 'fp64', 0, 0), ('noecm_r50_s9_vgj', 'fp64', 256, 0), ('ecm_r50_s3', 'fp64', 256, 0),
    (None, 'fp64', 256, 0),
    ('noecm_r80_s1', 'split', 256, 'tile'), ('noecm_r80_s1', 'split', 256, 'persistent'),
    ('noecm_r80_s1', 'split', 256, 'factored'), ('noecm_r80_s1', 'split', 192, 'pipelined'),
    ('noecm_r80_s1', 'split', 256, 'resident')])
def test_other_charges_after_create(name, precision, tpb, kernel, back):
    from betse_gb300.engine import ClusterEngine
    a = gi.load(name) if name else synthetic.ragged_fixture(n_cells=400)
    b = _other_ions(a)
    if back:
        a, b = b, a
    ia, ib = gi.engine_inputs(a), gi.engine_inputs(b)
    got = []
    for change in (True, False):
        with ClusterEngine(ib[0], ia[1] if change else ib[1], precision) as e:
            e.set_membrane_diffusivity(ib[2])
            if ib[1].is_ecm:
                e.set_env_diffusivity(ib[4])
            if tpb:
                e.set_launch_config(tpb, kernel)
            if change:
                e.upload(**ia[3])
                e.step(40)
                e.set_params(ib[1])
            e.upload(**ib[3])
            e.step(40)
            e.check_stable()
            got.append(e.download())
    for k in got[1]:
        assert np.array_equal(got[0][k], got[1][k]), k
