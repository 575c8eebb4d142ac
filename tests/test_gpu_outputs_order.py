"""bx_outputs_download into device memory that work on the default stream still
reads: the download waits for that work, as a copy on the default stream does
(the handle's own stream does not wait for it by itself)."""
import ctypes as ct

import numpy as np
import pytest

import golden_io as gi

pytestmark = pytest.mark.gpu


def test_a_destination_still_in_use_is_not_overwritten():
    import torch
    from betse_gb300 import _lib
    from betse_gb300.engine import ClusterEngine
    cg, sp, Dm, st, _ = gi.engine_inputs(gi.load('noecm_r80_s1'))
    with ClusterEngine(cg, sp, 'fp64') as e:
        e.set_membrane_diffusivity(Dm)
        e.upload(**st)
        e.step(3, outputs=True)
        ref = e.outputs()['vm_ave']
        buf = torch.empty(cg.n_cells, dtype=torch.float64, device='cuda')
        seen = torch.empty_like(buf)
        o = _lib.BxOutputs()
        o.vm_ave = ct.cast(ct.c_void_p(buf.data_ptr()), _lib._dp)
        for _ in range(2):                           # (the first call loads its kernel, which waits for everything)
            buf.fill_(7.0)
            torch.cuda.synchronize()
            torch.cuda._sleep(200_000_000)           # 0.1 s on the default stream, then a read
            seen.copy_(buf)
            _lib.check(_lib.load().bx_outputs_download(e.h, ct.byref(o)), 'bx_outputs_download')
            torch.cuda.synchronize()
    assert torch.all(seen == 7.0)
    assert np.array_equal(buf.cpu().numpy(), ref)
