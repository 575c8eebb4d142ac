"""A multigrid hierarchy carried on to a single node and beyond (18 levels, the
last ones of one node each) solves as the shorter one does: the levels above the
dense one are not used."""
import ctypes as ct

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_more_than_sixteen_levels():
    import scipy.sparse as sp
    import torch
    from betse_gb300 import _lib
    from betse_gb300.dense import LapGJ, _incidence, graph_levels
    from test_gpu_graph_solver import _grid
    n = 1001
    edges, tri, vor, area = _grid(n)
    D = _incidence(edges, n)
    levels, _ = graph_levels(D.T @ D, 1)
    while len(levels) < 18:
        levels.append(sp.csr_matrix(np.zeros((1, 1))))
    Lw = sp.csr_matrix(D.T @ sp.diags(tri / vor) @ D)
    keep = []

    def lvl(A):
        a = [np.ascontiguousarray(A.indptr, np.int32), np.ascontiguousarray(A.indices, np.int32),
             np.ascontiguousarray(A.data, np.float64)]
        a = [x if x.size else np.zeros(1, x.dtype) for x in a]
        keep.extend(a)
        return _lib.BxGraphLevel(n=A.shape[0], nnz=A.nnz, row_ptr=_lib.iptr(a[0]), col=_lib.iptr(a[1]),
                                 val=_lib.dptr(a[2]))

    lib = _lib.load()
    h = ct.c_void_p()
    pinv = np.zeros(1)
    arr = (_lib.BxGraphLevel * len(levels))(*[lvl(A) for A in levels])
    wl = lvl(Lw)
    _lib.check(lib.bx_graph_create(len(levels), arr, _lib.dptr(pinv), ct.byref(wl), _lib.dptr(np.asarray(area)), 3,
                                   ct.byref(h)), 'bx_graph_create')
    X = torch.randn(n, 3, dtype=torch.float64, device='cuda', generator=torch.Generator('cuda').manual_seed(1))
    Y = torch.empty_like(X)
    torch.cuda.synchronize()
    _lib.check(lib.bx_lap_gj_apply(h, ct.c_void_p(X.data_ptr()), ct.c_void_p(Y.data_ptr()), 3, 1e-12, 1000, None, None,
                                   ct.c_void_p(0)), 'bx_lap_gj_apply')
    torch.cuda.synchronize()
    lib.bx_graph_destroy(h)
    with LapGJ(edges, tri, vor, area, max_rhs=3) as op:
        assert torch.equal(Y, op.apply(X, tol=1e-12))
