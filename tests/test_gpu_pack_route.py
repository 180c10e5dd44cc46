"""Which plans have their operator packed on the GPU: sorted CSR of one-source
plans, and nothing else (unsorted rows, CSC, v5 and batched plans take the host
path, which gives the same operator, so only the counter shows the route)."""
import ctypes

import numpy as np
import pytest
import scipy.sparse as sp

import modelgen
from test_gpu_pack import _plan, _view

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def bfe():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from bfe_gb300 import build
    build.build()
    import bfe_gb300
    bfe_gb300.load()
    return bfe_gb300


def _packed(bfe, plan):
    from bfe_gb300 import _lib
    info = _lib.BfeMarchInfo()
    _lib.check(bfe.load().bfe_plan_march_info(plan._h, ctypes.byref(info)))
    return info.packed_on_gpu


@pytest.mark.parametrize("prec", ["double", "single"])
def test_routes(bfe, prec):
    m = modelgen.coupled_model(W=2e-3, Hw=1e-3, Hs=1e-3, h=0.1e-3)
    K = sp.csr_matrix(m["K"])
    K.sort_indices()
    n = K.shape[0]
    zeros = sp.csr_matrix(K + 0.0 * (abs(K) @ abs(K)))
    zeros.sort_indices()
    rev = K.copy()
    for i in range(n):
        a, b = rev.indptr[i], rev.indptr[i + 1]
        rev.indices[a:b] = rev.indices[a:b][::-1].copy()
        rev.data[a:b] = rev.data[a:b][::-1].copy()
    for A, csc, on_gpu in ((K, False, 1), (zeros, False, 1), (rev, False, 0), (K.tocsc(), True, 0)):
        v, keep = _view(A, csc)
        with _plan(bfe, v, m, prec, n) as plan:
            assert _packed(bfe, plan) == on_gpu
    for mode, one, on_gpu in ((bfe.VEL_CURRENT, True, 1), (bfe.VEL_LAST_HALF, True, 1), (bfe.VEL_CURRENT, False, 0),
                              (bfe.V5, True, 0)):
        with bfe.Plan(m["K"], m["C"], m["M"], m["dt"], mode, prec, m["gl"], one_source=one) as plan:
            assert _packed(bfe, plan) == on_gpu
