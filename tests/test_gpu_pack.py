"""The operator of a one-source plan is packed on the GPU from sorted CSR; any
other input takes the host path. Both give the same operator, so the marches
are compared bit for bit: sorted CSR against the same matrix with unsorted
rows, explicit zeros, a missing diagonal entry and as CSC. Irregular matrices
are refused with the host path's errors."""
import ctypes

import numpy as np
import pytest
import scipy.sparse as sp

import modelgen

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


def _view(A, csc=False):
    from bfe_gb300 import _lib
    p, i, v = (np.ascontiguousarray(x, t) for x, t in ((A.indptr, np.int64), (A.indices, np.int64), (A.data, float)))
    return _lib.BfeSparse(A.shape[0], A.shape[1], v.size, _lib.BFE_CSC if csc else _lib.BFE_CSR,
                          _lib.ptr(p, ctypes.c_int64), _lib.ptr(i, ctypes.c_int64), _lib.ptr(v, ctypes.c_double)), (p, i, v)


def _plan(bfe, Kv, m, prec, n):
    from bfe_gb300 import _lib
    from bfe_gb300.solver import dof_maps_from_lookup
    Cv, c = _view(sp.csr_matrix(m["C"]))
    Mv, k = _view(sp.csr_matrix(m["M"]))
    node, typ = dof_maps_from_lookup(m["gl"], n)
    lib = bfe.load()
    return bfe.Plan.from_handle_factory(
        lambda out, mode, pr: lib.bfe_plan_create_ex(ctypes.byref(Kv), ctypes.byref(Cv), ctypes.byref(Mv), m["dt"],
                                                     mode, pr, _lib.ptr(node, ctypes.c_int64),
                                                     _lib.ptr(typ, ctypes.c_int32), _lib.BFE_PLAN_ONE_SOURCE, out),
        n, m["dt"], bfe.VEL_CURRENT, prec)


@pytest.mark.parametrize("prec", ["double", "single"])
@pytest.mark.parametrize("name", ["tiny", "plate", "dof3", "coupled"])
def test_same_operator_as_the_host_path(bfe, name, prec):
    m = dict(tiny=lambda: modelgen.solid_plate(W=0.2e-3, H=0.2e-3, h=0.1e-3, n_mon=2),
             plate=lambda: modelgen.solid_plate(W=2.3e-3, H=1.1e-3, h=0.1e-3),
             dof3=lambda: modelgen.solid_plate(W=1.1e-3, H=0.9e-3, h=0.1e-3, dof_to_use=(1, 2, 3)),
             coupled=lambda: modelgen.coupled_model(W=2e-3, Hw=1e-3, Hs=1e-3, h=0.1e-3))[name]()
    K = sp.csr_matrix(m["K"])
    K.sort_indices()
    n = K.shape[0]
    if name == "plate" and prec == "double":             # a row without its diagonal entry
        K = K.tolil()
        K[7, 7] = 0.0
        K = sp.csr_matrix(K)
        K.eliminate_zeros()
    rev = K.copy()                                        # every row in reverse order
    for i in range(n):
        a, b = rev.indptr[i], rev.indptr[i + 1]
        rev.indices[a:b] = rev.indices[a:b][::-1].copy()
        rev.data[a:b] = rev.data[a:b][::-1].copy()
    zeros = K.tocoo()                                     # explicit zeros, sorted
    pattern = abs(K) @ abs(K)
    zeros = sp.csr_matrix((K + 0.0 * pattern))
    full = sp.csr_matrix((np.zeros(pattern.nnz), pattern.indices, pattern.indptr), shape=K.shape)
    r = np.repeat(np.arange(n), np.diff(pattern.indptr))
    full.data = np.asarray(K[r, pattern.indices]).ravel()
    full.sort_indices()
    t, s = modelgen.pulse(120, m["dt"])
    out = []
    for A, csc in ((K, False), (rev, False), (full, False), (K.tocsc(), True)):
        v, keep = _view(A, csc)
        with _plan(bfe, v, m, prec, n) as plan:
            h, _, _ = plan.run(t, [1 + n // 2], s, np.arange(1, n + 1))
            st = plan.stats()
            out.append((h, st["nnz_stored"], st["nnz_padded"], st["n_direct_rows"]))
    assert np.abs(out[0][0]).max() > 0
    for o in out[1:]:
        assert np.array_equal(o[0], out[0][0]) and o[1:] == out[0][1:]


@pytest.mark.parametrize("what,status", [("index", 1), ("pointer", 1), ("nan", 4)])
def test_irregular_matrices_are_refused(bfe, what, status):
    m = modelgen.solid_plate(W=1e-3, H=1e-3, h=0.1e-3)
    K = sp.csr_matrix(m["K"]).copy()
    n = K.shape[0]
    v, (p, i, x) = _view(K)
    if what == "index":
        i[5] = n
    elif what == "pointer":
        p[3] = p[4] + 1
    else:
        x[9] = np.nan
    with pytest.raises(bfe.BfeError) as e:
        _plan(bfe, v, m, "double", n)
    assert e.value.status == status and "K" in str(e.value)
