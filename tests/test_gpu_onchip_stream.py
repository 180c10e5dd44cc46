"""On-chip marches whose operator does not fit in shared memory: slices that
stream from L2 beside resident ones, slots used in turn across steps, slices of
several chunks. Bit for bit against one launch per step (BFE_NO_GRAPH=1): the
same operations in the same order."""
import numpy as np
import pytest

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


def _models():
    from bfe_gb300 import model
    # operator blocks of 40 MB and more: the SMs hold about 34
    yield "plate", "double", lambda: model.steel_plate(61e-3, 30e-3, 0.1e-3, 16)
    yield "coupled", "double", lambda: model.coupled_water_steel(90e-3, 30e-3, 15e-3, 0.1e-3, abs_wavelengths=3.0)
    yield "brick", "double", lambda: model.steel_block_3d(6.4e-3, 6.4e-3, 3.2e-3, 0.2e-3, n_mon=4)
    yield "plate", "single", lambda: model.steel_plate(90e-3, 45e-3, 0.1e-3, 16)
    yield "coupled", "single", lambda: model.coupled_water_steel(60e-3, 20e-3, 10e-3, 0.05e-3, abs_wavelengths=3.0)
    yield "brick", "single", lambda: model.steel_block_3d(9.2e-3, 9.2e-3, 4.6e-3, 0.2e-3, n_mon=4)


@pytest.mark.parametrize("name,prec", [(n, p) for n, p, _ in _models()])
def test_streamed_operators(bfe, name, prec, monkeypatch):
    import ctypes
    from bfe_gb300 import _lib
    m = {(n, p): make for n, p, make in _models()}[name, prec]()
    n = m["K"].shape[0]
    t, s = modelgen.pulse(301, m["dt"])
    rng = np.random.default_rng(8)
    fi = np.sort(rng.choice(n, 40, replace=False)) + 1
    F = np.outer(rng.uniform(0.5, 2.0, 40), s)
    hi = np.concatenate([rng.choice(n, 500, replace=False) + 1, [1, n]])

    def run():
        with bfe.Plan(m["K"], m["C"], m["M"], m["dt"], bfe.VEL_CURRENT, prec, m["gl"], one_source=True) as plan:
            out = [plan.run(t, fi, F * k, hi, 150, True)[:2] for k in (1.0, -0.5)]
            info = _lib.BfeMarchInfo()
            _lib.check(bfe.load().bfe_plan_march_info(plan._h, ctypes.byref(info)))
            return out, plan.stats()["step_launches"], info.partition_bytes

    monkeypatch.delenv("BFE_NO_GRAPH", raising=False)
    on, launches, kept = run()
    assert launches == 1 and kept > 40e6
    monkeypatch.setenv("BFE_NO_GRAPH", "1")
    off, launches, _ = run()
    assert launches == 301 - np.argmax(s != 0)
    for a, b in zip(on, off):
        for x, y in zip(a, b):
            assert np.abs(y).max() > 0 and np.array_equal(x, y)
