"""Marches that stay on the chip when they cannot be finished there: faults
injected on the host (bfe_plan_set_march_fault), the results compared bit for
bit with a run that takes one launch per step from the start (BFE_NO_GRAPH=1).
"""
import numpy as np
import pytest

import modelgen

pytestmark = pytest.mark.gpu

LONG = 8400                                       # samples: more than the 8,192 steps of one launch


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


@pytest.fixture(scope="module")
def models():
    from bfe_gb300 import model
    b = model.steel_block_3d(0.9e-3, 0.7e-3, 0.5e-3, 0.1e-3, n_mon=4)
    return dict(plate=(modelgen.solid_plate(W=2.3e-3, H=1.1e-3, h=0.1e-3), 2),
                damped=(modelgen.solid_plate(W=3e-3, H=2e-3, h=0.1e-3, abs_thick=0.6e-3), 2),
                coupled=(modelgen.coupled_model(W=2e-3, Hw=1e-3, Hs=1e-3, h=0.1e-3), 4),
                brick=(dict(b, frc_nd=b["src_nodes"][0], mon_nds=b["mon_nodes"]), 3))


def _fault(bfe, plan, fault):
    from bfe_gb300 import _lib
    _lib.check(bfe.load().bfe_plan_set_march_fault(plan._h, fault))


def _same(a, b):
    return all(np.array_equal(x, y) and np.abs(y).max() > 0 for x, y in zip(a, b))


def _v5(bfe, m, prec, nt, fault):
    """A v5 run whose dynamic velocity matters: prescribed DOFs in the
    absorbing layer (their C enters it) and frames that show it."""
    t, s = modelgen.pulse(nt, m["dt"])
    nds = m["mod"]["nds"]
    low = np.nonzero(np.isclose(nds[:, 0], nds[:, 0].min()))[0] + 1
    di = modelgen.gi_of(m["gl"], low, 2)
    D = 1e-9 * np.linspace(0.5, 1.0, di.size)[:, None] * s[None, :]
    fi = modelgen.gi_of(m["gl"], [m["frc_nd"]], 2)
    hi = np.concatenate([di[:2], modelgen.gi_of(m["gl"], m["mon_nds"], 1)])
    with bfe.Plan(m["K"], m["C"], m["M"], m["dt"], bfe.V5, prec, m["gl"], one_source=True) as plan:
        _fault(bfe, plan, fault)
        h, f, frc, _ = plan.run_v5(t, fi, s, di, D, hi, 600)
        return (h, f, frc), plan.stats()


@pytest.mark.parametrize("prec", ["double", "single"])
def test_v5_starts_again_from_rest_when_a_later_launch_is_refused(bfe, models, prec, monkeypatch):
    from bfe_gb300 import _lib
    m, _ = models["damped"]
    monkeypatch.delenv("BFE_NO_GRAPH", raising=False)
    on, st = _v5(bfe, m, prec, LONG, _lib.BFE_MARCH_FAULT_LAUNCH)
    assert st["step_launches"] == 1 + LONG        # the first piece, then every step
    monkeypatch.setenv("BFE_NO_GRAPH", "1")
    off, _ = _v5(bfe, m, prec, LONG, _lib.BFE_MARCH_FAULT_NONE)
    assert _same(on, off)
