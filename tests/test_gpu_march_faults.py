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


def _info(bfe, plan):
    import ctypes
    from bfe_gb300 import _lib
    info = _lib.BfeMarchInfo()
    _lib.check(bfe.load().bfe_plan_march_info(plan._h, ctypes.byref(info)))
    return info


def _march(bfe, models, route, prec, nt, faults):
    """Two runs of one plan, with the given faults: outputs, launches and what
    is kept after each."""
    from bfe_gb300 import model
    name = dict(run="plate", coupled="coupled", brick="brick", v5="damped", batch="plate").get(route)
    if route.startswith("adjoint"):
        a = model.steel_plate_adjoint(W=2e-3, H=1e-3, h=0.1e-3, n_src=3, n_rec=4, abs_wavelengths=0.3)
        t, s = modelgen.pulse(nt, a["dt"])
        hi = model.global_indices(a["gl"], a["rec_nodes"], 2)
        srcs = [model.global_indices(a["gl"], x, 2) for x in a["src_nodes"]]
        obs = np.asfortranarray(np.broadcast_to(1e-13 * s[None, :, None], (hi.size, nt, 3)))
        make = lambda: bfe.Plan(a["K"], a["C"], a["M"], a["dt"], bfe.VEL_CURRENT, prec, a["gl"])   # noqa: E731
        every = dict(adjoint=0, adjoint_kept=0, adjoint_segments=nt - 100)[route]
        go = lambda p: p.adjoint_gradient(a["element_data"], t, srcs, s, hi, obs, ckpt_every=every,  # noqa: E731
                                          return_history=True)[1:]
    else:
        m, dof = models[name]
        t, s = modelgen.pulse(nt, m["dt"])
        fi = modelgen.gi_of(m["gl"], [m["frc_nd"]], dof)
        n = m["K"].shape[0]
        hi = np.arange(1, n + 1, 7)
        make = lambda: bfe.Plan(m["K"], m["C"], m["M"], m["dt"], bfe.V5 if route == "v5" else bfe.VEL_CURRENT,  # noqa: E731
                                prec, m["gl"], one_source=route != "batch")
        srcs = [fi, fi + 2, np.array([1]), np.array([n])]
        di = modelgen.gi_of(m["gl"], np.nonzero(np.isclose(m["mod"]["nds"][:, 0], 0.0))[0] + 1, 2) if route == "v5" else None
        go = (lambda p: (p.run_batched(t, srcs, s, hi),)) if route == "batch" else \
            (lambda p: p.run_v5(t, fi, s, di, 1e-9 * np.outer(np.linspace(0.5, 1.0, di.size), s), hi, nt // 9)[:3]) \
            if route == "v5" else (lambda p: p.run(t, fi, s, hi, nt // 9, True)[:2])
    out = []
    with make() as plan:
        for f in faults:
            _fault(bfe, plan, f)
            r = go(plan)
            out.append((r, plan.stats()["step_launches"], _info(bfe, plan)))
    return out


ROUTES = ["run", "coupled", "brick", "v5", "batch", "adjoint", "adjoint_segments"]


@pytest.mark.parametrize("fault", ["BFE_MARCH_FAULT_WAIT", "BFE_MARCH_FAULT_MEMORY"])
@pytest.mark.parametrize("route,prec", [(r, "single") for r in ROUTES] + [("run", "double"), ("batch", "double")])
def test_given_up_marches_step_and_keep_nothing(bfe, models, route, prec, fault, monkeypatch):
    """A wait that runs out, and no memory for the partition: the same bits
    from step kernels, no partition kept, and none built for the next run."""
    from bfe_gb300 import _lib
    monkeypatch.delenv("BFE_NO_GRAPH", raising=False)
    nt = 400
    (sane, _, info), = _march(bfe, models, route, prec, nt, [0])
    assert info.partition_bytes > 0
    for r, launches, info in _march(bfe, models, route, prec, nt, [getattr(_lib, fault), 0]):
        assert info.partition_bytes == 0
        assert launches >= nt
        assert _same(r, sane)


@pytest.mark.parametrize("fault", [0, 1])
@pytest.mark.parametrize("route,prec", [("run", "double"), ("run", "single"), ("coupled", "single"), ("brick", "single"),
                                        ("v5", "double"), ("batch", "double"), ("batch", "single"),
                                        ("adjoint_kept", "single"), ("adjoint_segments", "single")])
def test_marches_of_more_than_one_launch(bfe, models, route, prec, fault, monkeypatch):
    """More samples than one launch marches: the second goes on from the states,
    frames, histories and velocities of the first, or is refused."""
    monkeypatch.delenv("BFE_NO_GRAPH", raising=False)
    (on, launches, _), = _march(bfe, models, route, prec, LONG, [fault])
    forward = LONG if route == "adjoint_segments" else 0           # checkpoints are made step by step
    assert launches < forward + 300 if fault == 0 else launches > forward + LONG - 100
    monkeypatch.setenv("BFE_NO_GRAPH", "1")
    (off, _, _), = _march(bfe, models, route, prec, LONG, [0])
    assert _same(on, off)
