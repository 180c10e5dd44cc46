"""Models that the on-chip marches leave to the step kernels: nothing is built
for them."""
import ctypes

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


def _first_run(bfe, m, prec, nt, R=1):
    from bfe_gb300 import _lib
    t, s = modelgen.pulse(nt, m["dt"])
    s[0] = 1e-3
    n = m["K"].shape[0]
    with bfe.Plan(m["K"], m["C"], m["M"], m["dt"], bfe.VEL_CURRENT, prec, m["gl"], one_source=R == 1) as plan:
        if R == 1:
            plan.run(t, [n // 2], s, [1, n])
        else:
            plan.run_batched(t, [np.array([n // 2 + r]) for r in range(R)], s, [1, n])
        info = _lib.BfeMarchInfo()
        _lib.check(bfe.load().bfe_plan_march_info(plan._h, ctypes.byref(info)))
        return plan.stats()["step_launches"], info


@pytest.mark.parametrize("prec", ["double", "single"])
def test_operators_over_the_limit(bfe, prec):
    """444,000 DOF in 3D: blocks of 330 MB in FP64 and at least 150 MB in FP32."""
    from bfe_gb300 import model
    launches, info = _first_run(bfe, model.steel_block_3d(13e-3, 13e-3, 6.6e-3, 0.2e-3, n_mon=4), prec, 400)
    assert launches == 400
    assert info.partitions_built == 0 and info.partition_bytes == 0


@pytest.mark.parametrize("side,kept", [(7.0e-3, True), (8.0e-3, False), (8.4e-3, False), (9.0e-3, True)])
def test_bricks_that_stream_only_where_that_is_faster(bfe, side, kept):
    """73,872 DOF fit in the SMs' shared memory, 152,352 stream against a step
    kernel that is out of L2; between them the step kernel is faster."""
    from bfe_gb300 import model
    launches, info = _first_run(bfe, model.steel_block_3d(side, side, side / 2, 0.2e-3, n_mon=4), "single", 400)
    assert launches == (1 if kept else 400)
    assert info.partitions_built == (1 if kept else 0) and (info.partition_bytes > 0) == kept


@pytest.mark.parametrize("R", [1, 4])
def test_short_runs_build_once_it_pays(bfe, R):
    """The first 100 samples of a plan of 40,602 DOF and four sources, and of one
    of 161,202 DOF and one, take the step kernels, later ones the chip."""
    from bfe_gb300 import model
    m = model.steel_plate(20e-3, 10e-3, 0.1e-3, 16) if R > 1 else model.steel_plate(40e-3, 20e-3, 0.1e-3, 16)
    t, s = modelgen.pulse(100, m["dt"])
    s[0] = 1e-3
    n = m["K"].shape[0]
    launches, out = [], []
    with bfe.Plan(m["K"], m["C"], m["M"], m["dt"], bfe.VEL_CURRENT, "double", m["gl"], one_source=R == 1) as plan:
        for _ in range(4):
            out.append(plan.run(t, [n // 2], s, [n // 2, n])[0] if R == 1 else
                       plan.run_batched(t, [np.array([n // 2 + r]) for r in range(R)], s, [n // 2, n]))
            launches.append(plan.stats()["step_launches"])
    assert launches == [100, 1, 1, 1]
    for x in out[1:]:
        assert np.abs(x).max() > 0 and np.array_equal(x, out[0])


@pytest.mark.parametrize("W,H,R,kept", [(20e-3, 10e-3, 48, True), (20e-3, 10e-3, 64, False), (30e-3, 15e-3, 24, True),
                                        (30e-3, 15e-3, 36, False), (40e-3, 20e-3, 12, True), (40e-3, 20e-3, 16, False),
                                        (200e-3, 2e-3, 24, True)])
def test_tiles_are_cut_only_for_source_counts_that_fit(bfe, W, H, R, kept):
    """Plates of 40,602, 90,902 and 161,202 DOF on both sides of what fits, and a
    thin one, whose parts have few neighbours."""
    from bfe_gb300 import model
    launches, info = _first_run(bfe, model.steel_plate(W, H, 0.1e-3, 16), "single", 700, R)
    assert (launches == 1) == kept
    assert info.partitions_built == (1 if kept else 0)
