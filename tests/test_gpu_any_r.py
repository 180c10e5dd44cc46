"""Batched runs with any number of sources on plans with node information:
the group kernels lay the states out in multiples of 4 (FP32) or 2 (FP64)
right-hand sides. Source counts around the multiples and around one pass of 64
right-hand sides, for 2D node blocks with fluid and interface rows and for 3D
ones; every source is compared with its own one-source run, to the bounds of
the other parity tests (1e-10 FP64, 1e-4 FP32, max-normalised)."""
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


@pytest.fixture(scope="module")
def models():
    from bfe_gb300 import model
    c = modelgen.coupled_model(W=2.1e-3, Hw=0.9e-3, Hs=1.0e-3, h=0.1e-3, abs_thick=0.3e-3)
    b = model.steel_block_3d(0.7e-3, 0.6e-3, 0.5e-3, 0.1e-3, n_mon=4)
    return dict(coupled=(c, 4, modelgen.gi_of(c["gl"], c["mon_nds"], 4)),
                brick=(b, 3, modelgen.gi_of(b["gl"], b["mon_nodes"], 3)))


@pytest.mark.parametrize("R", [2, 3, 5, 12, 17, 31, 63, 65, 70])
@pytest.mark.parametrize("prec,tol", [("double", 1e-10), ("single", 1e-4)])
@pytest.mark.parametrize("name", ["coupled", "brick"])
def test_every_source_matches_its_own_run(bfe, models, name, prec, tol, R):
    m, dof, hi = models[name]
    t, s = modelgen.pulse(150, m["dt"])
    nodes = np.nonzero(m["gl"][:, dof - 1] > 0)[0] + 1
    srcs = [modelgen.gi_of(m["gl"], [nodes[(7 * r) % nodes.size]], dof) for r in range(R)]
    F = np.stack([(1.0 + 0.1 * r) * s[None, :] for r in range(R)], axis=2)
    with bfe.Plan(m["K"], m["C"], m["M"], m["dt"], bfe.VEL_CURRENT, prec, m["gl"]) as plan:
        h = plan.run_batched(t, srcs, F, hi)
        assert h.shape == (hi.size, t.size, R)
        for r in {0, R // 2, R - 1}:
            h1, _, _ = plan.run(t, srcs[r], F[:, :, r], hi)
            assert np.abs(h1).max() > 0
            assert np.abs(h[:, :, r] - h1).max() <= tol * np.abs(h1).max(), r


@pytest.mark.parametrize("prec,variant", [("single", 24), ("single", 25), ("single", 26), ("double", 4), ("double", 5)])
@pytest.mark.parametrize("name", ["coupled", "brick"])
def test_forced_variants(bfe, models, name, prec, variant, monkeypatch):
    m, dof, hi = models[name]
    t, s = modelgen.pulse(150, m["dt"])
    nodes = np.nonzero(m["gl"][:, dof - 1] > 0)[0] + 1
    srcs = [modelgen.gi_of(m["gl"], [nodes[(11 * r) % nodes.size]], dof) for r in range(22)]
    monkeypatch.setenv("BFE_VARIANT", str(variant))
    with bfe.Plan(m["K"], m["C"], m["M"], m["dt"], bfe.VEL_CURRENT, prec, m["gl"]) as plan:
        h = plan.run_batched(t, srcs, s, hi)
        assert plan.stats()["variant"] == variant
        h1, _, _ = plan.run(t, srcs[21], s, hi)
    tol = 1e-10 if prec == "double" else 1e-4
    assert np.abs(h[:, :, 21] - h1).max() <= tol * np.abs(h1).max()


def test_adjoint_of_three_sources_is_the_sum_over_sources(bfe):
    from bfe_gb300 import model
    m = model.steel_plate_adjoint(W=2e-3, H=1e-3, h=0.1e-3, n_src=3, n_rec=4, abs_wavelengths=0.3)
    t, s = modelgen.pulse(120, m["dt"])
    hi = model.global_indices(m["gl"], m["rec_nodes"], 2)
    srcs = [model.global_indices(m["gl"], n, 2) for n in m["src_nodes"]]
    obs = np.zeros((hi.size, t.size, 3))
    with bfe.Plan(m["K"], m["C"], m["M"], m["dt"], bfe.VEL_CURRENT, "double", m["gl"]) as plan:
        J, gs, gr = plan.adjoint_gradient(m["element_data"], t, srcs, s, hi, obs)
        one = [plan.adjoint_gradient(m["element_data"], t, [x], s, hi, obs[:, :, :1]) for x in srcs]
    assert abs(J - sum(o[0] for o in one)) <= 1e-10 * abs(J)
    for g, k in ((gs, 1), (gr, 2)):
        ref = sum(o[k] for o in one)
        assert np.abs(g - ref).max() <= 1e-10 * np.abs(ref).max()


@pytest.mark.parametrize("name,R", [("coupled", 48), ("coupled", 61), ("coupled", 128), ("brick", 61), ("brick", 52)])
def test_states_beyond_l2(bfe, name, R):
    """States that exceed L2: the group kernels prefetch the rows and blocks of
    later CTAs, up to the ends of the arrays. Every source against its own run,
    to the FP32 bound of the other parity tests."""
    import torch
    from bfe_gb300 import model
    if name == "coupled":
        m = model.coupled_water_steel(60e-3, 20e-3, 10e-3, 0.1e-3, abs_wavelengths=3.0)
        dof = 4
    else:
        m = model.steel_block_3d(10e-3, 10e-3, 5.6e-3, 0.2e-3, n_mon=4)
        dof = 3
    t, s = modelgen.pulse(40, m["dt"])
    rows = np.nonzero(m["gl"][:, dof - 1] > 0)[0] + 1
    pick = np.r_[rows[0], rows[-1], rows[np.linspace(1, rows.size - 2, R - 2).astype(int)]]
    srcs = [modelgen.gi_of(m["gl"], [x], dof) for x in pick]
    hi = modelgen.gi_of(m["gl"], pick[:4], dof)
    with bfe.Plan(m["K"], m["C"], m["M"], m["dt"], bfe.VEL_CURRENT, "single", m["gl"]) as plan:
        assert 12 * plan.n * R > torch.cuda.get_device_properties(0).L2_cache_size
        h = plan.run_batched(t, srcs, s, hi)
        for r in (0, 1, 2, R - 1):
            h1, _, _ = plan.run(t, srcs[r], s, hi)
            if r < 3:
                assert np.abs(h1).max() > 0
            assert np.abs(h[:, :, r] - h1).max() <= 1e-4 * np.abs(h1).max(), r
