"""The one-source march that stays on the chip against the step kernels it
replaces: the same operations in the same order, so every output is compared
bit for bit (no tolerance). BFE_NO_GRAPH=1 selects one launch per step.

Sizes: a model of a single slice of 32 rows, ones whose last slice and last
part are partly filled, one with more parts than SMs would need, a 3D model
whose rows are read by many parts, and rows numbered at random (every part
reads from every other)."""
import numpy as np
import pytest
import scipy.sparse as sp

import modelgen
from oracle import solver as osolver

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
    yield "one_slice", modelgen.solid_plate(W=0.3e-3, H=0.3e-3, h=0.1e-3, n_mon=4), 2
    yield "ragged", modelgen.solid_plate(W=2.3e-3, H=1.1e-3, h=0.1e-3), 2
    yield "dof3", modelgen.solid_plate(W=1.7e-3, H=1.1e-3, h=0.1e-3, dof_to_use=(1, 2, 3)), 2
    yield "plate", modelgen.solid_plate(W=12e-3, H=5e-3, h=0.1e-3), 2
    yield "coupled", modelgen.coupled_model(W=5e-3, Hw=1.5e-3, Hs=1.5e-3, h=0.1e-3, blob=True), 4
    b = model.steel_block_3d(1.1e-3, 1.3e-3, 0.7e-3, 0.1e-3, n_mon=9)
    yield "brick", dict(b, frc_nd=b["src_nodes"][0], mon_nds=b["mon_nodes"]), 3


MODELS = ["one_slice", "ragged", "dof3", "plate", "coupled", "brick"]


@pytest.fixture(scope="module")
def models():
    return {name: (m, dof) for name, m, dof in _models()}


def _both(bfe, monkeypatch, run):
    monkeypatch.delenv("BFE_NO_GRAPH", raising=False)
    on, launches = run()
    monkeypatch.setenv("BFE_NO_GRAPH", "1")
    off, launches0 = run()
    assert launches < 16 <= launches0             # the two really took different routes
    return on, off


@pytest.mark.parametrize("prec", ["double", "single"])
@pytest.mark.parametrize("mode", [osolver.VEL_CURRENT, osolver.VEL_LAST_HALF])
@pytest.mark.parametrize("name", MODELS)
def test_same_bits_as_the_step_kernels(bfe, models, name, mode, prec, monkeypatch):
    m, dof = models[name]
    nt = 301
    t, s = modelgen.pulse(nt, m["dt"])
    s = np.concatenate([np.zeros(13), s[:-13]])
    fi = modelgen.gi_of(m["gl"], np.unique([m["frc_nd"], max(m["frc_nd"] - 1, 1)]), dof)
    F = np.vstack([s, -0.5 * s])[: fi.size]
    n = m["K"].shape[0]
    hi = np.concatenate([modelgen.gi_of(m["gl"], m["mon_nds"], dof), [1, n, n]])      # repeated monitor

    def run():
        with bfe.Plan(m["K"], m["C"], m["M"], m["dt"], mode, prec, m["gl"], one_source=True) as plan:
            return plan.run(t, fi, F, hi, 50, True)[:2], plan.stats()["step_launches"]

    (h1, f1), (h0, f0) = _both(bfe, monkeypatch, run)
    assert np.abs(h0).max() > 0
    assert np.array_equal(h1, h0)
    assert np.array_equal(f1, f0)


@pytest.mark.parametrize("prec", ["double", "single"])
def test_random_row_order_and_repeated_runs(bfe, models, prec, monkeypatch):
    """Rows numbered at random (no node information) and three runs of one
    plan, the last with another start sample."""
    m, dof = models["ragged"]
    n = m["K"].shape[0]
    q = np.random.default_rng(3).permutation(n)
    K, C, M = (sp.csr_matrix(A)[q][:, q] for A in (m["K"], m["C"], m["M"]))
    t, s = modelgen.pulse(200, m["dt"])

    def run():
        with bfe.Plan(K, C, M, m["dt"], osolver.VEL_CURRENT, prec) as plan:
            out = [plan.run(t, [5], np.roll(s, k), np.arange(1, n + 1))[0] for k in (0, 0, 40)]
            return out, plan.stats()["step_launches"]

    on, off = _both(bfe, monkeypatch, run)
    for a, b in zip(on, off):
        assert np.array_equal(a, b)
    assert np.array_equal(on[0], on[1])


@pytest.mark.parametrize("ftype", ["sqrt(KE)", "mean(u2)", "div(v)"])
def test_element_fields(bfe, models, ftype, monkeypatch):
    m, dof = models["plate"]
    t, s = modelgen.pulse(260, m["dt"])
    fi = modelgen.gi_of(m["gl"], [m["frc_nd"]], dof)

    def run():
        with bfe.FieldOutput(m["mod"]["nds"], m["mod"]["els"], m["gl"], m["M"], ftype) as fo, \
                bfe.Plan(m["K"], m["C"], m["M"], m["dt"]) as plan:
            return plan.run(t, fi, s, fi, 37, ftype != "mean(u2)", field=fo)[1], plan.stats()["step_launches"]

    on, off = _both(bfe, monkeypatch, run)
    assert np.abs(off).max() > 0 and np.array_equal(on, off)


@pytest.mark.parametrize("prec", ["double", "single"])
@pytest.mark.parametrize("name,cut", [("ragged", 0), ("plate", 0), ("coupled", 5)])
def test_v5_prescribed_displacements(bfe, models, name, cut, prec, monkeypatch):
    """Prescribed DOFs on chip: a repeated one (the last entry sets it), one
    that is forced too, one that is monitored, rows with absorbing damping;
    reactions and frames included."""
    m, _ = models[name]
    nt = 260
    t, s = modelgen.pulse(nt, m["dt"])
    nds = m["mod"]["nds"]
    low = np.nonzero(nds[:, 1] < nds[:, 1].max() / 3)[0] + 1            # solid, away from the interface
    low = low[np.linspace(cut, low.size - 1, 37).astype(int)]
    di = modelgen.gi_of(m["gl"], low, 2)
    di = np.concatenate([di, di[:1]])
    D = 1e-9 * np.linspace(0.5, 1.0, di.size)[:, None] * np.roll(s, 9)[None, :]
    fi = np.concatenate([modelgen.gi_of(m["gl"], [m["frc_nd"]], 4 if name == "coupled" else 2), di[3:4]])
    hi = np.concatenate([di[:4], modelgen.gi_of(m["gl"], low + 1, 1)])

    def run():
        with bfe.Plan(m["K"], m["C"], m["M"], m["dt"], bfe.V5, prec, m["gl"], one_source=True) as plan:
            h, f, frc, _ = plan.run_v5(t, fi, s, di, D, hi, 45)
            return (h, f, frc), plan.stats()["step_launches"]

    on, off = _both(bfe, monkeypatch, run)
    for a, b in zip(on, off):
        assert np.abs(b).max() > 0 and np.array_equal(a, b)


@pytest.mark.parametrize("prec", ["double", "single"])
@pytest.mark.parametrize("R", [2, 3, 8, 15])
@pytest.mark.parametrize("name", ["one_slice", "ragged", "dof3", "plate", "brick"])
def test_several_sources(bfe, models, name, R, prec, monkeypatch):
    """Several sources on chip against the group kernels, bit for bit: two
    forced DOFs per source, one of them shared by all, repeated monitors."""
    m, dof = models[name]
    if prec == "double" or name == "brick":               # more take the step kernels
        R = min(R, 7 if name != "brick" or prec == "single" else 4)
    t, s = modelgen.pulse(140, m["dt"])
    n = m["K"].shape[0]
    nodes = np.nonzero(m["gl"][:, dof - 1] > 0)[0] + 1
    both = modelgen.gi_of(m["gl"], [m["frc_nd"]], dof)
    srcs = [np.concatenate([both, modelgen.gi_of(m["gl"], [nodes[(5 * r + 1) % nodes.size]], dof)]) for r in range(R)]
    F = np.stack([np.vstack([s, -0.3 * s]) * (1 + r) for r in range(R)], axis=2)
    hi = np.concatenate([modelgen.gi_of(m["gl"], m["mon_nds"], dof), [1, n, n]])

    def run():
        with bfe.Plan(m["K"], m["C"], m["M"], m["dt"], bfe.VEL_CURRENT, prec, m["gl"]) as plan:
            h = [plan.run_batched(t, srcs, F[:, :, :] * k, hi) for k in (1.0, 2.0)]
            return h, plan.stats()["step_launches"]

    on, off = _both(bfe, monkeypatch, run)
    for a, b in zip(on, off):
        assert np.abs(b).max() > 0 and np.array_equal(a, b)


def _tile_models():
    from bfe_gb300 import model
    p = modelgen.solid_plate(W=9e-3, H=4.7e-3, h=0.1e-3)
    yield "wide", p["K"], p["C"], p["M"], p["gl"], p["dt"], 2
    p = modelgen.solid_plate(W=3.1e-3, H=12e-3, h=0.1e-3)
    yield "tall", p["K"], p["C"], p["M"], p["gl"], p["dt"], 2
    p = modelgen.solid_plate(W=9e-3, H=4.7e-3, h=0.1e-3, dof_to_use=(3,))
    yield "one_dof", p["K"], p["C"], p["M"], p["gl"], p["dt"], 3
    p = model.steel_subdomain(6e-3, 0.1e-3, seed=3, n_src=4, n_mon=4)      # a void: columns in two pieces
    yield "void", p["K"], p["C"], p["M"], p["gl"], p["dt"], 2


@pytest.mark.parametrize("prec", ["double", "single"])
@pytest.mark.parametrize("name", ["wide", "tall", "one_dof", "void"])
def test_tiles(bfe, name, prec, monkeypatch):
    """Parts cut as tiles against the step kernels, bit for bit: sources and
    monitors all over the model, each in its own order."""
    K, C, M, gl, dt, dof = {x[0]: x[1:] for x in _tile_models()}[name]
    n = K.shape[0]
    rng = np.random.default_rng(5)
    t, s = modelgen.pulse(130, dt)
    nodes = rng.permutation(np.nonzero(gl[:, dof - 1] > 0)[0] + 1)
    srcs = [modelgen.gi_of(gl, nodes[[r, r + 8]], dof) for r in range(8)]
    hi = np.concatenate([rng.permutation(np.arange(1, n + 1))[:700], [1, n, n]])

    def run():
        with bfe.Plan(K, C, M, dt, bfe.VEL_CURRENT, prec, gl) as plan:
            h = [plan.run_batched(t, srcs, s * k, hi) for k in (1.0, 2.0)]
            return h, plan.stats()["step_launches"]

    on, off = _both(bfe, monkeypatch, run)
    for a, b in zip(on, off):
        assert np.abs(b).max() > 0 and np.array_equal(a, b)
