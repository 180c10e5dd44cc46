"""Marches that become non-finite return what the kernels that sum a row's own
entries give, wherever they ran: on the chip and in the any-R group kernels
node blocks hold zeros for absent entries, and 0 x inf is NaN. Time steps far
above the stability limit; every sample is compared, NaN for NaN, with the
one-launch-per-step kernels (BFE_NO_GRAPH=1) or the slice kernel
(BFE_VARIANT=0)."""
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
    b = model.steel_block_3d(1.1e-3, 1.3e-3, 0.7e-3, 0.1e-3, n_mon=9)
    return dict(plate=(modelgen.solid_plate(W=5e-3, H=2.3e-3, h=0.1e-3), 2),
                coupled=(modelgen.coupled_model(W=5e-3, Hw=1.5e-3, Hs=1.5e-3, h=0.1e-3, blob=True), 4),
                brick=(dict(b, frc_nd=b["src_nodes"][0]), 3))


def _inputs(m, dof, prec):
    nt, scale = (600, 2.2) if prec == "double" else (300, 1.8)
    t = np.arange(nt) * scale * m["dt"]
    k = np.arange(nt)
    s = np.sin(k / 3.0) * np.exp(-((k - 10) / 6.0) ** 2)
    return t, s, modelgen.gi_of(m["gl"], [m["frc_nd"]], dof)


def _unstable(bfe, call):
    with pytest.raises(bfe.BfeError) as e:
        call()
    assert e.value.status == 7
    return e.value.outputs


def _equal(a, b):
    assert not np.isfinite(b).all()
    assert np.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("prec", ["double", "single"])
@pytest.mark.parametrize("name", ["plate", "coupled", "brick"])
def test_one_source(bfe, models, name, prec, monkeypatch):
    m, dof = models[name]
    t, s, fi = _inputs(m, dof, prec)
    n = m["K"].shape[0]

    def run():
        with bfe.Plan(m["K"], m["C"], m["M"], t[1], bfe.VEL_CURRENT, prec, m["gl"], one_source=True) as plan:
            return _unstable(bfe, lambda: plan.run(t, fi, s, np.arange(1, n + 1), 50, True))

    monkeypatch.delenv("BFE_NO_GRAPH", raising=False)
    on = run()
    monkeypatch.setenv("BFE_NO_GRAPH", "1")
    off = run()
    _equal(on[0], off[0])
    _equal(on[1], off[1])


@pytest.mark.parametrize("prec", ["double", "single"])
@pytest.mark.parametrize("name,R", [("plate", 3), ("plate", 21), ("coupled", 5), ("brick", 4)])
def test_several_sources(bfe, models, name, R, prec, monkeypatch):
    m, dof = models[name]
    t, s, fi = _inputs(m, dof, prec)
    n = m["K"].shape[0]
    srcs = [np.array([(int(fi[0]) + 31 * r) % n + 1]) for r in range(R)]
    hi = np.arange(1, n + 1, 3)

    def run():
        with bfe.Plan(m["K"], m["C"], m["M"], t[1], bfe.VEL_CURRENT, prec, m["gl"]) as plan:
            return _unstable(bfe, lambda: plan.run_batched(t, srcs, s, hi))

    monkeypatch.delenv("BFE_VARIANT", raising=False)
    on = run()
    monkeypatch.setenv("BFE_VARIANT", "0")
    _equal(on, run())


@pytest.mark.parametrize("prec", ["double", "single"])
def test_prescribed_displacements(bfe, models, prec, monkeypatch):
    m, _ = models["plate"]
    t, s, fi = _inputs(m, 2, prec)
    di = modelgen.gi_of(m["gl"], np.nonzero(np.isclose(m["mod"]["nds"][:, 0], 0.0))[0] + 1, 2)
    D = 1e-9 * np.linspace(0.5, 1.0, di.size)[:, None] * s[None, :]

    def run():
        with bfe.Plan(m["K"], m["C"], m["M"], t[1], bfe.V5, prec, m["gl"], one_source=True) as plan:
            h, f, frc, _ = _unstable(bfe, lambda: plan.run_v5(t, fi, s, di, D, np.arange(1, plan.n + 1), 45))
            return h, f, frc

    monkeypatch.delenv("BFE_NO_GRAPH", raising=False)
    on = run()
    monkeypatch.setenv("BFE_NO_GRAPH", "1")
    for a, b in zip(on, run()):
        _equal(a, b)


@pytest.mark.parametrize("every", [0, 60])
@pytest.mark.parametrize("prec", ["double", "single"])
def test_adjoint(bfe, prec, every, monkeypatch):
    """The history of an adjoint's forward march, kept or from checkpoints, is
    that of the slice kernel, and the gradient does not depend on the route."""
    from bfe_gb300 import model
    m = model.steel_plate_adjoint(W=3e-3, H=1.5e-3, h=0.1e-3, n_src=3, n_rec=9, abs_wavelengths=0.3)
    nt, scale = (700, 2.2) if prec == "double" else (400, 1.8)
    dt = scale * m["dt"]
    t, k = np.arange(nt) * dt, np.arange(nt)
    s = np.sin(k / 3.0) * np.exp(-((k - 10) / 6.0) ** 2)
    hi = model.global_indices(m["gl"], m["rec_nodes"], 2)
    srcs = [model.global_indices(m["gl"], x, 2) for x in m["src_nodes"]]
    obs = np.zeros((hi.size, nt, 3), order="F")

    def run():
        with bfe.Plan(m["K"], m["C"], m["M"], dt, bfe.VEL_CURRENT, prec, m["gl"]) as plan:
            return plan.adjoint_gradient(m["element_data"], t, srcs, s, hi, obs, ckpt_every=every, return_history=True)

    monkeypatch.delenv("BFE_NO_GRAPH", raising=False)
    on = run()
    monkeypatch.setenv("BFE_NO_GRAPH", "1")
    off = run()
    for a, b in zip(on[1:3], off[1:3]):
        assert np.array_equal(a, b, equal_nan=True)
    _equal(on[3], off[3])
    monkeypatch.setenv("BFE_VARIANT", "0")
    with bfe.Plan(m["K"], m["C"], m["M"], dt, bfe.VEL_CURRENT, prec, m["gl"]) as plan:
        _equal(on[3], _unstable(bfe, lambda: plan.run_batched(t, srcs, s, hi)))
