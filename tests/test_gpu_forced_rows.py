"""Rows that are forced in every source of a batched FP32 run, as an adjoint's
receivers are: the group kernels add a lane's right-hand sides in one pass over
a row's sorted entries. Sources that lack a row, rows forced in one source
only, and counts of sources that fill a lane's four right-hand sides or not;
every source against its own run, to the FP32 bound of the other parity tests
(1e-4, max-normalised)."""
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


@pytest.mark.parametrize("R,variant", [(R, v) for R in (5, 24, 70) for v in (24, 26)] + [(64, 20), (64, 22), (16, 20), (32, 22)])
def test_rows_forced_in_every_source(bfe, R, variant, monkeypatch):
    m = modelgen.coupled_model(W=2.1e-3, Hw=0.9e-3, Hs=1.0e-3, h=0.1e-3, abs_thick=0.3e-3)
    n = m["K"].shape[0]
    t, s = modelgen.pulse(150, m["dt"])
    rng = np.random.default_rng(2)
    common = rng.choice(n, 6, replace=False) + 1
    srcs, F = [], np.zeros((8, t.size, R))
    for r in range(R):
        rows = np.concatenate([common[: 6 if r % 3 else 4], [1 + (17 * r) % n, 1 + (29 * r + 3) % n]])
        srcs.append(rows)
        F[: rows.size, :, r] = rng.uniform(-1, 1, (rows.size, 1)) * s
    hi = np.arange(1, n + 1, 5)
    monkeypatch.setenv("BFE_VARIANT", str(variant))
    with bfe.Plan(m["K"], m["C"], m["M"], m["dt"], bfe.VEL_CURRENT, "single", m["gl"]) as plan:
        h = plan.run_batched(t, srcs, F, hi)
        assert plan.stats()["variant"] == variant
        for r in range(R):
            h1, _, _ = plan.run(t, srcs[r], F[: len(srcs[r]), :, r], hi)
            assert np.abs(h1).max() > 0
            assert np.abs(h[:, :, r] - h1).max() <= 1e-4 * np.abs(h1).max(), r
