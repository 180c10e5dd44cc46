"""FP32 group kernels above 64 right-hand sides, where the L2 prefetches change
their distance (128, 192), stop (320) or start with the size of the states
(192, 256): every source against its own run, to the FP32 bound of the other
parity tests (1e-4, max-normalised)."""
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


@pytest.mark.parametrize("W,R", [(40e-3, 128), (40e-3, 192), (50e-3, 192), (60e-3, 256), (75e-3, 256), (40e-3, 320)])
def test_many_sources_on_a_plate(bfe, W, R):
    import torch
    from bfe_gb300 import model
    m = model.steel_plate(W, W / 2, 0.1e-3, 16)
    t, s = modelgen.pulse(30, m["dt"])
    rows = np.nonzero(m["gl"][:, 1] > 0)[0] + 1
    pick = np.r_[rows[0], rows[-1], rows[np.linspace(1, rows.size - 2, R - 2).astype(int)]]
    srcs = [modelgen.gi_of(m["gl"], [x], 2) for x in pick]
    hi = modelgen.gi_of(m["gl"], pick[:4], 2)
    with bfe.Plan(m["K"], m["C"], m["M"], m["dt"], bfe.VEL_CURRENT, "single", m["gl"]) as plan:
        assert 12 * plan.n * R > torch.cuda.get_device_properties(0).L2_cache_size
        h = plan.run_batched(t, srcs, s, hi)
        for r in (0, 1, 2, R - 1):
            h1, _, _ = plan.run(t, srcs[r], s, hi)
            if r < 3:
                assert np.abs(h1).max() > 0
            assert np.abs(h[:, :, r] - h1).max() <= 1e-4 * np.abs(h1).max(), r
