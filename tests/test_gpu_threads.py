"""Plans of different sizes on threads of their own: every march stays on the
chip (one launch) and gives the bits it gives alone, although the plans share
the kernels whose shared-memory limit each launch sets."""
import threading

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


@pytest.mark.parametrize("R", [1, 4])
def test_marches_on_three_threads(bfe, R, monkeypatch):
    monkeypatch.delenv("BFE_NO_GRAPH", raising=False)
    monkeypatch.delenv("BFE_VARIANT", raising=False)
    jobs = []
    for W, H in ((1e-3, 0.6e-3), (9e-3, 6e-3), (0.4e-3, 0.3e-3)):
        m = modelgen.solid_plate(W=W, H=H, h=0.1e-3)
        t, s = modelgen.pulse(160, m["dt"])
        n = m["K"].shape[0]
        srcs = [np.array([1 + (7 * r) % n]) for r in range(R)]
        plan = bfe.Plan(m["K"], m["C"], m["M"], m["dt"], bfe.VEL_CURRENT, "single", m["gl"], one_source=R == 1)
        hi = np.arange(1, n + 1, 5)

        def run(plan=plan, t=t, s=s, srcs=srcs, hi=hi):
            h = plan.run(t, srcs[0], s, hi)[0] if R == 1 else plan.run_batched(t, srcs, s, hi)
            return h, plan.stats()["step_launches"]

        jobs.append((plan, run, run()))
        assert jobs[-1][2][1] == 1
    bad = []

    def work(k):
        for _ in range(300):
            h, launches = jobs[k][1]()
            if launches != 1 or not np.array_equal(h, jobs[k][2][0]):
                bad.append((k, launches))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(jobs))]
    for x in threads:
        x.start()
    for x in threads:
        x.join()
    for plan, _, _ in jobs:
        plan.close()
    assert not bad
