"""The server's estimate of a request covers what it holds on the device: its
buffers and its plan's workspace (admission keeps the sum of the estimates
within the HBM budget)."""
import re

import numpy as np
import pytest
import torch

from viscoelasticinversion_b200 import StepPlan, media
from viscoelasticinversion_b200._abi import BudgetError
from viscoelasticinversion_b200.gradient import misfit_gradient
from viscoelasticinversion_b200.serve import Server

pytestmark = pytest.mark.gpu


# planes of more than the estimate's 16 MB of slack; each medium and precision,
# rows with and without padding
@pytest.mark.parametrize("kind", ["iso", "vti", "tti"])
@pytest.mark.parametrize("nsls", [0, 1, 3])
@pytest.mark.parametrize("nx", [2048, 2049])
@pytest.mark.parametrize("precision", ["f32", "f64"])
def test_estimate_covers_buffers_and_workspace(kind, nsls, nx, precision):
    nz, nt, e = 1024, 5, 8 if precision == "f64" else 4
    w = media.homogeneous_iso(nx=nx, nz=nz, nt=nt, pml=10, nrec=4)
    one = np.ones((nz, nx))
    med = {"rho": 2000 * one, "c13": 4e9 * one, "c55": 4e9 * one}
    if kind != "iso":
        med.update(c11=1.2e10 * one, c33=1.2e10 * one)
    if kind == "tti":
        med.update(c15=0 * one, c35=0 * one)
    if nsls:
        med["tau"] = 0.01 * one
    w.kind, w.medium, w.taus = kind, med, np.geomspace(1e-3, 1e-1, nsls) if nsls else np.zeros(0)
    obs = np.zeros((2, len(w.receivers), nt))
    plan = StepPlan.for_workload(w, precision)
    dmed, wav = plan.medium_to_device(med), torch.as_tensor(w.wavelets, dtype=plan.dtype, device="cuda").contiguous()
    held = {}
    # a request's buffers: eight medium planes, state, wavelets, traces (for a
    # gradient: observed traces and eight FP64 planes)
    buf = (8 + 5 + 3 * nsls) * nx * nz * e + (w.wavelets.size + 2 * len(w.receivers) * nt) * e
    # a gradient request checkpoints every ceil(sqrt(nt)) steps
    misfit_gradient(plan, dmed, w.sources, wav, w.receivers, torch.zeros(*obs.shape, dtype=plan.dtype, device="cuda"),
                    checkpoint_every=3)
    held["gradient"] = buf + plan.workspace_bytes() + 64 * nx * nz + obs.size * e
    plan.close()
    plan = StepPlan.for_workload(w, precision)
    st = plan.zeros_state()
    plan.step(dmed, st, nsteps=1, sources=w.sources, wavelets=wav, receivers=w.receivers)
    plan.status()
    held["forward"] = buf + plan.workspace_bytes()
    plan.close()
    del st, dmed
    server = Server(hbm_budget_bytes=1)
    try:
        for kind_, submit in (("forward", lambda: server.submit_forward(w, precision)),
                              ("gradient", lambda: server.submit_gradient(w, obs, precision))):
            with pytest.raises(BudgetError) as err:
                submit()
            estimate = int(re.search(r"needs (\d+) device bytes", str(err.value)).group(1))
            assert held[kind_] <= estimate, (kind_, estimate - held[kind_])
    finally:
        server.stop()
