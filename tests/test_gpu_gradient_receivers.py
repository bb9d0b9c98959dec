"""Receivers that share a cell: their residuals are added in the order of the
list, so the gradient is the same, bit for bit, from run to run and for every
checkpoint interval."""
import numpy as np
import pytest
import torch

from viscoelasticinversion_b200 import StepPlan, media
from viscoelasticinversion_b200.gradient import GRADIENT_PLANES, misfit_gradient
from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz,kind,precision,tol", [(131, 40, "vti", "f32", 1e-3), (75, 37, "tti", "f64", 1e-10)])
def test_gradient_with_many_receivers_in_a_cell(oracle_lib, nx, nz, kind, precision, tol):
    w = media.layered(nx=nx, nz=nz, nt=40, kind=kind, seed=3, pml=6, nrec=6, nlayers=3, f0=30.0)
    cells = [(nx // 2, 9), (nx // 2 + 1, 9), (nx // 2, 10)]
    # 3 x 60 in turn, and 150 in a row, all in one tile
    w.receivers = list(w.receivers) + 60 * cells + 150 * cells[:1]
    rng = np.random.default_rng(1)
    obs = rng.standard_normal((2, len(w.receivers), w.nt)) * 10.0 ** rng.uniform(-12, -8, (1, len(w.receivers), 1))
    plan = StepPlan.for_workload(w, precision)
    med = plan.medium_to_device(w.medium)
    wav = torch.as_tensor(w.wavelets, dtype=plan.dtype, device=plan.device).contiguous()
    o = torch.as_tensor(obs, dtype=plan.dtype, device=plan.device).contiguous()
    J, g = misfit_gradient(plan, med, w.sources, wav, w.receivers, o)
    for k in range(30):
        Jk, gk = misfit_gradient(plan, med, w.sources, wav, w.receivers, o, checkpoint_every=(0, 7, 40)[k % 3])
        assert Jk == J and torch.equal(gk, g), k
    plan.close()
    J0, g0 = oracle_lib.gradient(w, obs)
    assert abs(J - J0) <= (1e-4 if precision == "f32" else 1e-12) * J0
    for n, k in enumerate(GRADIENT_PLANES):
        if np.any(g0[n]):
            assert rel_l2(g[n].cpu().numpy(), g0[n]) <= tol, k
