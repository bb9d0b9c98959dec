"""A grid with more rows than a launch has blocks in y: the padded copies of
odd rows take it, as the fused kernel did.  Against the plain path on the last
rows alone: two steps carry nothing over more than 32 rows."""
import pytest
import torch

from viscoelasticinversion_b200 import StepPlan
from viscoelasticinversion_b200.solver import make_config

pytestmark = pytest.mark.gpu


def test_padded_copies_of_a_tall_grid():
    nx, nz, part = 13, 8 * 65536 + 21, 400  # one row of 8-row blocks more than 65535
    g = torch.Generator(device="cuda").manual_seed(0)
    out = {}
    for variant, rows in ((0, nz), (1, part)):
        plan = StepPlan(make_config(nx, rows, 5.0, 5.0, 4e-4, free_surface=True))
        med = {"rho": torch.full((rows, nx), 2000.0, device="cuda"), "c13": torch.full((rows, nx), 4e9, device="cuda"),
               "c55": torch.full((rows, nx), 4e9, device="cuda")}
        g.manual_seed(0)
        st = {k: torch.randn(*t.shape[:-2], nz, nx, generator=g, device="cuda")[..., nz - rows:, :].contiguous()
              for k, t in plan.zeros_state().items()}
        st["v"] *= 1e-7
        plan.step(med, st, nsteps=2, variant=variant)
        plan.status()
        assert plan.last_kernel() == ("split" if variant == 0 else "plain")
        out[variant] = st
        plan.close()
    for k in ("v", "s"):
        a, b = out[0][k][..., 64 - part:, :].double(), out[1][k][..., 64:, :].double()
        assert (a - b).norm() <= 1e-6 * b.norm(), k
        assert torch.equal(a[..., -4:, :], b[..., -4:, :])
