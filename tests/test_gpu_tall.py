"""A grid with more rows than a launch has blocks in y: the padded copies of
odd rows take it, as the fused kernel does."""
import pytest
import torch

from viscoelasticinversion_b200 import StepPlan
from viscoelasticinversion_b200.solver import make_config

pytestmark = pytest.mark.gpu


def test_padded_copies_of_a_tall_grid():
    nx, nz = 13, 8 * 65536 + 21  # one row of 8-row blocks more than 65535
    cfg = make_config(nx, nz, 5.0, 5.0, 4e-4, free_surface=True)
    g = torch.Generator(device="cuda").manual_seed(0)
    out = []
    for variant in (0, 2):
        plan = StepPlan(cfg)
        med = {"rho": torch.full((nz, nx), 2000.0, device="cuda"), "c13": torch.full((nz, nx), 4e9, device="cuda"),
               "c55": torch.full((nz, nx), 4e9, device="cuda")}
        g.manual_seed(0)
        st = {k: torch.randn(t.shape, generator=g, device="cuda") for k, t in plan.zeros_state().items()}
        st["v"] *= 1e-7
        plan.step(med, st, nsteps=2, variant=variant)
        plan.status()
        assert plan.last_kernel() == ("split" if variant == 0 else "fused")
        out.append(st)
        plan.close()
    for k in ("v", "s"):
        a, b = out[0][k].double(), out[1][k].double()
        assert (a - b).norm() <= 1e-6 * b.norm(), k
        assert torch.equal(out[0][k][..., -4:, :], out[1][k][..., -4:, :])
