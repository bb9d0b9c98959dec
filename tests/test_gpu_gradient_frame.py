"""The gradient does not depend on medium values that no updated cell's step
reads: C11, C13, C33 and tau outside the update region, rho beyond the next
cell to the right and the next row, C15, C35 and C55 beyond both.  Zero,
infinite or NaN there, it is bit for bit the one of a filled medium.  Ragged
last groups (nx % 4 in FP32, nx % 2 in FP64) and full ones."""
import numpy as np
import pytest
import torch

from viscoelasticinversion_b200 import StepPlan, media
from viscoelasticinversion_b200.gradient import misfit_gradient

pytestmark = pytest.mark.gpu

L = 4  # half width of the stencil: the frame around the update region


def _read(name, nx, nz):
    """Cells of a plane that the steps of the updated cells read."""
    r = np.zeros((nz, nx), bool)
    r[L:nz - L, L:nx - L] = True
    if name == "rho":
        r[L:nz - L, nx - L] = True
        r[nz - L, L:nx - L] = True
    elif name in ("c15", "c35", "c55"):
        r[L:nz - L + 1, L:nx - L + 1] = True
    return r


@pytest.mark.parametrize("nx,nz,kind,nsls,fs", [
    (75, 37, "tti", 3, True), (75, 37, "vti", 3, True), (75, 37, "iso", 3, True), (74, 40, "tti", 0, False),
    (73, 33, "vti", 1, False), (76, 36, "tti", 2, True), (136, 24, "vti", 2, True)])
@pytest.mark.parametrize("precision", ["f32", "f64"])
def test_gradient_ignores_medium_cells_no_step_reads(nx, nz, kind, nsls, fs, precision):
    w = media.layered(nx=nx, nz=nz, nt=60, kind=kind, seed=nx, pml=7, nrec=6, nlayers=3, f0=30.0, nsls=nsls,
                      free_surface=fs)
    w.sources = list(w.sources) + [(nx - 5, nz // 2, 1, 0.4)]
    w.wavelets = np.repeat(w.wavelets, 2, axis=0)
    w.receivers = list(w.receivers) + [(nx - 5, 8)]
    obs = 1e-9 * np.random.default_rng(nz).standard_normal((2, len(w.receivers), w.nt))
    plan = StepPlan.for_workload(w, precision)
    wav = torch.as_tensor(w.wavelets, dtype=plan.dtype, device=plan.device).contiguous()
    obs = torch.as_tensor(obs, dtype=plan.dtype, device=plan.device).contiguous()

    def run(fill):
        med = {k: np.where(_read(k, nx, nz), v, v if fill is None else fill) for k, v in w.medium.items()}
        return misfit_gradient(plan, plan.medium_to_device(med), w.sources, wav, w.receivers, obs, checkpoint_every=9)

    J, g = run(None)
    assert torch.isfinite(g).all() and g.abs().max() > 0
    for fill in (0.0, np.inf, np.nan):
        Jf, gf = run(fill)
        assert Jf == J and torch.equal(gf, g), fill
    plan.close()
