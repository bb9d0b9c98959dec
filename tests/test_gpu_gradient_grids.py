"""The adjoint sweep's tile edges: grids whose rows are no multiple of the
vector width, tile remainders, every mechanism count, receivers that share a
cell, the summed form and unaligned media, against the oracle's discrete
adjoint (FP64 1e-10, FP32 1e-3, the bars of test_gpu_gradient.py)."""
import dataclasses

import numpy as np
import pytest
import torch

from viscoelasticinversion_b200 import StepPlan, media
from viscoelasticinversion_b200.gradient import GRADIENT_PLANES, misfit_gradient
from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu


def _problem(nx, nz, kind, nsls, fs, force, nt=90):
    w = media.layered(nx=nx, nz=nz, nt=nt, kind=kind, seed=nx, pml=7, nrec=6, nlayers=3, f0=30.0, nsls=nsls,
                      free_surface=fs)
    i, j = nx - 5, nz // 2  # a source and two receivers on the last updated column
    w = dataclasses.replace(w, receivers=list(w.receivers) + [(i, 8), (i, 8), (4, 4)],
                            sources=list(w.sources) + ([(i, j, 1, 0.4), (nx - 6, j, 2, 0.3)] if force else []))
    wav = w.wavelets[0]
    w = dataclasses.replace(w, wavelets=np.stack([np.roll(wav, 3 * q) for q in range(len(w.sources))]))
    rng = np.random.default_rng(nz)
    obs = 1e-9 * rng.standard_normal((2, len(w.receivers), nt))
    return w, obs


def _run(w, obs, precision, K=0, plan=None, med=None, **kw):
    plan = plan or StepPlan.for_workload(w, precision)
    med = med or plan.medium_to_device(w.medium)
    wav = torch.as_tensor(w.wavelets, dtype=plan.dtype, device=plan.device).contiguous()
    obs_d = torch.as_tensor(obs, dtype=plan.dtype, device=plan.device).contiguous()
    return misfit_gradient(plan, med, w.sources, wav, w.receivers, obs_d, checkpoint_every=K, **kw)


# widths 8 * 64 cells and one to three more or fewer; one row and one short row
# of tiles; the smallest updated region that holds the surface's images
CASES = [(73, 41, "iso", 3, True, False), (70, 48, "vti", 3, True, True), (75, 37, "tti", 3, True, False),
         (137, 21, "tti", 2, False, True), (72, 20, "vti", 5, True, False), (139, 52, "iso", 0, False, True),
         (67, 33, "tti", 0, True, True), (81, 29, "tti", 5, True, False), (78, 30, "vti", 1, False, False)]


@pytest.mark.parametrize("nx,nz,kind,nsls,fs,force", CASES)
def test_gradient_on_ragged_grids_equals_oracle_adjoint(oracle_lib, nx, nz, kind, nsls, fs, force):
    w, obs = _problem(nx, nz, kind, nsls, fs, force)
    J0, g0 = oracle_lib.gradient(w, obs)
    J, g = _run(w, obs, "f64")
    assert abs(J - J0) <= 1e-12 * J0
    Jk, gk = _run(w, obs, "f64", K=8)  # checkpoints and recomputed segments
    assert Jk == J and torch.equal(g, gk)
    J32, g32 = _run(w, obs, "f32")
    assert abs(J32 - J0) <= 1e-4 * J0
    for n, k in enumerate(GRADIENT_PLANES):
        ref = g0[n]
        if not np.any(ref):
            assert not torch.any(g[n]) and not torch.any(g32[n]), k
            continue
        assert rel_l2(g[n].cpu().numpy(), ref) <= 1e-10, k
        assert rel_l2(g32[n].cpu().numpy(), ref) <= 1e-3, k


def test_summed_gradients_and_unaligned_media(oracle_lib):
    w, obs = _problem(76, 40, "vti", 3, True, False)
    plan = StepPlan.for_workload(w, "f32")
    med = plan.medium_to_device(w.medium)
    J, g = _run(w, obs, "f32", plan=plan, med=med)
    total = g.clone()
    J2, out = _run(w, obs, "f32", plan=plan, med=med, grad=total, accumulate=True)
    assert J2 == J and out is total and torch.equal(total, 2.0 * g)  # g + g is exact
    off = {}
    for k, t in med.items():
        flat = torch.zeros(t.numel() + 1, device="cuda")
        flat[1:] = t.reshape(-1)
        off[k] = flat[1:].view(t.shape)
    J3, g3 = _run(w, obs, "f32", plan=plan, med=off)
    assert J3 == J and torch.equal(g3, g)
