"""A step that stages lists stays refused under stream capture, also when its
lists are already on the device: a graph of it would replay one call's
arguments (the resident form's pass numbers, TTI's current buffer)."""
import pytest
import torch

from viscoelasticinversion_b200 import StepPlan, ViError, media

pytestmark = pytest.mark.gpu


# resident, pair, TTI pair, padded copies, the fused kernel
@pytest.mark.parametrize("nx,nz,kind,nsteps,variant", [
    (256, 128, "vti", 20, 0), (256, 128, "vti", 4, 0), (256, 128, "tti", 20, 0), (131, 101, "iso", 20, 0),
    (256, 128, "iso", 4, 2)])
@pytest.mark.parametrize("shot", [True, False])
def test_staged_step_is_refused_under_capture(nx, nz, kind, nsteps, variant, shot):
    w = media.layered(nx=nx, nz=nz, nt=80, kind=kind, seed=5, pml=12, nrec=8)
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        plan = StepPlan.for_workload(w, "f32")
        med, a = plan.medium_to_device(w.medium), plan.zeros_state()
        wav = torch.as_tensor(w.wavelets, dtype=torch.float32, device="cuda")
        tr = torch.zeros(2, len(w.receivers), w.nt, device="cuda")
        kw = dict(sources=w.sources, wavelets=wav, receivers=w.receivers, traces=tr) if shot else {}
        plan.step(med, a, nsteps=nsteps, variant=variant, **kw)
        torch.cuda.synchronize()
        before = {k: t.clone() for k, t in a.items()}
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        g.capture_begin(capture_error_mode="thread_local")
        try:
            with pytest.raises(ViError):
                plan.step(med, a, nsteps=nsteps, variant=variant, **kw)
        finally:
            g.capture_end()
        torch.cuda.synchronize()
        assert all(torch.equal(before[k], a[k]) for k in a)
        # and the plan goes on
        plan.step(med, a, it0=nsteps, nsteps=nsteps, variant=variant, **kw)
        torch.cuda.synchronize()
        plan.status()
        plan.close()
