"""The resident form of the split pair (one cooperative kernel per call, ISO and
VTI grids that fit on the chip, 16 steps or more): bitwise equal to the
two-launch form (kernel variant 5), which the oracle tests pin."""
import numpy as np
import pytest
import torch

from viscoelasticinversion_b200 import StepPlan, media
from tests.helpers import run_gpu

pytestmark = pytest.mark.gpu


def _same(a, b):
    assert np.array_equal(a[0], b[0])
    for k in a[1]:
        assert np.array_equal(a[1][k], b[1][k]), k


# one tile; one row and one column of tiles; tiles cut off at the right and the
# bottom; two groups per thread (1024 x 512); tiles inside and across the CPML;
# sources and receivers on tile edges
@pytest.mark.parametrize("nx,nz,kind,precision,nsls,fs,pml", [
    (20, 22, "iso", "f32", 3, True, 4), (16, 40, "vti", "f64", 1, False, 3), (300, 14, "vti", "f32", 2, True, 4),
    (256, 256, "iso", "f64", 3, True, 20), (300, 203, "vti", "f32", 3, True, 17), (140, 301, "iso", "f32", 0, False, 9),
    (520, 333, "vti", "f32", 3, True, 30), (1024, 512, "vti", "f32", 3, True, 40), (212, 100, "vti", "f64", 5, True, 12),
    (404, 404, "iso", "f32", 5, False, 20), (1000, 300, "iso", "f32", 4, True, 24)])
def test_resident_steps_equal_the_pair(nx, nz, kind, precision, nsls, fs, pml):
    w = media.layered(nx=nx, nz=nz, nt=70, kind=kind, seed=nx + nz, pml=pml, nrec=40, nsls=nsls, free_surface=fs)
    i, j = nx // 2 // 4 * 4, max(5, nz // 2)
    w.sources = list(w.sources) + [(i, j, 1, 0.5), (i + 1, j - 1, 2, 0.25), (nx - 5, nz - 5, 0, 1.0), (4, 5, 2, 0.1)]
    w.wavelets = np.stack([np.roll(w.wavelets[0], 5 * q) for q in range(len(w.sources))])
    w.receivers = list(w.receivers) + [(4, 4), (nx - 5, nz - 5), (i, j)]
    pair = run_gpu(w, precision, 5)
    _same(run_gpu(w, precision, 0), pair)
    # long calls, calls below the resident form's smallest, and odd divisions
    _same(run_gpu(w, precision, 0, chunks=[16, 3, 33, 1, 17]), pair)


def test_resident_form_runs_and_reports_nonfinite():
    from torch.profiler import ProfilerActivity, profile

    from viscoelasticinversion_b200 import ViError

    w = media.layered(nx=256, nz=128, nt=40, kind="vti", seed=5, pml=12, nrec=8)
    plan = StepPlan.for_workload(w, "f32")
    med, st = plan.medium_to_device(w.medium), plan.zeros_state()
    plan.step(med, st, nsteps=20)
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        plan.step(med, st, nsteps=20)
        torch.cuda.synchronize()
    names = [e.name for e in p.events()]
    assert any("k_resident" in n for n in names) and not any("k_split" in n for n in names)
    plan.status()
    st["s"][0, 60, 100] = float("nan")
    plan.step(med, st, nsteps=20)
    with pytest.raises(ViError):
        plan.status()
    plan.close()


def test_plans_taking_turns_on_a_stream_stay_resident():
    # blocks of more than 128 threads: resident unless other streams' steps are in flight
    from torch.profiler import ProfilerActivity, profile

    w = media.layered(nx=256, nz=256, nt=90, kind="iso", seed=5, pml=12, nrec=8)
    plans = [StepPlan.for_workload(w, "f64") for _ in range(3)]
    med = plans[0].medium_to_device(w.medium)
    states = [p.zeros_state() for p in plans]
    for p, s in zip(plans, states):
        p.step(med, s, nsteps=20)
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        for _ in range(3):
            for p, s in zip(plans, states):
                p.step(med, s, nsteps=20)
        torch.cuda.synchronize()
    names = [e.name for e in prof.events()]
    assert sum("k_resident" in n for n in names) >= 9 and not any("k_split" in n for n in names)
    for p in plans:
        p.status()
        p.close()


def test_resident_steps_on_several_streams():
    """Plans stepped from several streams at once give their own results."""
    works = [media.layered(nx=nx, nz=nz, nt=64, kind="vti", seed=nx, pml=10, nrec=6)
             for nx, nz in ((128, 96), (256, 160), (200, 120), (320, 100))]
    want = [run_gpu(w, "f32", 5) for w in works]
    runs = []
    for w in works:
        s = torch.cuda.Stream()
        plan = StepPlan.for_workload(w, "f32")
        med, st = plan.medium_to_device(w.medium), plan.zeros_state()
        wav = torch.as_tensor(w.wavelets, dtype=torch.float32, device="cuda")
        tr = torch.zeros(2, len(w.receivers), w.nt, device="cuda")
        runs.append((s, plan, med, st, wav, tr, w))
    torch.cuda.synchronize()
    for it in range(0, 64, 16):
        for s, plan, med, st, wav, tr, w in runs:
            plan.step(med, st, nsteps=16, it0=it, sources=w.sources, wavelets=wav, receivers=w.receivers, traces=tr,
                      stream=s)
    torch.cuda.synchronize()
    for (s, plan, med, st, wav, tr, w), (tr5, st5) in zip(runs, want):
        plan.status()
        assert np.array_equal(tr.double().cpu().numpy(), tr5)
        assert np.array_equal(st["v"].double().cpu().numpy(), st5["v"])
        plan.close()
