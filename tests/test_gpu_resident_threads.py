"""Plans of different grids stepped in the resident form from several host
threads at once: every launch gets the shared memory its own tiling needs."""
import threading

import numpy as np
import pytest
import torch

from viscoelasticinversion_b200 import StepPlan, media
from tests.helpers import run_gpu

pytestmark = pytest.mark.gpu

STEPS, CALLS = 16, 400


def test_resident_steps_from_several_threads():
    # one kernel (VTI FP32, one cell a thread) at three sizes of shared memory
    # above the 48 KB that need no opt-in; every round starts on an idle GPU, so
    # no plan sees another's steps in flight
    works = [media.layered(nx=nx, nz=nz, nt=STEPS, kind="vti", seed=nx, pml=8, nrec=4)
             for nx, nz in ((256, 256), (320, 320), (360, 360))]
    want = [run_gpu(w, "f32", 5) for w in works]
    got, failed = [None] * len(works), []
    start = threading.Barrier(len(works))

    def work(k):
        w = works[k]
        try:
            s = torch.cuda.Stream()
            with torch.cuda.stream(s):
                plan = StepPlan.for_workload(w, "f32")
                med, st = plan.medium_to_device(w.medium), plan.zeros_state()
                wav = torch.as_tensor(w.wavelets, dtype=torch.float32, device="cuda")
                tr = torch.zeros(2, len(w.receivers), STEPS, device="cuda")
            for _ in range(CALLS):  # each call from rest
                with torch.cuda.stream(s):
                    for t in st.values():
                        t.zero_()
                plan.reset(s)
                s.synchronize()
                start.wait(timeout=60)
                plan.step(med, st, nsteps=STEPS, sources=w.sources, wavelets=wav, receivers=w.receivers, traces=tr,
                          stream=s)
            plan.status(s)
            got[k] = (tr.double().cpu().numpy(), st["v"].double().cpu().numpy())
            plan.close()
        except Exception as e:
            failed.append((w.nx, w.nz, repr(e)))
            start.abort()

    ts = [threading.Thread(target=work, args=(k,)) for k in range(len(works))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not failed, failed
    for (tr, v), (tr5, st5) in zip(got, want):
        assert np.array_equal(tr, tr5) and np.array_equal(v, st5["v"])
