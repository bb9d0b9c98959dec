"""Plans and batches may be destroyed, by a garbage collector for one, while the
thread captures a stream: the capture goes on."""
import numpy as np
import pytest
import torch

from viscoelasticinversion_b200 import StepPlan, media
from viscoelasticinversion_b200.batch import ShotBatch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["thread_local", "global"])
@pytest.mark.parametrize("batch", [False, True])
def test_destroying_during_a_capture_leaves_it(mode, batch):
    w = media.layered(nx=128, nz=64, nt=20, kind="vti", seed=5, pml=12, nrec=8)
    if batch:
        obj = ShotBatch([w, w], "f32")
        obj.run()
    else:
        obj = StepPlan.for_workload(w, "f32")
        obj.step(obj.medium_to_device(w.medium), obj.zeros_state(), nsteps=20)
    st, x = torch.cuda.Stream(), torch.zeros(1024, device="cuda")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(st):
        g.capture_begin(capture_error_mode=mode)
        x.add_(1.0)
        obj.close()
        x.add_(2.0)
        g.capture_end()
    g.replay()
    torch.cuda.synchronize()
    assert np.all(x.cpu().numpy() == 3.0)
