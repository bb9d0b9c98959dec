"""A long call of resident steps runs as launches of at most 128 steps (256 with one
cell a thread): the same bits as the pair, and other streams' kernels get their
turn in between."""
import time

import numpy as np
import pytest
import torch

from viscoelasticinversion_b200 import StepPlan, media
from tests.helpers import run_gpu

pytestmark = pytest.mark.gpu


# one launch, two, a share of one step more in one of them; one and two cells a thread
@pytest.mark.parametrize("nx,nz,kind,precision,nt", [
    (256, 256, "vti", "f32", 256), (256, 256, "iso", "f64", 257), (400, 300, "iso", "f32", 257),
    (512, 512, "vti", "f32", 300), (512, 256, "iso", "f64", 129)])
def test_resident_launches_equal_the_pair(nx, nz, kind, precision, nt):
    w = media.layered(nx=nx, nz=nz, nt=nt, kind=kind, seed=nz, pml=20, nrec=30)
    a, b = run_gpu(w, precision, 0), run_gpu(w, precision, 5)
    assert np.array_equal(a[0], b[0])
    for k in a[1]:
        assert np.array_equal(a[1][k], b[1][k]), k


def test_other_streams_get_their_turn():
    w = media.layered(nx=512, nz=512, nt=10, kind="vti", seed=1, pml=20, nrec=8)
    plan = StepPlan.for_workload(w, "f32")
    med, st = plan.medium_to_device(w.medium), plan.zeros_state()
    a = torch.randn(4096, 4096, device="cuda", dtype=torch.bfloat16)
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    turns = []
    for _ in range(4):  # the first one warms up
        torch.cuda.synchronize()
        steps, product = torch.cuda.Event(), torch.cuda.Event()
        plan.step(med, st, nsteps=6000, stream=s1)  # some 45 ms
        steps.record(s1)
        time.sleep(0.002)
        with torch.cuda.stream(s2):
            a @ a  # does not fit beside the resident CTAs
        product.record(s2)
        product.synchronize()
        turns.append(not steps.query())
    torch.cuda.synchronize()
    plan.status()
    plan.close()
    assert all(turns[1:]), turns
