"""Grids whose rows are no multiple of 4 cells, and planes off a 16-byte
boundary, run the split pair on padded copies (from 8192 cells up): against
the FP64 oracle, the usual parity bars (FP32 1e-5, FP64 1e-10)."""
import numpy as np
import pytest
import torch

from viscoelasticinversion_b200 import StepPlan, media
from tests.helpers import compare, run_gpu

pytestmark = pytest.mark.gpu

TOL = {"f32": 1e-5, "f64": 1e-10}


# row remainders 1, 2, 3; a last group of 1 to 3 cells, a tile edge on and
# next to the last cell (136 = 2 * 64 + 8); each medium, surface and not
@pytest.mark.parametrize("nx,nz,kind,nsls,fs", [
    (137, 96, "iso", 3, True), (138, 71, "vti", 3, True), (139, 101, "tti", 3, True),
    (201, 77, "tti", 2, False), (135, 90, "vti", 0, False), (263, 45, "tti", 5, True),
    (131, 64, "tti", 1, True), (91, 91, "iso", 1, True)])
@pytest.mark.parametrize("precision", ["f32", "f64"])
def test_odd_rows_match_oracle(oracle_lib, nx, nz, kind, nsls, fs, precision):
    w = media.layered(nx=nx, nz=nz, nt=121, kind=kind, seed=nx, pml=11, nrec=9, nsls=nsls, free_surface=fs)
    w.sources = list(w.sources) + [(nx - 5, nz // 2, 1, 0.5), (nx - 6, nz // 2, 2, 0.25), (nx - 5, nz // 3, 0, 1.0)]
    w.wavelets = np.repeat(w.wavelets, 4, axis=0)
    w.receivers = list(w.receivers) + [(nx - 5, nz // 2)]
    tr_ref, st_ref = oracle_lib.run(w, precision="f64")
    info = {}
    tr, st = run_gpu(w, precision, 0, info=info)
    assert info["kernel"] == "split"
    err = compare(tr, st, tr_ref, st_ref, w.nsls)
    assert max(err.values()) < TOL[precision], err
    # any division of the steps over calls gives the same bits
    tr2, st2 = run_gpu(w, precision, 0, chunks=[1, 2, 57, 60, 1])
    assert np.array_equal(tr, tr2)
    for k in st:
        assert np.array_equal(st[k], st2[k]), k


def test_cells_outside_the_update_region_stay():
    """Only the updated cells and the stress images are written."""
    nx, nz = 203, 66
    w = media.layered(nx=nx, nz=nz, nt=8, kind="tti", seed=1, pml=10, nrec=4, free_surface=False)
    plan = StepPlan.for_workload(w, "f32")
    med = plan.medium_to_device(w.medium)
    g = torch.Generator().manual_seed(0)
    st = {k: 1e-3 * torch.randn(t.shape, generator=g).cuda() for k, t in plan.zeros_state().items()}
    before = {k: t.clone() for k, t in st.items()}
    plan.step(med, st, nsteps=3)
    assert plan.last_kernel() == "split"
    for k, t in st.items():
        edge = torch.ones(nz, nx, dtype=torch.bool, device="cuda")
        edge[4:-4, 4:-4] = False
        assert torch.equal(t[..., edge], before[k][..., edge]), k
        assert not torch.equal(t, before[k])
    plan.close()


@pytest.mark.parametrize("kind", ["vti", "tti"])
def test_unaligned_planes_give_the_aligned_bits(kind):
    w = media.layered(nx=160, nz=80, nt=40, kind=kind, seed=3, pml=10, nrec=8)
    out = []
    for shift in (0, 1):
        plan = StepPlan.for_workload(w, "f32")
        def moved(t):
            flat = torch.zeros(t.numel() + shift, device="cuda", dtype=t.dtype)
            flat[shift:] = t.reshape(-1)
            return flat[shift:].view(t.shape)
        med = {k: moved(t) for k, t in plan.medium_to_device(w.medium).items()}
        st = {k: moved(t) for k, t in plan.zeros_state().items()}
        wav = torch.as_tensor(w.wavelets, dtype=torch.float32, device="cuda")
        tr = torch.zeros(2, len(w.receivers), w.nt, device="cuda")
        plan.step(med, st, nsteps=w.nt, sources=w.sources, wavelets=wav, receivers=w.receivers, traces=tr)
        assert plan.last_kernel() == "split"
        plan.status()
        out.append((tr, st))
        plan.close()
    assert torch.equal(out[0][0], out[1][0])
    for k in out[0][1]:
        assert torch.equal(out[0][1][k], out[1][1][k]), k
