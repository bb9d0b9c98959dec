"""Odd rows and short columns: grids around the 2048 cells from which the padded
copies run (the fused kernel below), down to an update region of two columns or
two rows, and CPML strips that meet in one 4-cell group; against the FP64 oracle
at the usual parity bars (FP32 1e-5, FP64 1e-10)."""
import numpy as np
import pytest

from viscoelasticinversion_b200 import StepPlan, ViError, media
from tests.helpers import compare, run_gpu

pytestmark = pytest.mark.gpu

TOL = {"f32": 1e-5, "f64": 1e-10}


@pytest.mark.parametrize("nx,nz,pml,kernel", [
    (47, 44, 6, "split"), (47, 43, 6, "fused"), (10, 205, 5, "split"), (10, 204, 5, "fused"), (11, 200, 4, "split"),
    (13, 160, 0, "split"), (301, 10, 3, "split"), (71, 39, 9, "split"), (201, 10, 3, "fused")])
@pytest.mark.parametrize("kind,nsls,fs", [("iso", 3, True), ("vti", 1, False), ("tti", 3, True), ("tti", 2, False)])
@pytest.mark.parametrize("precision", ["f32", "f64"])
def test_narrow_odd_grids_match_oracle(oracle_lib, nx, nz, pml, kernel, kind, nsls, fs, precision):
    w = media.layered(nx=nx, nz=nz, nt=60, kind=kind, seed=nx, pml=pml, nrec=2, nlayers=3, f0=30.0, nsls=nsls,
                      free_surface=fs)
    i, j = nx // 2, nz // 2
    w.sources = [(i, j, 0, 1.0), (nx - 5, nz - 5, 1, 0.5), (4, j, 2, 0.25)]
    w.wavelets = np.repeat(w.wavelets, 3, axis=0)
    w.receivers = [(4, 4), (i, j), (nx - 5, nz - 5)]
    tr_ref, st_ref = oracle_lib.run(w, precision="f64")
    info = {}
    if fs and nz - 8 < 5:  # a surface needs five updated rows under it
        plan = StepPlan.for_workload(w, precision)
        with pytest.raises(ViError, match="at least 5 rows"):
            plan.step(plan.medium_to_device(w.medium), plan.zeros_state(), nsteps=2)
        plan.close()
        return
    tr, st = run_gpu(w, precision, 0, info=info)
    assert info["kernel"].startswith(kernel)
    err = compare(tr, st, tr_ref, st_ref, w.nsls)
    assert max(err.values()) < TOL[precision], err
