"""Which grids step in the resident form: told by the shadow of the five planes
that the plan then holds."""
import pytest

from viscoelasticinversion_b200 import StepPlan, media

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz,kind,precision,nsls,fs,pml,resident", [
    (20, 22, "iso", "f32", 3, True, 4, True), (16, 40, "vti", "f64", 1, False, 3, True),
    (300, 14, "vti", "f32", 2, True, 4, True), (256, 256, "iso", "f64", 3, True, 20, True),
    (300, 203, "vti", "f32", 3, True, 17, True), (140, 301, "iso", "f32", 0, False, 9, True),
    (520, 333, "vti", "f32", 3, True, 30, True), (212, 100, "vti", "f64", 5, True, 12, True),
    (404, 404, "iso", "f32", 5, False, 20, True), (512, 512, "vti", "f32", 3, True, 20, True),
    (1024, 512, "vti", "f32", 3, True, 40, False),  # more than 2048 cells an SM
    (256, 256, "tti", "f32", 3, True, 20, False), (301, 203, "vti", "f32", 3, True, 17, False),
    (256, 256, "vti", "f32c", 3, True, 20, False)])
def test_resident_form_is_the_one_that_runs(nx, nz, kind, precision, nsls, fs, pml, resident):
    w = media.layered(nx=nx, nz=nz, nt=20, kind=kind, seed=1, pml=pml, nrec=4, nsls=nsls, free_surface=fs)
    shadow = 5 * nx * nz * 2 * (8 if precision == "f64" else 4)
    held = {}
    for steps in (15, 16):  # one step short of the smallest resident call
        plan = StepPlan.for_workload(w, precision)
        plan.step(plan.medium_to_device(w.medium), plan.zeros_state(), nsteps=steps)
        plan.status()
        assert plan.last_kernel() == "split"
        held[steps] = plan.workspace_bytes()
        plan.close()
    extra = held[16] - held[15]
    # (the tile lists of the two forms differ by a few bytes)
    assert abs(extra - (shadow if resident else 0)) < 64 * 1024 and (not resident or extra > 0.5 * shadow)
