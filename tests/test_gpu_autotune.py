"""What the autotuner reports is what the context then launches."""
import pytest

from cases import random_state, small_params, small_params_2d, table_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("option,prec,nz,key,pencil", [
    (4, "f64", 20, "threads_per_cta", 8), (4, "f64", 48, "threads_per_cta", 16), (4, "f64", 75, "threads_per_cta", 32),
    (4, "f64", 150, "threads_per_cta", 64), (17, "f64", 300, "threads_per_cta", 128), (2, "f64", 200, "threads_per_cta", 96),
    (2, "f32", 75, "threads_per_cta", 32), (2, "f32", 150, "threads_per_cta", 64), (4, "f32", 48, "modes_per_cta", 1),
    (4, "f32", 400, "modes_per_cta", 1), (17, "f32", 300, "modes_per_cta", 1), (17, "f32", 400, "threads_per_cta", 1)])
def test_autotune_reports_the_launched_shape(gpu_lib, option, prec, nz, key, pencil):
    """The key names the unit of the kernel in use, and the threads per CTA of the
    whole-step kernel are those of whole pencils: 8 and 16 threads a pencil up to
    24 and 48 levels on few modes, then warps of 96 levels."""
    from sparc_gb300.solver import Solver
    mk = small_params_2d if option == 17 else small_params
    p = mk(option=option, precision=prec, nz=nz, npmlbot=4, npmltop=4)
    with Solver(p, table_for(p)) as s:
        s.set_state(*random_state(p, scale=1e-6))
        pick = s.autotune(1)
        assert list(pick) == [key, "ms_per_step"] and pick[key] % pencil == 0 and pick[key] > 0
        assert s.time in (4, 6)               # two variants or three, warm and timed
