"""Contexts on different grids side by side, as a serving process holds them: the
step kernels' shared-memory limits belong to the functions, so a context on a
shorter grid must not lower them for one on a taller grid."""
import numpy as np
import pytest

from cases import random_state, small_params, table_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("option,prec,tall,short", [(4, "f64", 300, 150), (4, "f32", 300, 200), (2, "f64", 160, 101),
                                                    (17, "f64", 300, 41), (17, "f32", 160, 41), (18, "f32", 300, 41)])
def test_a_shorter_context_leaves_a_taller_one_alone(gpu_lib, option, prec, tall, short):
    """A context stepped before and after one on a shorter grid (which is
    stepped too) equals one stepped alone, bit for bit."""
    from sparc_gb300.background import flux_sheet_background
    from sparc_gb300.solver import Solver

    def make(nz):
        p = small_params(nx=64, ny=1 if option in (17, 18) else 64, nz=nz, option=option, npmlbot=4, npmltop=4,
                         precision=prec, nsrc=4, **({"xlength": 400e8} if option == 18 else {}))
        s = Solver(p, table_for(p))
        if option == 18:
            s.set_mhd2d_background(*flux_sheet_background(p, table_for(p), z_fade_mm=-1.0))
        for k in range(p.nsrc):
            a, pml = random_state(p, seed=3 + k, scale=1e-6)
            if option == 18:
                a[1] = a[4] = 0.0
                pml = np.zeros((s.npv, p.nzpml, p.ny, p.nx))
            s.set_state(a, pml, slot=k)
        return s

    with make(tall) as one:
        one.step(3)
        want = one.state(3)[0]
    with make(tall) as a, make(short) as b:
        b.step(2)
        a.step(2)
        b.step(1)
        a.step(1)
        got = a.state(3)[0]
        b.sync()
    assert np.array_equal(got, want)
