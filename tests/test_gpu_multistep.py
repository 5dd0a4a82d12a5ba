"""Several time steps per launch.  The quiet-Sun step kernels keep a pencil on
chip over the steps of a launch: n steps in one call must give what n calls of
one step give, bit for bit -- the state, the PML auxiliaries, the last
right-hand side and the surface records -- at the step counts around the
launch's limit, for one source and for a batch whose slots run on different
clocks, and for both source kinds."""
import numpy as np
import pytest

from cases import gaussian_plane, random_state, small_params, small_params_2d, table_for

pytestmark = pytest.mark.gpu


def _build(p, lagrange):
    from sparc_gb300 import sources
    from sparc_gb300.solver import Solver
    s = Solver(p, table_for(p))
    for k in range(p.nsrc):
        a, pml = random_state(p, seed=11 + k)
        s.set_state(a, pml, slot=k)
        if lagrange:
            rng = np.random.default_rng(60 + k)
            s.set_source_lagrange(rng.standard_normal((8, p.ny, p.nx)) * 1e-4, slot=k)
        else:
            s.set_source_series(gaussian_plane(p, x0_mm=float(k)), sources.ricker_series(p, 20, delay=20.0) * 1e3, slot=k)
    s.record_surface(8)
    return s


def _all(s):
    out = []
    for k in range(s.p.nsrc):
        out += [*s.state(k), s.records(k), s.field(s.nf + 3, k), s.field(s.nf + 5, k)]
    return out


@pytest.mark.parametrize("n", [2, 15, 16, 17, 33])
@pytest.mark.parametrize("form,prec,lagrange", [("3d", "f32", False), ("3d", "f32", True), ("2d", "f32", True)])
def test_steps_of_one_call_equal_single_steps(gpu_lib, n, form, prec, lagrange):
    mk = small_params_2d if form == "2d" else small_params
    p = mk(precision=prec, nsrc=3, compute_forward=not lagrange, compute_adjoint=lagrange)
    with _build(p, lagrange) as one, _build(p, lagrange) as many:
        for s in (one, many):
            s.step(3)
            s.slot_reset(1)                     # slot 1 runs three steps behind the others
        for _ in range(n):
            one.step(1)
        many.step(n)
        for x, y in zip(_all(one), _all(many)):
            assert np.array_equal(x, y)
