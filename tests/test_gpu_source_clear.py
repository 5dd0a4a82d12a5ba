"""A context whose sources are all cleared steps without forcing, on every form:
captured steps hold the source mode, so a replay after clear_source must not be
one of a step that still had the source."""
import numpy as np
import pytest

from cases import gaussian_plane, random_state, small_params, small_params_2d, smooth_state, table_for

pytestmark = pytest.mark.gpu


def _solver(option, prec):
    from sparc_gb300.background import flux_sheet_background, flux_tube_background
    from sparc_gb300.solver import Solver
    mhd = option in (8, 10, 18)
    mk = small_params_2d if option in (17, 18) else small_params
    kw = {"xlength": 400e8} if option == 18 else {}
    p = mk(option=option, precision=prec, nsrc=2, npmltop=0 if option == 10 else 6, **kw)
    tab = table_for(p)
    s = Solver(p, tab)
    if option == 18:
        s.set_mhd2d_background(*flux_sheet_background(p, tab, z_fade_mm=-1.0))
    elif mhd:
        s.set_mhd_background(*flux_tube_background(p, tab))
    a, pml = smooth_state(p, seed=5, scale=1e-6, nf=s.nf, npv=6) if mhd else random_state(p, scale=1e-6)
    for k in range(2):
        s.set_state(a, pml, slot=k)
    return s


@pytest.mark.parametrize("lagrange", [False, True])
@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("option", [2, 4, 17, 8, 10, 18])
def test_cleared_source_stops_forcing(gpu_lib, option, prec, lagrange, monkeypatch):
    """step(3), both sources cleared, step(3): the same bits from replayed and
    from directly launched steps, and not those of a run that keeps its sources;
    a source that is set again acts again.  (At the default plane: the velocity
    forms' source profile is centred on it.)"""
    out = {}
    for name in ("graphs", "direct", "kept"):
        with monkeypatch.context() as mp:
            if name == "direct":
                mp.setenv("SPARC_NO_GRAPHS", "1")
            s = _solver(option, prec)
        plane = gaussian_plane(s.p)
        planes = np.stack([plane * w for w in (1.0, 2.0, 1.5, 1.0, 0.5, 1.0, 2.0, 1.0)])

        def force():
            for k in range(2):
                if lagrange:
                    s.set_source_lagrange(planes, slot=k)
                else:
                    s.set_source_series(plane, np.ones(64), slot=k)
        with s:
            force()
            s.step(3)
            if name != "kept":
                s.clear_source(0)
                s.clear_source(1)
            s.step(3)
            cleared = s.state(1)[0]
            force()
            s.step(3)
            out[name] = cleared, s.state(1)[0]
    for q in range(2):
        assert np.array_equal(out["graphs"][q], out["direct"][q])
        assert not np.array_equal(out["graphs"][q], out["kept"][q])
    assert np.isfinite(out["graphs"][1]).all()
