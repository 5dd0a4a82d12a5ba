"""Magnetic steps replayed from graphs (of four steps and a rest) against the
same steps launched directly: two slots on different clocks across the steps of
the horizontal filter, which is gated on the device clock, both source kinds,
surface records, and every count of steps around the graph's; and the z solve
of these forms at the edges of its chunks against the oracle."""
import numpy as np
import pytest

from cases import gaussian_plane, small_params, small_params_2d, smooth_state, table_for

pytestmark = pytest.mark.gpu


def _params(option, prec, nz=48, **kw):
    mk = small_params_2d if option == 18 else small_params
    base = {"xlength": 400e8} if option == 18 else {"nx": 16}
    pml = min(6, nz // 4)
    return mk(**{**base, "option": option, "precision": prec, "nz": nz, "npmlbot": pml,
                 "npmltop": 0 if option == 10 else pml, "src_k": nz // 2, **kw})


def _background(p, tab):
    from sparc_gb300.background import flux_sheet_background, flux_tube_background
    return flux_sheet_background(p, tab, z_fade_mm=-1.0) if p.option == 18 else flux_tube_background(p, tab)


@pytest.mark.parametrize("lagrange", [False, True])
@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("option", [8, 10, 18])
def test_replayed_steps_equal_direct_ones(gpu_lib, option, prec, lagrange, monkeypatch):
    from sparc_gb300.solver import Solver
    p = _params(option, prec, nsrc=2)
    tab = table_for(p)
    bg = _background(p, tab)
    plane = gaussian_plane(p)
    out = []
    for direct in (False, True):
        rng = np.random.default_rng(7)
        with monkeypatch.context() as mp:
            if direct:
                mp.setenv("SPARC_NO_GRAPHS", "1")
            s = Solver(p, tab)
        with s:
            (s.set_mhd2d_background if option == 18 else s.set_mhd_background)(*bg)
            for k in range(2):
                a, pml = smooth_state(p, seed=30 + k, scale=1e-6, nf=s.nf, npv=6)
                s.set_state(a, pml, slot=k)
                if lagrange:
                    s.set_source_lagrange(rng.standard_normal((8, 1, 1)) * 1e-6 * plane[None], slot=k)
                else:
                    s.set_source_series(plane, 1e-6 * np.sin(np.arange(80.0) + k), slot=k)
            s.record_surface(8)
            for n in (1, 4, 5):
                s.step(n)
            s.slot_reset(0)                       # slot 0 runs ten steps behind slot 1
            s.set_state(*smooth_state(p, seed=40, scale=1e-6, nf=s.nf, npv=6), slot=0)
            for n in (9, 4, 9, 5, 4, 1):          # both slots pass a filter step
                s.step(n)
            assert s.time == 42
            out.append([(*s.state(k), s.records(k)) for k in range(2)])
    for x, y in zip(*out):
        for u, v in zip(x, y):
            assert np.isfinite(u).all() and np.array_equal(u, v)


@pytest.fixture(scope="module")
def oracle_mod():
    from oracle import oracle
    oracle.build()
    return oracle


@pytest.mark.parametrize("option", [8, 10, 18])
@pytest.mark.parametrize("prec,tol,rtol", [("f64", 1e-10, 1e-10), ("f32", 1e-4, 1e-3)])
@pytest.mark.parametrize("nz", [16, 19, 20, 21, 30, 41, 300])
def test_z_derivatives_at_the_edges_of_the_chunks(gpu_lib, oracle_mod, option, prec, tol, rtol, nz):
    """One step from a smooth state, state and last right-hand side, against the
    FP64 oracle: 16 and 19 levels (a second chunk that holds the end row and
    its closure), 20 (whole chunks), 21 and 41 (the end row alone in its
    chunk), 30 and 300.  FP64 1e-10; FP32 1e-4 of a field of the state, as the
    other magnetic FP32 steps, and 1e-3 of the right-hand side, as the whole-step
    kernels' (a derivative amplifies the rounding of its field by the number
    of levels per scale height, some tens)."""
    from sparc_gb300.solver import Solver
    p = _params(option, prec, nz=nz)
    tab = table_for(p)
    bg = _background(p, tab)
    a0, pml0 = smooth_state(p, seed=8, scale=1e-6, nf=8 if option == 8 else 6, npv=6)
    o = oracle_mod.Oracle(p, tab)
    with Solver(p, tab) as g:
        (g.set_mhd2d_background if option == 18 else g.set_mhd_background)(*bg)
        (o.set_mhd2d if option == 18 else o.set_mhd)(*bg)
        for s in (g, o):
            s.set_state(a0, pml0)
            s.step(1)
        ag, pg = g.state()
        rg = np.stack([g.field(g.nf + f) for f in range(g.nf)])
    ao, ro, po = o.state()
    nrm = np.linalg.norm
    for f in range(len(ao)):
        assert nrm(ag[f] - ao[f]) <= tol * nrm(ao[f]), f
    assert nrm(rg - ro) <= rtol * nrm(ro)
    assert nrm(pg - po) <= rtol * nrm(po)


@pytest.mark.parametrize("option,nx,ny", [(8, 8, 8), (10, 8, 8), (10, 4, 16), (10, 16, 4), (8, 4, 4), (18, 8, 1)])
@pytest.mark.parametrize("prec,tol", [("f64", 1e-10), ("f32", 1e-4)])
def test_grids_below_the_line_transforms(gpu_lib, oracle_mod, option, nx, ny, prec, tol):
    """Three steps of two sources on grids of 4 or 8 points a side, whose x and y
    derivatives take all fields and sources of a group per launch: each slot
    against the oracle, as the other magnetic steps."""
    from sparc_gb300.solver import Solver
    p = _params(option, prec, nz=41, nx=nx, ny=ny, nsrc=2)
    tab = table_for(p)
    bg = _background(p, tab)
    with Solver(p, tab) as g:
        (g.set_mhd2d_background if option == 18 else g.set_mhd_background)(*bg)
        want = []
        for k in range(2):
            a0, pml0 = smooth_state(p, seed=50 + k, scale=1e-6, nf=g.nf, npv=6)
            o = oracle_mod.Oracle(p, tab)
            (o.set_mhd2d if option == 18 else o.set_mhd)(*bg)
            o.set_state(a0, pml0)
            g.set_state(a0, pml0, slot=k)
            o.step(3)
            want.append(o.state()[0])
        g.step(3)
        for k in range(2):
            got = g.state(k)[0]
            for f in range(g.nf):
                assert np.linalg.norm(got[f] - want[k][f]) <= tol * np.linalg.norm(want[k][f]), (k, f)
