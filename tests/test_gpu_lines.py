"""The line transforms at every size they cover (16 to 1024 points, along x and
along y): spectral derivatives of the FP64 primitives and a magnetic step
against torch.fft / the oracle, and the physical -> spectral -> physical round
trip of the state in both precisions, on rows and planes whose counts leave the
last CTA partly empty."""
import numpy as np
import pytest

from cases import small_params, small_params_2d, table_for

pytestmark = pytest.mark.gpu

SIZES = [16, 32, 64, 128, 256, 512, 1024]


def _params(nx, ny, nz, **kw):
    mk = small_params_2d if ny == 1 else small_params
    return mk(nx=nx, ny=ny, nz=nz, npmlbot=4, npmltop=4, **kw)


@pytest.mark.parametrize("nx,ny,nz", [(n, 4, 17) for n in SIZES] + [(8, n, 17) for n in SIZES] + [(1024, 32, 16)])
def test_derivatives_match_fft(gpu_lib, nx, ny, nz):
    """d/dx and d/dy of FP64 noise within 1e-12 relative L2 of numpy's FFT with
    the same multipliers (rounding of n log n sums is 1e-15)."""
    from sparc_gb300.solver import Solver
    p = _params(nx, ny, nz)
    v = np.random.default_rng(3).standard_normal((nz, ny, nx))
    with Solver(p, table_for(p)) as s:
        dx, dy = s.ddx(v), s.ddy(v)
        _, pt = s.tables()
    kx, ky = pt[0].reshape(ny, -1), pt[1].reshape(ny, -1)
    f = np.fft.rfft2(v)
    nrm = np.linalg.norm
    for d, k in ((dx, kx), (dy, ky)):
        want = np.fft.irfft2(1j * k * f, s=(ny, nx))
        assert nrm(d - want) <= 1e-12 * nrm(want)


@pytest.mark.parametrize("prec,tol", [("f64", 1e-14), ("f32", 1e-6)])
@pytest.mark.parametrize("nx,ny,nz", [(n, 1, 17) for n in SIZES] + [(16, n, 17) for n in SIZES[:-1]] + [(512, 512, 16)])
def test_state_round_trip(gpu_lib, nx, ny, nz, prec, tol):
    """set_state then state returns the fields: forward and inverse transforms of
    every size, to their rounding (about 4 log2(n) units: 1e-14 FP64, 1e-6 FP32)."""
    from sparc_gb300.solver import Solver
    p = _params(nx, ny, nz, precision=prec)
    a = np.random.default_rng(4).standard_normal((6, nz, ny, nx))
    with Solver(p, table_for(p)) as s:
        s.set_state(a)
        b, _ = s.state()
    assert np.linalg.norm(b - a) <= tol * np.linalg.norm(a)


@pytest.fixture(scope="module")
def oracle_mod():
    from oracle import oracle
    oracle.build()
    return oracle


@pytest.mark.parametrize("option,nx,ny", [(10, 16, 32), (10, 128, 16), (10, 32, 128), (8, 128, 32), (18, 128, 1),
                                          (18, 512, 1), (18, 1024, 1), (10, 512, 16), (10, 16, 512)])
@pytest.mark.parametrize("prec,tol", [("f64", 1e-10), ("f32", 1e-4)])
def test_magnetic_step_matches_oracle(gpu_lib, oracle_mod, option, nx, ny, prec, tol):
    """One step of the magnetic forms (derivatives, damping and horizontal filter
    through the line transforms; step 0 takes the filter in 3-D) from a smooth
    state: FP64 <= 1e-10, FP32 <= 1e-4 relative L2 per field, the tolerances of the
    flux tube against the oracle."""
    from cases import smooth_state
    from sparc_gb300.background import flux_sheet_background, flux_tube_background
    from sparc_gb300.solver import Solver
    nz = 40
    p = _params(nx, ny, nz, option=option, precision=prec, xlength=200e8 if ny == 1 else 50e8)
    tab = table_for(p)
    bg = flux_sheet_background(p, tab, z_fade_mm=-1.0) if option == 18 else flux_tube_background(p, tab)
    a0, pml0 = smooth_state(p, seed=8, nf=8 if option == 8 else 6, npv=6)
    a0, pml0 = a0 * 1e-3, pml0 * 1e-3
    o = oracle_mod.Oracle(p, tab)
    with Solver(p, tab) as g:
        (g.set_mhd2d_background if option == 18 else g.set_mhd_background)(*bg)
        (o.set_mhd2d if option == 18 else o.set_mhd)(*bg)
        for s in (g, o):
            s.set_state(a0, pml0)
            s.step(1)
        ag, _ = g.state()
    ao, _, _ = o.state()
    for f in range(len(ao)):
        assert np.linalg.norm(ag[f] - ao[f]) <= tol * np.linalg.norm(ao[f]), f


@pytest.mark.parametrize("nx,nz", [(8, 17), (16, 24), (64, 17), (64, 41), (256, 33), (256, 100), (32, 300), (16, 720)])
def test_fp32_sheet_step_matches_oracle(gpu_lib, oracle_mod, nx, nz):
    """One FP32 step of option 18, whose rows and z derivatives have kernels of
    their own: rows of 64 and 256 points and other sizes, odd row counts, chunks
    of the z solve that are empty (nz = 17), uneven and whole, and boxes above
    its limit (720): <= 1e-4 relative L2 per field, as the flux tube's."""
    from cases import smooth_state
    from sparc_gb300.background import flux_sheet_background
    from sparc_gb300.solver import Solver
    p = _params(nx, 1, nz, option=18, precision="f32", xlength=200e8)
    tab = table_for(p)
    bg = flux_sheet_background(p, tab, z_fade_mm=-1.0)
    a0, pml0 = smooth_state(p, seed=8, npv=6)
    a0, pml0 = a0 * 1e-3, pml0 * 1e-3
    o = oracle_mod.Oracle(p, tab)
    with Solver(p, tab) as g:
        g.set_mhd2d_background(*bg)
        o.set_mhd2d(*bg)
        for s in (g, o):
            s.set_state(a0, pml0)
            s.step(1)
        ag, _ = g.state()
    ao, _, _ = o.state()
    for f in range(len(ao)):
        assert np.linalg.norm(ag[f] - ao[f]) <= 1e-4 * np.linalg.norm(ao[f]), f


@pytest.mark.parametrize("nx", [32, 64])
def test_fp32_sheet_filter_follows_the_slots(gpu_lib, nx):
    """Option 18, FP32, two slots on different clocks through the horizontal
    filter's steps: 40 steps of one call equal 40 calls, bit for bit, and a slot
    equals the same slot run alone."""
    from cases import smooth_state
    from sparc_gb300.background import flux_sheet_background
    from sparc_gb300.solver import Solver
    out = []
    for nsrc, calls in ((2, 40), (2, 1), (1, 1)):
        p = _params(nx, 1, 41, option=18, precision="f32", xlength=400e8, nsrc=nsrc)
        tab = table_for(p)
        a0, pml0 = smooth_state(p, seed=9, npv=6)
        with Solver(p, tab) as g:
            g.set_mhd2d_background(*flux_sheet_background(p, tab, z_fade_mm=-1.0))
            for k in range(nsrc):
                g.set_state(a0 * 1e-3, pml0 * 1e-3, slot=k)
            if nsrc == 2:
                g.step(7)
                g.slot_reset(0)
                g.set_state(a0 * 1e-3, pml0 * 1e-3, slot=0)
            for _ in range(calls):
                g.step(40 // calls)
            out.append(g.state(0))
    for b in out[1:]:
        assert np.array_equal(out[0][0], b[0]) and np.array_equal(out[0][1], b[1])
