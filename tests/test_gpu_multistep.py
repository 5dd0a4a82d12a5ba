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
@pytest.mark.parametrize("form,prec,lagrange", [("3d", "f32", False), ("3d", "f32", True), ("2d", "f32", True),
                                                ("3d", "f64", False), ("2d", "f64", True), ("vel", "f64", False),
                                                ("vel", "f32", True)])
def test_steps_of_one_call_equal_single_steps(gpu_lib, n, form, prec, lagrange):
    mk = small_params_2d if form == "2d" else small_params
    kw = {"option": 2} if form == "vel" else {}
    p = mk(precision=prec, nsrc=3, **kw, compute_forward=not lagrange, compute_adjoint=lagrange)
    with _build(p, lagrange) as one, _build(p, lagrange) as many:
        for s in (one, many):
            s.step(3)
            s.slot_reset(1)                     # slot 1 runs three steps behind the others
        for _ in range(n):
            one.step(1)
        many.step(n)
        for x, y in zip(_all(one), _all(many)):
            assert np.array_equal(x, y)


@pytest.fixture(scope="module")
def oracle_mod():
    from oracle import oracle
    oracle.build()
    return oracle


# levels at the edges of the chunks (3 and 5 levels a thread) and of the warps
# (96 and 160 levels), the smallest and the largest box, and both chunk rules:
# 4 x 4 and 32 x 1 modes are few (3 levels a thread), 64 x 64 many
@pytest.mark.parametrize("option,nx,ny,nz,nsteps", [
    (4, 4, 4, 16, 31), (4, 8, 4, 96, 3), (4, 8, 8, 97, 3), (4, 4, 8, 193, 2), (4, 64, 64, 150, 2), (4, 64, 64, 160, 2),
    (4, 64, 64, 161, 2), (4, 64, 64, 200, 2), (4, 8, 4, 321, 2), (4, 64, 64, 400, 1), (4, 4, 4, 1024, 1),
    (17, 64, 1, 16, 31), (17, 64, 1, 95, 3), (17, 128, 1, 300, 31), (17, 8, 1, 769, 2),
    (2, 4, 4, 17, 31), (2, 8, 4, 101, 3), (2, 64, 64, 101, 2), (2, 64, 64, 321, 1)])
@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_pencil_step_matches_oracle(gpu_lib, oracle_mod, option, nx, ny, nz, nsteps, prec):
    """The whole-step kernel on chunked pencils (FP64, and FP32 in the velocity
    form) against the FP64 oracle: FP64 <= 1e-10 relative L2 of the state and
    the PML auxiliaries, FP32 <= 2e-5 of the state, as the other step kernels."""
    if prec == "f32" and option != 2:
        pytest.skip("FP32 options 4 and 17 do not run this kernel")
    from cases import smooth_state
    from sparc_gb300.background import polytrope_table
    from sparc_gb300.solver import Solver
    pml_n = max(2, min(10, nz // 6))
    p = small_params(nx=nx, ny=ny, nz=nz, option=option, npmlbot=pml_n, npmltop=pml_n, precision=prec,
                     src_k=nz // 2)
    tab = polytrope_table(nz, z_bot_mm=-25.0 if nz > 100 else -6.0, z_top_mm=1.0)
    a0, pml0 = smooth_state(p, seed=5)
    if option == 2:
        a0[5] = 0.0
    plane = gaussian_plane(p)
    series = oracle_mod.forward_source(p, 64) * 1e3
    o = oracle_mod.Oracle(p, tab)
    with Solver(p, tab) as g:
        for s in (g, o):
            s.set_state(a0, pml0)
        g.set_source_series(plane, series)
        # the oracle's delta_width is that of its default plane whatever src_k says
        width = g.info()["delta_width"] / o.info()["delta_width"] if option != 2 else 1.0
        o.set_source(1, plane[None] * width, series)
        g.step(nsteps)
        o.step(nsteps)
        ag, pg = g.state()
        rhs = np.stack([g.field(6 + f) for f in range(6)])
    ao, so, po = o.state()
    nrm = np.linalg.norm
    tol = 1e-10 if prec == "f64" else 2e-5
    assert nrm(ag - ao) <= tol * nrm(ao)
    assert nrm(rhs - so) <= (1e-10 if prec == "f64" else 1e-3) * nrm(so)
    if prec == "f64":
        assert nrm(pg - po) <= tol * nrm(po)


# the edges of the fused FP32 step's shapes: 3 levels a thread (one and two
# warps a pencil), 5 levels (one, two and three warps), the smallest box and the largest
@pytest.mark.parametrize("option,nz", [(4, k) for k in (16, 95, 96, 97, 161, 192, 193, 321, 480)]
                         + [(17, k) for k in (16, 96, 160, 161, 320)])
def test_fused_step_shapes(gpu_lib, oracle_mod, option, nz, monkeypatch):
    """The fused FP32 step against the FP64 oracle: the same sums in another
    order than the per-stage FP32 kernels, so its error is theirs but for the
    scatter of rounding (a factor 3 allowed, and never held below 1e-6, eight
    roundings); and bit for bit the same for every number of modes per CTA."""
    from cases import smooth_state
    from sparc_gb300.background import polytrope_table
    from sparc_gb300.solver import Solver
    pml_n = max(2, min(10, nz // 6))
    p = small_params(nx=16, ny=1 if option == 17 else 8, nz=nz, option=option, npmlbot=pml_n, npmltop=pml_n,
                     precision="f32")
    tab = polytrope_table(nz, z_bot_mm=-25.0 if nz > 100 else -6.0, z_top_mm=1.0)
    a0, pml0 = smooth_state(p, seed=7)
    plane = gaussian_plane(p)
    series = oracle_mod.forward_source(p, 64) * 1e3
    o = oracle_mod.Oracle(p, tab)
    o.set_state(a0, pml0)
    o.set_source(1, plane[None], series)
    o.step(3)
    ao = o.state()[0]
    out = {}
    for env, v in [("SPARC_FP32_PER_STAGE", "1")] + [("SPARC_FUSED_MODES", m) for m in "248"]:
        with monkeypatch.context() as mp:
            mp.setenv(env, v)
            with Solver(p, tab) as g:
                g.set_state(a0, pml0)
                g.set_source_series(plane, series)
                g.step(3)
                out[v] = g.state()
    err = {v: np.linalg.norm(out[v][0] - ao) / np.linalg.norm(ao) for v in out}
    assert err["4"] <= max(3 * err["1"], 1e-6)
    for v in "28":
        assert np.array_equal(out[v][0], out["4"][0]) and np.array_equal(out[v][1], out["4"][1])


@pytest.mark.parametrize("nx,ny,nz", [(16, 16, 17), (64, 32, 41), (32, 64, 75)])
@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_kernels_of_a_batch_equal_single_sources(gpu_lib, nx, ny, nz, prec):
    """A small grid's snapshot and accumulation transform all sources, and three
    fields, per launch: the kernels of each slot of a batch are bit for bit those
    of the same source run alone (batches of 3, and of 9: a full group and a rest)."""
    from sparc_gb300.solver import Solver
    def run(nsrc, first):
        fwd = small_params(nx=nx, ny=ny, nz=nz, npmlbot=4, npmltop=4, precision=prec, nsrc=nsrc)
        adj = small_params(nx=nx, ny=ny, nz=nz, npmlbot=4, npmltop=4, precision=prec, nsrc=nsrc, compute_forward=False,
                           compute_adjoint=True)
        with Solver(fwd, table_for(fwd)) as f, Solver(adj, table_for(adj)) as a:
            for k in range(nsrc):
                f.set_state(*random_state(fwd, seed=20 + first + k), slot=k)
                a.set_state(*random_state(adj, seed=40 + first + k), slot=k)
            for _ in range(2):
                f.step(1)
                a.step(1)
                f.snapshot(0, 1)
                a.kernel_accumulate(f, 0)
            return [a.kernels(k) for k in range(nsrc)]
    alone = [run(1, k)[0] for k in range(9)]
    for nsrc in (3, 9):
        for k, got in enumerate(run(nsrc, 0)):
            for x, y in zip(got, alone[k]):
                assert np.array_equal(x, y)
