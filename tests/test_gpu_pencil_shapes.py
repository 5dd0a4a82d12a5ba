"""FP64 boxes of few levels: two or four of their pencils share a warp (a quarter
of a warp holds 24 to 56 levels, a half 48 to 112), and on grids with many modes
the shortest run the per-stage kernels."""
import numpy as np
import pytest

from cases import gaussian_plane, small_params, table_for

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def oracle_mod():
    from oracle import oracle
    oracle.build()
    return oracle


# the smallest box, both sides of every chunk length of a quarter (24, 32, 40, 48,
# 56: 3 to 7 levels a thread) and of half a warp (48, 64, 80, 96, 112), the first box of
# a whole warp (113), few modes (4 x 4), modes that leave the last CTA partly
# empty (1024 x 4: 2052), and both sides of the line to the per-stage kernels
@pytest.mark.parametrize("option", [4, 2])
@pytest.mark.parametrize("nx,ny,nz", [(64, 64, k) for k in (16, 24, 25, 32, 33, 40, 41, 48, 49, 56, 57, 64, 65, 80, 81, 96, 97, 112, 113)]
                         + [(4, 4, k) for k in (16, 24, 25, 48, 49)]
                         + [(1024, 4, 48), (1024, 4, 100), (1024, 4, 17), (256, 256, 20), (256, 256, 21), (512, 512, 41)])
def test_short_boxes_match_the_oracle(gpu_lib, oracle_mod, option, nx, ny, nz):
    """Two steps with a source against the FP64 oracle, as the other FP64 step
    kernels: <= 1e-10 relative L2 of the state, the PML auxiliaries and the last
    right-hand side (one step on the largest grid)."""
    from cases import smooth_state
    from sparc_gb300.solver import Solver
    pml_n = min(6, nz // 4)
    p = small_params(nx=nx, ny=ny, nz=nz, option=option, npmlbot=pml_n, npmltop=pml_n)
    tab = table_for(p)
    a0, pml0 = smooth_state(p, seed=5)
    if option == 2:
        a0[5] = 0.0
    plane = gaussian_plane(p)
    series = oracle_mod.forward_source(p, 64) * 1e3
    n = 1 if nx * ny > 65536 else 2
    o = oracle_mod.Oracle(p, tab)
    with Solver(p, tab) as g:
        for s in (g, o):
            s.set_state(a0, pml0)
        g.set_source_series(plane, series)
        o.set_source(1, plane[None], series)
        g.step(n)
        o.step(n)
        ag, pg = g.state()
        rhs = np.stack([g.field(6 + f) for f in range(6)])
    ao, so, po = o.state()
    for got, want in ((ag, ao), (rhs, so), (pg, po)):
        assert np.linalg.norm(got - want) <= 1e-10 * np.linalg.norm(want)


@pytest.mark.parametrize("option", [4, 2])
@pytest.mark.parametrize("nz", [20, 41, 75, 101, 150])
def test_short_boxes_do_not_depend_on_the_batch(gpu_lib, option, nz):
    """A slot of a batch of three, reset while the others run, equals the same
    run alone, bit for bit, and n steps of a call n calls of one step (launches of
    16, 8 or 4 steps, by the size of the batch)."""
    from cases import random_state
    from sparc_gb300.solver import Solver
    def run(nsrc, calls):
        p = small_params(nx=64, ny=64, nz=nz, option=option, nsrc=nsrc, npmlbot=min(6, nz // 4), npmltop=min(6, nz // 4))
        with Solver(p, table_for(p)) as s:
            if nsrc > 1:
                for k in range(nsrc):
                    s.set_state(*random_state(p, seed=k), slot=k)
                s.step(5)
                s.slot_reset(1)
            s.set_state(*random_state(p, seed=9), slot=nsrc // 2)
            for _ in range(calls):
                s.step(32 // calls)
            return s.state(nsrc // 2)
    alone = run(1, 1)
    for nsrc, calls in ((3, 1), (1, 32)):
        got = run(nsrc, calls)
        assert np.array_equal(got[0], alone[0]) and np.array_equal(got[1], alone[1])
