"""The FP64 step against the oracle, bit for bit, where the sweeps' splits and
the straight-line solvers can go wrong: rows at the edges of a 32-face chunk
and of the parts a row is cut in, the shortest grids, marches of one cell, PPM's
ring on four cells; and states whose divisions and roots leave the range of
the straight-line arithmetic or meet zeros (every face is then redone with
the operators, or none is)."""
import numpy as np
import pytest

import oracle as orc
from gpluto_dev_b200 import api, ics

pytestmark = pytest.mark.gpu


def check(st, limiter="mc", rk=2, nsteps=4, first_dt=1e-4):
    hd, rmhd = st.physics == api.HD, st.physics == api.RMHD
    rs, ct = ("hllc", "uct_hll") if hd else ("hlld", "uct_hll" if rmhd else "uct_hlld")
    cfl = 0.3 if rmhd else 0.4
    # RMHD: the oracle with correctly rounded trigonometry (tests/test_gpu_rmhd.py)
    orc.set_cr_trig(rmhd)
    orc.set_rmhd_strict(rmhd)
    try:
        o = orc.Oracle(st, limiter=limiter, solver=rs, ct=ct, rk=rk, cfl=cfl)
        ohist, oerr = o.run(nsteps, first_dt)
        Vo, Uo, Bo = o.state()
    finally:
        orc.set_cr_trig(False)
        orc.set_rmhd_strict(False)
    sch = api.Scheme(physics=st.physics, limiter=limiter, riemann=rs, ct_emf=ct, gamma=st.gamma,
                     rk=rk, cfl=cfl)
    s = api.Solver.from_state(st, sch)
    _, hist, out = s.run(nsteps, first_dt)
    V, U, Bs = s.download()
    assert out.err_bits == oerr
    np.testing.assert_array_equal(hist, ohist[:-1])
    for a, b in zip([V, U, *Bs], [Vo, Uo, *Bo]):
        np.testing.assert_array_equal(a.view(np.int64), np.ascontiguousarray(b).view(np.int64))


@pytest.mark.parametrize("n", [(2, 5), (31, 9), (32, 9), (33, 9), (62, 4), (63, 4), (64, 3),
                               (95, 2), (257, 3), (3, 130), (2, 3, 4), (33, 2, 2)])
def test_row_parts_and_march_lengths(n):
    gen = ics.mhd2d_turbulence if len(n) == 2 else ics.mhd3d_turbulence
    check(gen(n=n, seed=sum(n)))
    check(ics.hd_turbulence(n=n, seed=sum(n)))


@pytest.mark.parametrize("n", [(4, 37), (32, 11), (33, 4), (5, 4, 9)])
def test_ppm_ring(n):
    gen = ics.mhd2d_turbulence if len(n) == 2 else ics.mhd3d_turbulence
    check(gen(n=n, seed=sum(n)), limiter="ppm", rk=3)
    check(ics.hd_turbulence(n=n, seed=sum(n)), limiter="ppm")


@pytest.mark.parametrize("physics", ["hd", "mhd", "rmhd"])
def test_faces_out_of_range(physics):
    """Densities of 2^-240: every face takes the operators."""
    st = {"hd": lambda: ics.hd_turbulence(n=(20, 12), seed=5),
          "mhd": lambda: ics.mhd2d_turbulence(n=(20, 12), seed=5),
          "rmhd": lambda: ics.rmhd3d_turbulence(n=(8, 10, 6), seed=5, lorentz_max=2.0)}[physics]()
    st.V[0] *= 2.0 ** -240
    st.V[-1] *= 2.0 ** -240
    st.V[4:-1] *= 2.0 ** -120
    st.Bs = [b * 2.0 ** -120 for b in st.Bs]
    check(st, nsteps=2)


@pytest.mark.parametrize("ndim", [2, 3])
def test_zeros(ndim):
    """Gas at rest without field beside a pressure jump, and a field along one
    direction: zero dividends of either sign, 0/0 in the face data's weights."""
    n = (24, 10) if ndim == 2 else (12, 10, 8)
    gen = ics.mhd2d_turbulence if ndim == 2 else ics.mhd3d_blast
    for field in (0.0, 0.7):
        st = gen(n=n, seed=3)
        st.V[:] = 0.0
        st.V[0] = 1.0
        st.V[7] = np.where(np.arange(n[0]) < n[0] // 2, 1.0, 0.1)
        st.V[4] = field
        st.Bs = [np.full_like(b, field if d == 0 else 0.0) for d, b in enumerate(st.Bs)]
        check(st, nsteps=3)


@pytest.mark.parametrize("precision", [api.FP64, api.MIXED])
@pytest.mark.parametrize("n", [(64, 48), (333, 31), (40, 36, 30)])
@pytest.mark.parametrize("physics", ["hd", "mhd"])
def test_overlapped_sweeps_match_serialized_launches(physics, n, precision):
    """MHD and mixed HD sweep all directions in one launch; profiling sweeps them in
    a launch each with events around it, which puts them in a row.  FP64 HD has a
    launch a sweep either way: there the events only undo the early launches."""
    gen = ics.hd_turbulence if physics == "hd" else \
        (ics.mhd2d_turbulence if len(n) == 2 else ics.mhd3d_turbulence)
    st = gen(n=n, seed=11)
    hd = physics == "hd"
    sch = api.Scheme(physics=st.physics, riemann="hllc" if hd else "hlld",
                     ct_emf="uct_hll" if hd else "uct_hlld", gamma=st.gamma, precision=precision)
    a, b = api.Solver.from_state(st, sch), api.Solver.from_state(st, sch)
    a.run(40, 1e-4)
    b.profile(40, 1e-4)
    for x, y in zip(a.download(), b.download()):
        np.testing.assert_array_equal(np.asarray(x), np.asarray(y))


@pytest.mark.parametrize("n, limiter", [((420, 300), "ppm"), ((500, 330), "mp5"),
                                        ((200, 20, 60), "wenoz")])
def test_x_rows_first(n, limiter):
    """Uncut rows that are the longest chains of a launch whose blocks do not all fit
    (the 2-D grids) come first, wrapped round the marches; the 3-D one does not wrap."""
    gen = ics.mhd2d_turbulence if len(n) == 2 else ics.mhd3d_turbulence
    check(gen(n=n, seed=sum(n)), limiter=limiter, nsteps=2)


@pytest.mark.parametrize("n, limiter", [((1100, 420), "ppm"), ((1100, 420), "wenoz"),
                                        ((20, 16, 12), "mp5"), ((36, 30, 44), "wenoz")])
def test_common_launch_matches_one_a_direction(n, limiter):
    """The same in FP32, where the profiled launches (one direction each, of the same
    kernel) give the bits; small 3-D grids of these forms also fix the memory split."""
    gen = ics.mhd2d_turbulence if len(n) == 2 else ics.mhd3d_turbulence
    st = gen(n=n, seed=7)
    sch = api.Scheme(physics=st.physics, limiter=limiter, gamma=st.gamma, precision=api.MIXED)
    a, b = api.Solver.from_state(st, sch), api.Solver.from_state(st, sch)
    a.run(6, 1e-4)
    b.profile(6, 1e-4)
    for x, y in zip(a.download(), b.download()):
        np.testing.assert_array_equal(np.asarray(x), np.asarray(y))
