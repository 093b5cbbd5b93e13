"""Grids with more rows than one launch dimension holds blocks of few rows (65535): the iteration kernels take
blocks of 2 to 4 rows, so these are 131070 and 262140 rows. One iteration from a random state against the oracle."""
import numpy as np
import pytest

from conftest import DT

pytestmark = pytest.mark.gpu


def _random(ps, g, o, names, dtn):
    rng = np.random.default_rng(5)
    for k in names:
        v = np.asfortranarray((0.1 * rng.standard_normal(o[k].shape)).astype(DT[dtn]))
        o[k][...] = v
        g[k].copy_(ps.from_host(v))


@pytest.mark.parametrize("ny", [131069, 131070, 140001])
def test_stokes2d(ps, oracle, ny):
    from ps_gb300.stokes import Stokes2D, Stokes2DParams, inclusion_setup
    from test_gpu_stokes2d import ALL

    nx, ly = 5, float(ny - 1)
    Mus, Rog = inclusion_setup(nx, ny, 4.0, ly)
    p = Stokes2DParams(nx, ny, 4.0, ly)
    g, o = Stokes2D(p, Mus, Rog), oracle.Stokes2D(nx, ny, p.dx, p.dy, Mus, Rog)
    g.compute_timesteps()
    o.compute_timesteps()
    _random(ps, g, o, ("Pt", "Vx", "Vy", "dVxdtau", "dVydtau"), "f64")
    g.iterate(1)
    o.step()
    for k in ALL:
        assert np.array_equal(g.host(k), o[k]), k


@pytest.mark.parametrize("dtn,ny", [("f64", 131070), ("f64", 140001), ("f32", 262140), ("f32", 262205)])
def test_stokes3d(ps, oracle, dtn, ny):
    from ps_gb300.stokes3d import Stokes3D, Stokes3DParams, inclusion_setup
    from test_gpu_stokes3d import STATE

    n, l = (4, ny, 3), (3.0, float(ny - 1), 2.0)
    Mus, Rog = inclusion_setup(*n, *l, dtype=DT[dtn])
    p = Stokes3DParams(*n, *l)
    g, o = Stokes3D(p, Mus, Rog, dtype=DT[dtn]), oracle.Stokes3D(*n, *p.h, Mus, Rog, dtype=DT[dtn])
    g.compute_timesteps()
    o.compute_timesteps()
    _random(ps, g, o, ("Pt", "Vx", "Vy", "Vz", "dVxdtau", "dVydtau", "dVzdtau"), dtn)
    g.iterate(1)
    o.step()
    for k in STATE:
        assert np.array_equal(g.host(k), o[k]), k


@pytest.mark.parametrize("ny", [131070, 140001])
def test_stokes2d_apt(ps, oracle, ny):
    from ps_gb300.stokes import Stokes2DAPT, Stokes2DAPTParams, inclusion_setup
    from test_gpu_stokes2d_apt import COEFFS, STATE

    nx, ly = 5, float(ny - 1)
    Mus, Rog = inclusion_setup(nx, ny, 4.0, ly, radius=2.0)
    p = Stokes2DAPTParams(nx, ny, 4.0, ly)
    g = Stokes2DAPT(p, Mus, Rog)
    o = oracle.Stokes2DAPT(nx, ny, p.dx, p.dy, Mus, Rog, p.Re, p.r, p.Vpdt, p.max_lxy)
    g.coefficients()
    for k in COEFFS:
        assert np.array_equal(g.host(k), o[k]), k
    _random(ps, g, o, ("Vx", "Vy", "Pt", "txx", "tyy", "txy"), "f64")
    g.iterate(1)
    o.step()
    for k in STATE:
        assert np.array_equal(g.host(k), o[k]), k


# The largest extents: one more row or plane of faces than of cells must be reached, and beyond them a call is
# refused as a whole.
@pytest.mark.parametrize("dtn,ny", [("f64", 524280), ("f64", 1048559), ("f32", 524279)])
def test_stokes2d_most_rows(ps, oracle, dtn, ny):
    from ps_gb300.stokes import Stokes2D, Stokes2DParams, inclusion_setup
    from ps_gb300 import PSError
    from test_gpu_stokes2d import ALL

    nx, ly = 4, float(ny - 1)
    Mus, Rog = inclusion_setup(nx, ny, 3.0, ly, dtype=DT[dtn])
    p = Stokes2DParams(nx, ny, 3.0, ly)
    g, o = Stokes2D(p, Mus, Rog, dtype=DT[dtn]), oracle.Stokes2D(nx, ny, p.dx, p.dy, Mus, Rog, dtype=DT[dtn])
    o.compute_timesteps()
    for k in ("dtauVx", "dtauVy", "dtauPt"):
        g[k].copy_(ps.from_host(o[k]))
    _random(ps, g, o, ("Pt", "Vx", "Vy", "dVxdtau", "dVydtau"), dtn)
    start = {k: o[k].copy(order="F") for k in ("Pt", "Vx", "Vy", "dVxdtau", "dVydtau")}
    for _ in range(2):
        o.step()
    g.iterate(2)
    for k in ALL:
        assert np.array_equal(g.host(k), o[k]), k
    if dtn == "f64":  # the solver, which makes its own pseudo-time steps
        for k, v in start.items():
            g[k].copy_(ps.from_host(v))
        with pytest.raises(PSError):  # two iterations do not reach tol
            g.solve(tol=1e-30, mode=0, max_iter=2, nout=2)
        for k in start:
            assert np.array_equal(g.host(k), o[k]), k


@pytest.mark.parametrize("dtn,ny", [("f64", 1048560), ("f32", 524280)])
def test_stokes2d_too_many_rows_is_refused_whole(ps, dtn, ny):
    from ps_gb300 import PSError
    from ps_gb300.stokes import Stokes2D, Stokes2DParams

    nx = 3
    g = Stokes2D(Stokes2DParams(nx, ny, 2.0, float(ny - 1)), np.ones((nx, ny), order="F", dtype=DT[dtn]),
                 np.ones((nx, ny), order="F", dtype=DT[dtn]), dtype=DT[dtn])
    g["Vx"].fill_(1.0)
    g["Vy"].copy_(ps.rand(nx, ny + 1, dtype=DT[dtn], seed=1))
    before = {k: g[k].clone() for k in ("Pt", "Vx", "Vy", "txx", "txy")}
    with pytest.raises(PSError, match="rows"):
        g.iterate(1)
    if dtn == "f64":
        for mode in (0, 1):
            with pytest.raises(PSError, match="rows"):
                g.solve(tol=1.0, mode=mode, max_iter=2, nout=2)
    assert all((g[k] == v).all().item() for k, v in before.items())


@pytest.mark.parametrize("dtn", ["f64", "f32"])
@pytest.mark.parametrize("n,one_launch", [((4, 3, 65535), False), ((4, 3, 65535), True), ((3, 4, 65534), False),
                                          ((4, 524280, 3), False), ((3, 524279, 3), False)])
def test_stokes3d_largest_extents(ps, oracle, dtn, n, one_launch):
    from ps_gb300.stokes3d import Stokes3D, Stokes3DParams, inclusion_setup
    from test_gpu_stokes3d import STATE

    l = tuple(float(m - 1) for m in n)
    Mus, Rog = inclusion_setup(*n, *l, dtype=DT[dtn])
    p = Stokes3DParams(*n, *l)
    g, o = Stokes3D(p, Mus, Rog, dtype=DT[dtn]), oracle.Stokes3D(*n, *p.h, Mus, Rog, dtype=DT[dtn])
    g.compute_timesteps()
    o.compute_timesteps()
    _random(ps, g, o, ("Pt", "Vx", "Vy", "Vz", "dVxdtau", "dVydtau", "dVzdtau"), dtn)
    g.iterate(3, one_launch=one_launch)
    for _ in range(3):
        o.step()
    for k in STATE:
        assert np.array_equal(g.host(k), o[k]), k
