"""Quotients by host-known numbers outside their fast path: kernels take them without a test per dividend, over
the whole FP32 / FP64 range of magnitudes (tiny and subnormal differences, zeros) evaluate a statement
again with the exact path, and divide by powers of two on the exponent. Each kernel from such a state against the
CPU oracle, bit for bit (values of at most 1, so that nothing overflows)."""
import numpy as np
import pytest

from conftest import DT

pytestmark = pytest.mark.gpu

EMIN = {"f32": -149, "f64": -1074}


def _spread(rng, shape, dtn):
    """Signed values whose exponents cover the type's range evenly, a tenth of them zero, in runs of up to
    three equal ones (zero differences)."""
    e = rng.integers(EMIN[dtn], 0, shape).astype(np.float64)
    e[rng.random(shape) < 0.3] = -3.0  # ordinary values between them
    v = np.ldexp(0.5 + 0.5 * rng.random(shape), e.astype(np.int64)) * rng.choice([-1.0, 1.0], shape)
    v[rng.random(shape) < 0.1] = 0.0
    same = rng.random(shape) < 0.2
    v[1:][same[1:]] = v[:-1][same[1:]]
    return np.asfortranarray(v.astype(DT[dtn]))


def _load(ps, g, o, names, rng, dtn):
    for k in names:
        v = _spread(rng, o[k].shape, dtn)
        o[k][...] = v
        g[k].copy_(ps.from_host(v))


@pytest.mark.parametrize("dtn", ["f64", "f32"])
@pytest.mark.parametrize("n,lx", [((45, 29), 10.0), ((33, 17), 16.0), ((9, 70), 0.3)])
def test_stokes2d(ps, oracle, dtn, n, lx):
    from test_gpu_stokes2d import ALL, _pair

    g, o = _pair(ps, oracle, *n, dtn, lx=lx)
    _load(ps, g, o, ("Pt", "Vx", "Vy", "dVxdtau", "dVydtau"), np.random.default_rng(n[0]), dtn)
    g.iterate(3)
    for _ in range(3):
        o.step()
    for k in ALL:
        assert np.array_equal(g.host(k), o[k]), k


@pytest.mark.parametrize("dtn", ["f64", "f32"])
@pytest.mark.parametrize("n,lx", [((21, 14, 11), 10.0), ((17, 9, 33), 16.0)])
@pytest.mark.parametrize("one_launch", [False, True])
def test_stokes3d(ps, oracle, dtn, n, lx, one_launch):
    from test_gpu_stokes3d import STATE, _pair

    g, o = _pair(ps, oracle, n, dtn, lx=lx)
    _load(ps, g, o, ("Pt", "Vx", "Vy", "Vz", "dVxdtau", "dVydtau", "dVzdtau"), np.random.default_rng(n[1]), dtn)
    g.iterate(3, one_launch=one_launch)
    for _ in range(3):
        o.step()
    for k in STATE:
        assert np.array_equal(g.host(k), o[k]), k


@pytest.mark.parametrize("dtn", ["f64", "f32"])
@pytest.mark.parametrize("h", [(40.0 / 14, 40.0 / 20, 0.37), (0.5, 1.0, 2.0)])
def test_acoustic3d(ps, oracle, dtn, h):
    n = (37, 19, 23)
    rng = np.random.default_rng(7)
    P = _spread(rng, n, dtn)
    Vs = [_spread(rng, tuple(m + (d == e) for e, m in enumerate(n)), dtn) for d in range(3)]
    dts = min(h) / 6.1
    d = [ps.from_host(a) for a in (*Vs, P)]
    ps.kernels.acoustic3d_run(*d, dts, 1.0, 1.0, *h, 4)
    for _ in range(4):
        oracle.acoustic3d_v(*Vs, P, dts, 1.0, *h)
        oracle.acoustic3d_p(P, *Vs, dts, 1.0, *h)
    for a, b in zip((*Vs, P), d):
        assert np.array_equal(ps.to_host(b), a)


@pytest.mark.parametrize("dtn", ["f64", "f32"])
@pytest.mark.parametrize("h", [(1.0 / 36, 1.0 / 18, 0.31), (0.25, 0.5, 1.0)])
@pytest.mark.parametrize("memopt", [False, True])
def test_diffusion_dividing_by_spacings(ps, oracle, dtn, h, memopt):
    n = (36, 19, 23)
    rng = np.random.default_rng(11)
    T, Ci = _spread(rng, n, dtn), _spread(rng, n, dtn)
    ref = T.copy(order="F")
    dts = min(h) ** 2 / 8.1
    oracle.diffusion3d_step(0, ref, T, Ci, None, 1.3, dts, *h)
    T2 = ps.from_host(T)
    ps.parallel(ps.kernels.diffusion3D_step, T2, ps.from_host(T), ps.from_host(Ci), 1.3, dts, *h, memopt=memopt)
    assert np.array_equal(ps.to_host(T2), ref)


def _near_underflow(rng, shape, e0):
    """Values around 2^e0, of both signs."""
    return np.asfortranarray(np.ldexp(0.5 + 0.5 * rng.random(shape), rng.integers(e0 - 6, e0 + 7, shape)) *
                             rng.choice([-1.0, 1.0], shape))


def test_stokes2d_stress_underflow(ps, oracle):
    """Viscosities and velocities whose product is about the smallest subnormal number: 2 mu e may be it where mu e
    is zero."""
    from test_gpu_stokes2d import ALL, _pair

    g, o = _pair(ps, oracle, 45, 29, "f64")
    rng = np.random.default_rng(3)
    for k, e0 in (("Mus", -500), ("Vx", -575), ("Vy", -575), ("Pt", -575)):
        v = _near_underflow(rng, o[k].shape, e0)
        o[k][...] = np.abs(v) if k == "Mus" else v
        g[k].copy_(ps.from_host(o[k]))
    g.iterate(1)
    o.step()
    assert 50 < np.count_nonzero(np.abs(o["txx"]) == 2.0 ** -1074) < o["txx"].size
    for k in ALL:
        assert np.array_equal(g.host(k), o[k]), k


def test_stokes3d_stress_underflow(ps, oracle):
    """As above in 3-D."""
    from test_gpu_stokes3d import STATE, _pair

    g, o = _pair(ps, oracle, (21, 14, 11), "f64")
    rng = np.random.default_rng(4)
    for k, e0 in (("Mus", -500), ("Vx", -575), ("Vy", -575), ("Vz", -575), ("Pt", -575)):
        v = _near_underflow(rng, o[k].shape, e0)
        o[k][...] = np.abs(v) if k == "Mus" else v
        g[k].copy_(ps.from_host(o[k]))
    g.iterate(1)
    o.step()
    assert 50 < np.count_nonzero(np.abs(o["txx"]) == 2.0 ** -1074) < o["txx"].size
    for k in STATE:
        assert np.array_equal(g.host(k), o[k]), k


# Spacings that no reciprocal pair serves (10/15 in FP32, 10/17 in FP64, found on the CPU): the kernels' variants that
# test every dividend at once, alone and beside spacings with pairs.
@pytest.mark.parametrize("dtn", ["f64", "f32"])
@pytest.mark.parametrize("n", [(45, 16), (18, 29), (16, 18)])
def test_stokes2d_without_pairs(ps, oracle, dtn, n):
    test_stokes2d(ps, oracle, dtn, n, 10.0)


@pytest.mark.parametrize("dtn", ["f64", "f32"])
@pytest.mark.parametrize("n", [(16, 18, 11), (21, 14, 16), (18, 9, 18)])
@pytest.mark.parametrize("one_launch", [False, True])
def test_stokes3d_without_pairs(ps, oracle, dtn, n, one_launch):
    test_stokes3d(ps, oracle, dtn, n, 10.0, one_launch)


@pytest.mark.parametrize("dtn", ["f64", "f32"])
@pytest.mark.parametrize("h", [(10.0 / 15, 10.0 / 17, 0.37), (0.5, 10.0 / 17, 10.0 / 15), (10.0 / 15, 1e-9, 10.0 / 17)])
def test_acoustic3d_without_pairs(ps, oracle, dtn, h):
    if min(h) > 1e-6:  # (1e-9: outside the pairs' range too; one step, so that nothing overflows)
        test_acoustic3d(ps, oracle, dtn, h)
    n = (37, 19, 23)
    rng = np.random.default_rng(8)
    P = _spread(rng, n, dtn)
    Vs = [_spread(rng, tuple(m + (d == e) for e, m in enumerate(n)), dtn) for d in range(3)]
    d = [ps.from_host(a) for a in (*Vs, P)]
    ps.parallel(ps.kernels.acoustic3D_compute_V, *d, 1e-3, 1.0, *h)
    ps.parallel(ps.kernels.acoustic3D_compute_P, d[3], *d[:3], 1e-3, 1.0, *h)
    oracle.acoustic3d_v(*Vs, P, 1e-3, 1.0, *h)
    oracle.acoustic3d_p(P, *Vs, 1e-3, 1.0, *h)
    for a, b in zip((*Vs, P), d):
        assert np.array_equal(ps.to_host(b), a)


@pytest.mark.parametrize("dtn", ["f64", "f32"])
@pytest.mark.parametrize("h", [(247.0 / 254, 110.0 / 254, 0.31), (0.25, 110.0 / 254, 247.0 / 254)])
@pytest.mark.parametrize("memopt", [False, True])
def test_diffusion_dividing_by_spacings_without_pairs(ps, oracle, dtn, h, memopt):
    test_diffusion_dividing_by_spacings(ps, oracle, dtn, h, memopt)
