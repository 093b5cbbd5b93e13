"""The TMA variant of run-time compiled 3-D sweeps (ps_jit_launch_tma): read-only stencil arrays
staged plane by plane in shared memory. Its results must equal the plain launch's (one point per
thread) and the register sweep's bit for bit, on extents that are not multiples of the tile, with
short and long sweeps; arrays that break TMA's 16-byte rules fall back to the register sweep."""
import numpy as np
import pytest

import jit_kernels as K

pytestmark = pytest.mark.gpu


def _dev(ps, a):
    return ps.from_host(np.asfortranarray(a))


def _case(ps, name, n, dt, rng):
    import bench

    src = bench.JIT_FLUX_LAM.format(opt="") if name == "FLUX_LAM" else getattr(K, name)
    r = lambda *sh: _dev(ps, rng.standard_normal(sh).astype(dt))  # noqa: E731
    p = lambda *sh: _dev(ps, (rng.random(sh) + 0.5).astype(dt))  # noqa: E731
    if name == "BLEND3D":
        ins, outs, sc = [r(*n), r(*n), p(*n)], [(n[0] - 2, n[1] - 2, n[2] - 2)], (0.3,)
    elif name == "TWO3D":
        ins, outs, sc = [r(*n)], [(n[0] - 2, n[1] - 2, n[2] - 1), n], (0.7,)
    elif name == "FACES3D":
        ins, outs, sc = [r(*n), r(*n)], [n], (0.25,)
    elif name == "FLUX_LAM":
        ins, outs, sc = [r(*n), p(*n), p(*n)], [n], (1e-3, 9.0, 11.0, 13.0)
    else:
        ins, outs, sc = [r(*n), p(*n)], [n], (0.7, 1e-3, 9.0, 11.0, 13.0)
    return src, ins, outs, sc


def _run(ps, k, name, ins, outs, sc, dt, **kw):
    o = [ps.zeros(*sh, dtype=dt) for sh in outs]
    if name == "TWO3D":
        args = [o[0], o[1], ins[0], *sc]
    else:
        args = [*o, *ins, *sc]
    ps.parallel(k, *args, **kw)
    return [ps.to_host(x) for x in o]


def _used_tma(k):
    return k.tma_launches > 0


@pytest.mark.parametrize("dt", [np.float64, np.float32], ids=["f64", "f32"])
@pytest.mark.parametrize("name", ["HEAT_FLUX", "HEAT_LAP", "BLEND3D", "TWO3D", "FACES3D", "FLUX_LAM"])
def test_tma_sweep_is_bit_identical(ps, name, dt):
    rng = np.random.default_rng(41)
    for n, loops in (((40, 33, 29), (0, 3, 64)), ((128, 96, 70), (0, 16))):
        src, ins, outs, sc = _case(ps, name, n, dt, rng)
        k = ps.parallel_kernel(src)
        ref = _run(ps, k, name, ins, outs, sc, dt, memopt=False)
        for ls in loops:
            k.tma = "always"  # FP64 too (by default FP64 kernels keep the register sweep)
            got = _run(ps, k, name, ins, outs, sc, dt, memopt=True, loopsize=ls)
            for a, b in zip(got, ref):
                assert np.array_equal(a, b), (name, n, ls)
        assert _used_tma(k), name
        k.tma = False
        got = _run(ps, k, name, ins, outs, sc, dt, memopt=True)
        k.tma = True
        for a, b in zip(got, ref):
            assert np.array_equal(a, b), (name, n, "register sweep")
        before = k.tma_launches
        _run(ps, k, name, ins, outs, sc, dt, memopt=True)
        assert (k.tma_launches > before) == (dt == np.float32), "default: TMA for FP32 arrays only"


def test_tma_sweep_split_fp64_matches_the_register_sweep(ps):
    """fp64="split" (FP32-pair arithmetic on FP64 arrays): the staged sweep gives the register
    sweep's bits."""
    rng = np.random.default_rng(43)
    src, ins, outs, sc = _case(ps, "FLUX_LAM", (64, 40, 33), np.float64, rng)
    k = ps.parallel_kernel(src)
    k.tma = "always"
    got = _run(ps, k, "FLUX_LAM", ins, outs, sc, np.float64, memopt=True, fp64="split")
    assert _used_tma(k)
    k.tma = False
    ref = _run(ps, k, "FLUX_LAM", ins, outs, sc, np.float64, memopt=True, fp64="split")
    k.tma = True
    assert np.array_equal(got[0], ref[0])


def test_tma_sweep_out_of_bounds_reads_still_reported(ps):
    """A statement whose stencil reaches past an input array is reported (BoundsError), as by the
    register sweep: staging reads zeros there, the bounds check does not depend on it."""
    from ps_gb300 import PSError

    src = "@parallel function oob!(R, A)\n    @inn(R) = @d2_zi(A)\n    return\nend"
    k = ps.parallel_kernel(src)
    R, A = ps.zeros(40, 12, 12, dtype=np.float32), ps.rand(40, 12, 10, dtype=np.float32, seed=3)
    with pytest.raises(PSError, match="BoundsError"):
        ps.parallel(k, R, A, memopt=True)


def test_tma_sweep_falls_back_for_unaligned_arrays(ps):
    """An x extent whose row is not a multiple of 16 bytes (FP64 nx = 37) cannot be staged: the
    register sweep runs, with the same results."""
    rng = np.random.default_rng(47)
    src, ins, outs, sc = _case(ps, "HEAT_LAP", (37, 20, 19), np.float64, rng)
    k = ps.parallel_kernel(src + "\n")  # a fresh kernel object (the cache is keyed by source)
    k.tma = "always"
    got = _run(ps, k, "HEAT_LAP", ins, outs, sc, np.float64, memopt=True)
    ref = _run(ps, k, "HEAT_LAP", ins, outs, sc, np.float64, memopt=False)
    assert not _used_tma(k)
    assert np.array_equal(got[0], ref[0])


# reads the array it writes, beside staged ones: evaluated only where the statement runs
_ACCUMULATE = """@parallel function accumulate!(A, S, B, c)
    @inn(A) = @inn(A) + c*(@d2_xi(B) + @d2_yi(B) + @d2_zi(B))
    @all(S) = @all(S) * c - @all(B)
    return
end"""


@pytest.mark.parametrize("n", [(4, 3, 3), (36, 17, 4), (128, 8, 300), (132, 9, 5), (260, 31, 67)])
def test_tma_sweep_ragged_tiles_and_written_arrays(ps, n):
    """FP32 tiles of 128 x 8 cells, two rows per thread: extents one cell above and below them, thin arrays, sweeps of
    one and several chunks (the default length and given ones), against one point per thread."""
    rng = np.random.default_rng(n[0])
    A, S, B = (rng.standard_normal(n).astype(np.float32) for _ in range(3))
    k = ps.parallel_kernel(_ACCUMULATE)

    def run(**kw):
        a, s = _dev(ps, A), _dev(ps, S)
        ps.parallel(k, a, s, _dev(ps, B), 0.3, **kw)
        return ps.to_host(a), ps.to_host(s)
    ref = run(memopt=False)
    before = k.tma_launches
    for kw in ({}, {"loopsize": 1}, {"loopsize": 7}):
        for x, y in zip(run(**kw), ref):
            assert np.array_equal(x, y), (n, kw)
    assert k.tma_launches == before + 3


@pytest.mark.parametrize("short", [0, 1, 2])
def test_tma_sweep_reports_a_stencil_that_leaves_an_array(ps, short):
    """One array is shorter along one dimension than the cells that read it."""
    from ps_gb300._lib import PSError

    n = [132, 20, 40]
    m = list(n)
    m[short] -= 4 if short == 0 else 1
    k = ps.parallel_kernel(_ACCUMULATE)
    a = [ps.zeros(*n, dtype=np.float32), ps.zeros(*n, dtype=np.float32), ps.zeros(*m, dtype=np.float32)]
    with pytest.raises(PSError, match="ps_jit_launch_tma.*BoundsError"):
        ps.parallel(k, *a, 0.3)


def test_tma_sweep_split_fp64_range_is_that_of_the_cells_that_run(ps):
    """Values outside the pairs' range in cells that no running statement reads (the faces of an array read as
    @inn only) are no error; in a cell that runs they are."""
    from ps_gb300 import PSError

    n = (64, 40, 33)
    src, ins, outs, sc = _case(ps, "FLUX_LAM", n, np.float64, np.random.default_rng(44))
    k = ps.parallel_kernel(src)
    args = dict(memopt=True, fp64="split")
    Ci = ps.to_host(ins[1])  # T2, T, Ci, lam
    ref = _run(ps, k, "FLUX_LAM", ins, outs, sc, np.float64, **args)
    Ci[[0, -1]], Ci[:, [0, -1]], Ci[:, :, [0, -1]] = 1e300, -1e300, np.inf
    k.tma = "always"
    before = k.tma_launches
    got = _run(ps, k, "FLUX_LAM", [ins[0], _dev(ps, Ci), ins[2]], outs, sc, np.float64, **args)
    assert k.tma_launches == before + 1
    assert np.array_equal(got[0], ref[0])
    Ci[20, 20, 20] = 1e300
    with pytest.raises(PSError):
        _run(ps, k, "FLUX_LAM", [ins[0], _dev(ps, Ci), ins[2]], outs, sc, np.float64, **args)
    k.tma = True


def _quotients(d, own):
    """A stencil statement with d divisions; own: added to the array it writes, beside a second one in place."""
    terms = ["@d2_xi(B)/h", "c/@inn(B)", "@d2_yi(B)/(h*c)", "@d2_zi(B)/c"]
    rhs = " + ".join(terms[:d] + [t.split("/")[0] if t[0] == "@" else "c*@inn(B)" for t in terms[d:]])
    more = "@inn(A) + " if own else ""
    second = "    @all(S) = @all(S)*c - @all(B)\n" if own else ""
    return (f"@parallel function quot{d}!(A, S, B, c, h)\n    @inn(A) = {more}{rhs}\n{second}"
            + ("" if own else "    @all(S) = @all(B)\n") + "    return\nend")


@pytest.mark.parametrize("n", [(128, 10, 9), (384, 8, 5), (132, 9, 7), (36, 17, 5), (32, 24, 6), (4, 64, 9)])
@pytest.mark.parametrize("d", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("own", [False, True])
def test_tma_sweep_forms_by_divisions_and_columns(ps, d, own, n):
    """All cells of a block, the cells that run, or point by point, by the divisions of the body and the columns
    outside the arrays (where divisors are zero): the same results as one point per thread."""
    rng = np.random.default_rng(d)
    A, S, B = ((0.5 + rng.random(n)).astype(np.float32) for _ in range(3))
    B[0] = B[:, -1] = 0.0  # divisors on the faces, which no statement reads as such
    k = ps.parallel_kernel(_quotients(d, own))

    def run(**kw):
        a, s = _dev(ps, A), _dev(ps, S)
        ps.parallel(k, a, s, _dev(ps, B), 0.7, 0.3, **kw)
        return ps.to_host(a), ps.to_host(s)
    before = k.tma_launches
    got = run()
    assert k.tma_launches == before + 1
    for x, y in zip(got, run(memopt=False)):
        assert np.array_equal(x, y)
    key = (3, "float", True, False, "tma")
    assert k._layouts[key]["flat"] == (d <= 2)
    form = "" if d > 2 else "points" if own and n[0] <= 32 else "cells" if d < 2 and n[0] <= 32 or d == 1 and n[0] % 128 else ""
    if form:  # (one kernel object serves all sizes)
        assert key + (form,) in k._handles


def test_tma_sweep_of_planes_beyond_32_bit_indices(ps):
    """Eight planes of more than 2^31 elements: staged by TMA all the same, point by point."""
    import torch

    n = (16384, 16400, 4)
    k = ps.parallel_kernel("@parallel function big!(A, B, c)\n    @inn(A) = c*@d2_xi(B) + @d2_zi(B)\n    return\nend")
    B = ps.rand(*n, dtype=np.float32, seed=3)
    A, A2 = ps.zeros(*n, dtype=np.float32), ps.zeros(*n, dtype=np.float32)
    ps.parallel(k, A, B, 0.3)
    assert k.tma_launches == 1 and (3, "float", True, False, "tma", "points") in k._handles
    ps.parallel(k, A2, B, 0.3, memopt=False)
    assert torch.equal(A, A2) and A.any().item()


def _captured(f, outs):
    """The results of f in a graph's replay and of a launch by itself (a tensor's former contents put back before each)."""
    import torch

    start = [x.clone() for x in outs]
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=torch.cuda.Stream()):
        f()
    got = []
    for run in (graph.replay, f):
        for x, s in zip(outs, start):
            x.copy_(s)
        run()
        torch.cuda.synchronize()
        got.append([x.cpu() for x in outs])
    return zip(*got)


@pytest.mark.parametrize("d", [0, 1, 3])
@pytest.mark.parametrize("warm,n", [(128, 128), (128, 16), (16, 128), (37, 128), (132, 16), (37, 132)])
def test_tma_sweep_captured_after_a_launch_of_another_size(ps, d, warm, n):
    """A launch under capture cannot compile the form its size would take: it takes one that is there."""
    import torch

    k = ps.parallel_kernel(_quotients(d, True))
    size = {m: [(torch.rand(30, 40, m) + 0.5).cuda().permute(2, 1, 0) for _ in range(2)] for m in (warm, n)}
    S = {m: torch.zeros_like(a[0]) for m, a in size.items()}
    run = lambda m: ps.parallel_async(k, size[m][0], S[m], size[m][1], 0.7, 0.3)  # noqa: E731
    run(warm)
    for x, y in _captured(lambda: run(n), [size[n][0], S[n]]):
        assert torch.equal(x, y)
