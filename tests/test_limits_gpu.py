"""Geometries, sizes and values at the ends of what the entry points accept:
distant sources and detectors, a flat fan, voxels of any side, tables of any
shape, infinite unknowns, calls that fail half way -- against the FP64 oracle."""
import threading

import numpy as np
import pytest

import xrd_tomography_gb300 as xt
from xrd_tomography_gb300 import synth
from tests.test_decisions_gpu import compare
from tests.test_sizes_gpu import sized_problem, some_rays
from tests.tolerances import FAST_RTOL, max_rel_err

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    c = xt.Context(0)
    yield c
    c.close()


def full_map(p, seed, listed=100000):
    """Inputs whose every voxel is listed, or `listed` of them."""
    inp = synth.make_inputs(p, seed)
    n = p.nx * p.ny
    inp.seg = np.ones(n, np.int32)
    if n > listed:
        inp.seg[np.random.default_rng(seed).permutation(n)[listed:]] = 0
    inp.a1 = np.full(n, 2e-5, np.float32)
    inp.a2 = np.full(n, 0.02, np.float32)
    return inp


# the integer decisions of both line integrals with endpoints thousands of
# voxels away, where a float holds them to 1e-3 of a voxel, a short sample step,
# thin maps that rays graze, and a large map
@pytest.mark.parametrize("nx,ny,r_src,r_det,step,rays", [
    (100, 100, 5000.0, 120.0, 0.25, 200), (100, 100, 30000.0, 120.0, 0.25, 200), (100, 100, 1e6, 1e6, 0.25, 100),
    (60, 50, 150.0, 5000.0, 0.25, 300), (100, 100, 5000.0, 5000.0, 0.05, 100), (3, 1000, 3000.0, 600.0, 0.1, 200),
    (1024, 1024, 8000.0, 1130.0, 0.25, 8)])
def test_decisions_with_distant_endpoints(ctx, oracle_lib, nx, ny, r_src, r_det, step, rays):
    p = sized_problem(nx, ny, 360, 64, 4, 4, 0)
    p.r_src, p.r_det, p.dq_step = r_src, r_det, step
    inp = full_map(p, 31)
    compare(inp, some_rays(p, rays, 32), ctx, oracle_lib)


# a flat fan (wedge angle 0: no photon passes, every output is 0) and the
# thinnest ones
@pytest.mark.parametrize("wedge", [0.0, 1e-12, 1e-4, -0.01])
def test_flat_fan(ctx, oracle_lib, wedge):
    p = sized_problem(14, 11, 3, 21, 7, 7, 2, nwt=40)
    p.wedge_angle = wedge
    inp = synth.make_inputs(p, 41)
    rays = np.arange(p.rays)
    N, C, A = xt.forward(p, *inp.args(), ctx=ctx)
    Nr, Cr, Ar, _ = oracle_lib.forward_rays(inp, rays, want_a=True)
    got, want = [N, C, A], [Nr, Cr, np.asarray(Ar).reshape(-1)]
    S1 = synth.coherent_table(inp)
    for bilinear in (False, True):
        got += xt.forward_tables(p, inp.spectrum, inp.seg, inp.a1, inp.a2, S1, inp.S2, *inp.args()[6:],
                                 bilinear=bilinear, ctx=ctx)
        want += oracle_lib.forward_tables(inp, S1, rays, bilinear=bilinear)
    rng = np.random.default_rng(42)
    x = rng.uniform(0.0, 1.0, (p.nx * p.ny, p.nwt)).astype(np.float32)
    x[inp.seg == 0] = 0.0
    w = rng.uniform(0.0, 2.0, p.rays).astype(np.float32)
    y_ref, g_ref = oracle_lib.vox_rays(inp, rays, x=x.reshape(-1), w=w)
    op = xt.Operator(p, inp.spectrum, inp.seg, inp.a1, inp.a2, ctx=ctx)
    got += [op.forward(x.reshape(-1)), op.adjoint(w)]
    want += [y_ref, g_ref.reshape(-1)]
    op.close()
    for a, b in zip(got, want):
        assert np.asarray(a).shape == np.asarray(b).shape
        if wedge == 0.0:
            assert not np.asarray(b).any() and not np.asarray(a).any()
        else:
            assert max_rel_err(a, b) < FAST_RTOL


# the scattering angle with the source, or the detector, thousands of times
# farther from the voxels than the other: a table of 65536 bins over 12 octaves
# shows an error of 1e-9 in sin(theta/2) in two terms of a million; the angle's
# float pairs hold it to 6e-13
@pytest.mark.parametrize("r_src,r_det", [(1e5, 90.0), (1e6, 90.0), (150.0, 1e5)])
def test_scattering_angles_far_away(ctx, oracle_lib, r_src, r_det):
    p = sized_problem(60, 60, 90, 64, 12, 12, 2)
    p.col_pitch *= max(1.0, r_det / 130.0)
    p.r_src, p.r_det = r_src, r_det
    p.nq, p.na = 65536, 1
    compare(full_map(p, 51), some_rays(p, 300, 52), ctx, oracle_lib)


# voxel centres that no float holds, on rays along the grid, whose lengths are
# multiples of the sample step; and sides that a float holds
@pytest.mark.parametrize("side", [0.7, 0.3, 0.9, 0.5, 0.75])
def test_decisions_at_any_voxel_side(ctx, oracle_lib, side):
    p = sized_problem(26, 18, 4, 9, 6, 6, 1)
    p.cx, p.cy = 0.5 * side * (p.nx + 1), 0.5 * side * (p.ny + 1)   # on a voxel centre
    p.r_src, p.r_det = 64.0, 60.0
    p.col_pitch = side
    p.vox_side = side
    compare(full_map(p, 61), np.arange(p.rays), ctx, oracle_lib)


def test_calls_of_different_sizes_on_two_threads(oracle_lib):
    """Kernels whose shared memory follows the problem's size, called with a
    small and a large one by two threads, each with a context of its own: the
    calls neither fail nor change."""
    small = synth.make_inputs(sized_problem(9, 7, 3, 11, 6, 6, 1, nwt=8, nqf=32), 71)
    large = synth.make_inputs(sized_problem(12, 10, 3, 13, 120, 100, 4, nwt=64, nqf=768, mats=6), 72)
    ctxs = [xt.Context(0), xt.Context(0)]
    errors = []

    def calls(inp, c):
        p = inp.problem
        T, G = xt.ct_sinogram(p, inp.spectrum, inp.a1, inp.a2, ctx=c)
        return [T, G, *xt.forward(p, *inp.args(), ctx=c)]

    try:
        want = [[a.copy() for a in calls(inp, c)] for inp, c in zip((small, large), ctxs)]

        def work(inp, c, ref, n):
            try:
                for _ in range(n):
                    for a, b in zip(calls(inp, c), ref):
                        if not np.array_equal(a, b):
                            raise AssertionError("a call's result changed")
            except Exception as e:   # noqa: BLE001 - reported by the main thread
                errors.append(e)

        threads = [threading.Thread(target=work, args=(inp, c, ref, 400)) for inp, c, ref in zip((small, large), ctxs, want)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    finally:
        for c in ctxs:
            c.close()
    assert not errors, errors


def test_infinite_unknowns_stay_in_their_energies_windows(ctx):
    """With detector bins that take one source bin each, a ray sees its own
    energy's window alone: an infinite coefficient reaches the same rays, and an
    infinite weight the same unknowns, whether the kernels take two energies
    together or the operator holds only one."""
    def operator(e0, e1, n):
        p = sized_problem(6, 5, 3, 65, n, n, 0, nwt=24)
        p.e_src_min = p.e_det_min = e0
        p.e_src_max = p.e_det_max = e1
        # far away, for windows narrower than the q grid
        p.r_src, p.r_det, p.col_pitch, p.z0 = 10 * p.r_src, 10 * p.r_det, 10 * p.col_pitch, 10 * p.z0
        inp = full_map(p, 81)
        inp.spectrum = np.eye(n, dtype=np.float32).reshape(-1)
        return p, xt.Operator(p, inp.spectrum, inp.seg, inp.a1, inp.a2, ctx=ctx)

    both, parts = operator(40.0, 44.0, 2), [operator(40.0, 42.0, 1), operator(42.0, 44.0, 1)]
    p, op = both
    pairs = p.rays // 2
    rng = np.random.default_rng(82)
    x = rng.uniform(0.1, 1.0, (p.nx * p.ny, p.nwt)).astype(np.float32)
    reached = 0
    for k in range(p.nwt):
        xi = x.copy()
        xi[k % (p.nx * p.ny), k] = np.inf
        y = op.forward(xi.reshape(-1)).reshape(2, pairs)
        for e, (_, one) in enumerate(parts):
            want = one.forward(xi.reshape(-1))
            assert np.array_equal(np.isnan(y[e]), np.isnan(want)) and np.array_equal(np.isinf(y[e]), np.isinf(want))
            ok = np.isfinite(want)
            assert max_rel_err(y[e][ok], want[ok]) < FAST_RTOL
            reached += int((~ok).sum())
    assert reached
    partly = 0
    for r in range(0, pairs, 13):
        for e in range(2):
            w = rng.uniform(0.5, 1.0, (2, pairs)).astype(np.float32)
            w[1 - e, r], w[e, r] = 1.0, np.inf
            g = op.adjoint(w.reshape(-1))
            want = parts[e][1].adjoint(w[e])
            assert np.array_equal(np.isfinite(g), np.isfinite(want))
            ok = np.isfinite(want)
            partly += bool(0 < (~ok).sum() < ok.size)
            w[e, r] = 0.0
            if ok.any():
                assert max_rel_err(g[ok], op.adjoint(w.reshape(-1))[ok]) < FAST_RTOL
    assert partly > 10
    for _, o in (both, *parts):
        o.close()


@pytest.mark.parametrize("bilinear", [False, True])
def test_table_path_takes_any_number_of_pattern_bins(ctx, oracle_lib, bilinear):
    """The table path reads no patterns: 100 materials of 768 fine bins, more
    than a block could hold, do not concern it."""
    p = sized_problem(16, 13, 3, 21, 9, 7, 2, nqf=768, mats=100)
    inp = synth.make_inputs(p, 91)
    S1 = synth.coherent_table(inp)
    N, C = xt.forward_tables(p, inp.spectrum, inp.seg, inp.a1, inp.a2, S1, inp.S2, *inp.args()[6:],
                             bilinear=bilinear, ctx=ctx)
    Nr, Cr = oracle_lib.forward_tables(inp, S1, np.arange(p.rays), bilinear=bilinear)
    assert max_rel_err(N, Nr) < FAST_RTOL
    assert max_rel_err(C, Cr) < FAST_RTOL


@pytest.mark.parametrize("what,change", [("patterns", dict(nqf=768, mats=100)), ("matrix", dict(nwt=4096, mats=15)),
                                         ("table", dict())])
def test_tables_that_no_block_holds_are_refused(ctx, what, change):
    """As unsupported, not as a failed launch; the context goes on; an empty
    phantom needs no tables and is 0 at any size."""
    p = sized_problem(10, 8, 2, 7, 4, 4, 1, **change)
    if what == "table":
        p.nq, p.na = 257, 256
    inp = synth.make_inputs(p, 92)
    matrix = what == "matrix"
    for call in ([lambda: xt.forward(p, *inp.args(), want_amatrix=matrix, ctx=ctx),
                  lambda: xt.forward_rays(p, np.arange(3), *inp.args(), want_amatrix=matrix, ctx=ctx)]):
        with pytest.raises(xt.XrdtError) as e:
            call()
        assert e.value.status == 7
    if matrix:
        assert xt.forward(p, *inp.args(), want_amatrix=False, ctx=ctx)[0].max() > 0
    inp.seg = np.zeros_like(inp.seg)
    assert not any(a.any() for a in xt.forward(p, *inp.args(), want_amatrix=matrix, ctx=ctx) if a is not None)


def random_table(p, seed):
    """Neighbouring bins differ by a third of their value, so that a term read
    from the wrong one shows."""
    return np.random.default_rng(seed).uniform(20.0, 255.0, p.nq * p.na).astype(np.float32)


# tables of any shape: two bins, odd and unequal sides, as long as a record's word
# holds, and too large for shared memory beside the rest; nearest lookups (and the
# fine-q path's) on rough tables, where a bin is right or wrong, bilinear ones on
# smooth ones
@pytest.mark.parametrize("nq,na", [(2, 2), (37, 91), (91, 37), (300, 3), (1024, 16), (256, 250), (32768, 2)])
def test_tables_of_any_shape(ctx, oracle_lib, nq, na):
    p = sized_problem(22, 17, 3, 40, 12, 11, 2)
    p.nq, p.na = nq, na
    inp = synth.make_inputs(p, 101)
    rays = np.arange(p.rays)
    S1 = synth.coherent_table(inp)
    got = xt.forward_tables(p, inp.spectrum, inp.seg, inp.a1, inp.a2, S1, inp.S2, *inp.args()[6:], bilinear=True, ctx=ctx)
    for a, b in zip(got, oracle_lib.forward_tables(inp, S1, rays, bilinear=True)):
        assert max_rel_err(a, b) < FAST_RTOL
    inp.S2, S1 = random_table(p, 102), random_table(p, 103)
    got = xt.forward_tables(p, inp.spectrum, inp.seg, inp.a1, inp.a2, S1, inp.S2, *inp.args()[6:], ctx=ctx)
    for a, b in zip(got, oracle_lib.forward_tables(inp, S1, rays)):
        assert max_rel_err(a, b) < FAST_RTOL
    N, C, _ = xt.forward(p, *inp.args(), want_amatrix=False, ctx=ctx)
    Nr, Cr = oracle_lib.forward_rays(inp, rays)[:2]
    assert max_rel_err(N, Nr) < FAST_RTOL
    assert max_rel_err(C, Cr) < FAST_RTOL


@pytest.mark.parametrize("nq,na", [(2, 3), (37, 91), (1024, 16), (256, 250), (32768, 2)])
def test_table_bins_at_any_shape(ctx, oracle_lib, nq, na):
    p = sized_problem(40, 33, 6, 40, 12, 11, 2)
    p.nq, p.na = nq, na
    compare(synth.make_inputs(p, 104), some_rays(p, 500, 105), ctx, oracle_lib)


def test_a_call_that_fails_half_way_leaves_the_next_one_alone(ctx, monkeypatch):
    """An allocation that fails after the tables are on their way: the call
    returns when the device is through with them, so the next call, with other
    tables in the same staging buffer, computes what it does on a context of its own."""
    torch = pytest.importorskip("torch")
    one = synth.make_inputs(sized_problem(30, 28, 40, 2, 16, 12, 2), 111)
    many = synth.make_inputs(sized_problem(30, 28, 8, 300, 16, 12, 2), 112)      # more pairs: records to allocate
    other = synth.make_inputs(sized_problem(30, 28, 37, 2, 16, 16, 3), 113)
    many_out = [torch.empty(many.problem.rays, device="cuda") for _ in range(2)]
    args = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in many.args()[:6]]
    torch.cuda.synchronize()
    want = xt.forward(other.problem, *other.args(), want_amatrix=False, ctx=ctx)[:2]
    c = xt.Context(0)
    try:
        for inp in (one, other):
            xt.forward(inp.problem, *inp.args(), want_amatrix=False, ctx=c)
        for _ in range(10):
            monkeypatch.setenv("XRDT_TEST_FAIL_ALLOC", "1")
            with pytest.raises(xt.XrdtError) as e:
                xt.forward(many.problem, *args, *many.args()[6:], Nphotons=many_out[0], Cphotons=many_out[1],
                           want_amatrix=False, ctx=c)
            assert e.value.status == 6
            monkeypatch.delenv("XRDT_TEST_FAIL_ALLOC")
            got = xt.forward(other.problem, *other.args(), want_amatrix=False, ctx=c)
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
        xt.forward(many.problem, *args, *many.args()[6:], Nphotons=many_out[0], Cphotons=many_out[1],
                   want_amatrix=False, ctx=c)
        assert float(many_out[0].max()) > 0
    finally:
        c.close()


@pytest.mark.parametrize("side", [300, 1024])
def test_ct_on_rough_maps(ctx, oracle_lib, side):
    """Every cell different from the next, so that a sample's position shows: the
    chord's offsets hold it to 1e-7 voxel and the line integral to 8e-8 of itself
    wherever the chord lies.  Exponents X below 8 (in log2) round to 6e-7 of
    the transmission, the integral's error and rounding times X ln 2 are 8e-7,
    exp2 is good to 2.4e-7 and the sum of one window's term to 6e-8: 1.7e-6."""
    p = sized_problem(side, side, 7, 301, 3, 3, 0)
    p.col_pitch *= 1.3
    inp = synth.make_inputs(p, 121)
    rng = np.random.default_rng(122)
    rough = np.where(rng.uniform(size=side * side) < 0.5, 0.0, rng.uniform(1.0, 2.0, side * side))
    inp.a1 = np.zeros(side * side, np.float32)
    inp.a2 = (3.0 / side * rough).astype(np.float32)
    T, G = xt.ct_sinogram(p, inp.spectrum, inp.a1, inp.a2, ctx=ctx)
    rays = some_rays(p, 4000, 123)
    Tr, Gr = oracle_lib.ct_rays(inp, rays)
    X = -np.log2(np.maximum(Tr, 1e-300) / np.maximum(Gr, 1e-300))
    ok = (Gr > 0) & (Tr > 0)
    assert 3.0 < X[ok].max() < 8.0
    assert np.max(np.abs(T[rays][ok] / Tr[ok] - 1.0)) < 1.7e-6


@pytest.mark.parametrize("side", [256, 1024])
def test_ct_chords_that_graze_a_side(ctx, oracle_lib, side):
    """Chords that leave through a side which they cross at 1e-3 of a voxel per
    length, that length within millionths of a step of a multiple, on a map that is 0
    but for the texels about the chord's end: a sample too many or too few is 10 % of T."""
    p = sized_problem(side, side, 1, 3, 1, 1, 0)
    p.col_pitch = 1.5e-3
    inp = synth.make_inputs(p, 131)
    inp.a1 = np.zeros(side * side, np.float32)
    ray = np.array([2])   # the pixel at +1.5e-3
    for j in range(24):
        p.cx = side - 0.75e-3 * (1.0 + 0.02 * j)
        sx, sy = p.cx, p.cy - p.r_src
        dx, dy = p.cx + 1.5e-3, p.cy + p.r_det
        ex, ey = dx - sx, dy - sy
        t0, t1 = (0.0 - sy) / ey, (side - sx) / ex
        length = (t1 - t0) * np.sqrt(ex * ex + ey * ey)
        end = int(length)
        a2 = np.zeros((side, side), np.float32)   # [y, x]
        a2[end - 2:end + 3, side - 1] = 1.0
        inp.a2 = a2.reshape(-1)
        for eps in (2e-7, 5e-7, 1e-6, 2e-6, 4e-6, 1e-5):
            for sign in (-1.0, 1.0):
                p.dq_step = length / (np.rint(4.0 * length) + sign * eps)
                T, _ = xt.ct_sinogram(p, inp.spectrum, inp.a1, inp.a2, ctx=ctx)
                Tr, _ = oracle_lib.ct_rays(inp, ray)
                assert max_rel_err(T[ray], Tr) < FAST_RTOL


def test_more_samples_than_a_float_counts(ctx, oracle_lib):
    """Steps of a millionth of a voxel: more than 2^24 samples on a ray."""
    p = sized_problem(24, 24, 1, 3, 2, 2, 0, nwt=8)
    p.dq_step = 1e-6
    inp = synth.make_inputs(p, 141)
    rays = np.arange(p.rays)
    T, G = xt.ct_sinogram(p, inp.spectrum, inp.a1, inp.a2, ctx=ctx)
    Tr, Gr = oracle_lib.ct_rays(inp, rays)
    assert max_rel_err(T, Tr) < FAST_RTOL and max_rel_err(G, Gr) < FAST_RTOL
    inp.seg = np.zeros_like(inp.seg)
    inp.seg[[24 * 3 + 20, 24 * 21 + 2]] = 1   # walks of 3e6 to 3e7 samples
    N, C, _ = xt.forward(p, *inp.args(), want_amatrix=False, ctx=ctx)
    Nr, Cr = oracle_lib.forward_rays(inp, rays)[:2]
    assert max_rel_err(N, Nr) < FAST_RTOL and max_rel_err(C, Cr) < FAST_RTOL


@pytest.mark.parametrize("side", [1.0, -1.0])
def test_detector_of_negative_area(ctx, oracle_lib, side):
    """A row pitch of the other sign makes the detector's area negative and sigma^2 with it,
    for some voxels and energies or for all: what a NaN term belongs to is NaN, as in
    the reference's arithmetic, not a finite sum without that term."""
    nans = 0
    for seed in range(6):
        rng = np.random.default_rng(150 + seed)
        p = sized_problem(12, 9, 3, 7, 7, 6, 2, nwt=24)
        p.row_pitch *= side * np.exp(rng.uniform(-3.0, 3.0))
        inp = synth.make_inputs(p, 151 + seed)
        rays = np.arange(p.rays)
        x = rng.uniform(0.1, 1.0, (p.nx * p.ny, p.nwt)).astype(np.float32)
        x[inp.seg == 0] = 0.0
        w = np.where(rng.uniform(size=p.rays) < 0.2, 1.0, 0.0).astype(np.float32)
        N, C, A = xt.forward(p, *inp.args(), ctx=ctx)
        op = xt.Operator(p, inp.spectrum, inp.seg, inp.a1, inp.a2, ctx=ctx)
        got = [N, C, A, op.forward(x.reshape(-1)), op.adjoint(w)]
        op.close()
        Nr, Cr, Ar, _ = oracle_lib.forward_rays(inp, rays, want_a=True)
        y_ref, g_ref = oracle_lib.vox_rays(inp, rays, x=x.reshape(-1), w=w)
        for a, b in zip(got, [Nr, Cr, np.asarray(Ar).reshape(-1), y_ref, np.asarray(g_ref).reshape(-1)]):
            assert np.array_equal(np.isnan(a), np.isnan(b))
            nans += int(np.isnan(b).sum())
    assert (nans > 0) == (side < 0)
