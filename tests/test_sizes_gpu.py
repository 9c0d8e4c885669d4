"""The kernels at the sizes where their splits change -- the smallest problems,
odd sizes, remainders of strips, tiles and warps -- against the FP64 oracle.
Tolerances are those of the parity tests (tests/tolerances.py)."""
import numpy as np
import pytest

import xrd_tomography_gb300 as xt
from xrd_tomography_gb300 import synth
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


def sized_problem(nx, ny, views, px, es, ed, dnrg, nwt=32, nqf=64, mats=3, e_det=(20.0, 80.0)):
    """A fan scanner around an nx x ny phantom of 2 mm voxels, scaled as a whole
    with the phantom so that the scattering angles stay on the q grid."""
    p = xt.reference_problem(nx, ny)
    p.n_src, p.n_col, p.n_row = views, px, 1
    p.nrg_src, p.nrg_det, p.dnrg = es, ed, dnrg
    p.e_src_min, p.e_src_max = 20.0, 80.0
    p.e_det_min, p.e_det_max = e_det
    p.nwt, p.nqf, p.n_mat = nwt, nqf, mats
    p.q_lo, p.q_hi, p.dq0 = 0.5, 4.0, 0.02 if nwt > 32 else 0.05
    side = max(nx, ny)
    return synth.scanner(p, 2.0, 3.0 * side, 2.2 * side, 2.6 * side / px, row_mm=0.02 * side, z0_mm=0.1 * side,
                         focal_mm=0.01 * side)


def some_rays(p, n, seed):
    rng = np.random.default_rng(seed)
    return np.sort(rng.choice(p.rays, min(n, p.rays), replace=False))


# the walk's strips: one voxel, a few, several (210 ray groups), and groups
# with few of their 32 pixels
@pytest.mark.parametrize("nx,ny,views,px", [(5, 3, 2, 3), (14, 9, 3, 33), (33, 20, 9, 70), (70, 50, 30, 200)])
def test_forward_over_walk_strips(ctx, oracle_lib, nx, ny, views, px):
    inp = synth.make_inputs(sized_problem(nx, ny, views, px, 16, 12, 3), 100 + nx)
    p = inp.problem
    N, C, _ = xt.forward(p, *inp.args(), want_amatrix=False, ctx=ctx)
    rays = some_rays(p, 200, nx)
    Nr, Cr = oracle_lib.forward_rays(inp, rays)[:2]
    assert max_rel_err(N[rays], Nr) < FAST_RTOL
    assert max_rel_err(C[rays], Cr) < FAST_RTOL


# line integrals shared by 8, 4, 2 lanes and by one, on both sides of a voxel
@pytest.mark.parametrize("nx,ny,views,px", [(9, 7, 3, 11), (16, 14, 5, 29), (16, 15, 6, 45), (31, 29, 7, 61)])
def test_walk_lanes_per_ray(ctx, oracle_lib, nx, ny, views, px):
    inp = synth.make_inputs(sized_problem(nx, ny, views, px, 12, 12, 2), 900 + nx + px)
    p = inp.problem
    N, C, _ = xt.forward(p, *inp.args(), want_amatrix=False, ctx=ctx)
    rays = some_rays(p, 300, px)
    Nr, Cr, _, _ = oracle_lib.forward_rays(inp, rays)
    assert max_rel_err(N[rays], Nr) < FAST_RTOL
    assert max_rel_err(C[rays], Cr) < FAST_RTOL
    # a few rays by themselves: the same bits
    Ns, Cs, _ = xt.forward_rays(p, rays[:5], *inp.args(), ctx=ctx)
    assert np.array_equal(Ns, N[rays[:5]]) and np.array_equal(Cs, C[rays[:5]])


# the forward's splits: tiles of one step, remainders of steps and tiles, two
# tiles and more; more and fewer energies than runs; source bins wider than
# detector bins (a range meets many channels) and a detector grid that only
# part of the source bins reaches; many detector bins per window (fewer warps)
@pytest.mark.parametrize("nx,ny,es,ed,dnrg,nqf,e_det", [
    (9, 5, 1, 1, 0, 7, (20.0, 80.0)), (24, 24, 7, 7, 3, 64, (20.0, 80.0)), (44, 40, 12, 12, 2, 96, (20.0, 80.0)),
    (31, 33, 65, 33, 4, 130, (20.0, 80.0)), (16, 12, 20, 61, 3, 64, (20.0, 80.0)),
    (20, 16, 16, 300, 4, 64, (20.0, 80.0)), (12, 12, 11, 900, 5, 64, (20.0, 80.0)),
    (20, 16, 40, 9, 1, 64, (30.0, 70.0)), (18, 18, 128, 128, 5, 64, (20.0, 80.0))])
def test_forward_over_splits(ctx, oracle_lib, nx, ny, es, ed, dnrg, nqf, e_det):
    inp = synth.make_inputs(sized_problem(nx, ny, 3, 40, es, ed, dnrg, nqf=nqf, e_det=e_det), 200 + nx + es)
    p = inp.problem
    N, C, _ = xt.forward(p, *inp.args(), want_amatrix=False, ctx=ctx)
    rays = some_rays(p, 300, nx)
    Nr, Cr = oracle_lib.forward_rays(inp, rays)[:2]
    assert max_rel_err(N[rays], Nr) < FAST_RTOL
    assert max_rel_err(C[rays], Cr) < FAST_RTOL
    N2, C2, _ = xt.forward(p, *inp.args(), want_amatrix=False, ctx=ctx)
    assert np.array_equal(N, N2) and np.array_equal(C, C2)
    S1 = synth.coherent_table(inp)
    for bilinear in (False, True):
        Nt, Ct = xt.forward_tables(p, inp.spectrum, inp.seg, inp.a1, inp.a2, S1, inp.S2, *inp.args()[6:],
                                   bilinear=bilinear, ctx=ctx)
        Nr, Cr = oracle_lib.forward_tables(inp, S1, rays, bilinear=bilinear)
        assert max_rel_err(Nt[rays], Nr) < FAST_RTOL
        assert max_rel_err(Ct[rays], Cr) < FAST_RTOL


# line integrals across uniform squares: larger than the largest radius a cell
# carries (31), cut by the map's edge and by thin borders; with a gradient
# that leaves no cell uniform; and the empty phantom but for one voxel
@pytest.mark.parametrize("kind", ["blocks", "gradient", "one voxel"])
def test_walks_across_uniform_squares(ctx, oracle_lib, kind):
    p = sized_problem(150, 137, 5, 64, 16, 16, 3)
    inp = synth.make_inputs(p, 300)
    seg = np.zeros((150, 137), np.int32)
    if kind == "one voxel":
        seg[70, 131] = 2
    else:
        seg[8:97, :120:3] = 1
        seg[20:140, 60] = 2
        seg[75, 3:130] = 3
    dens = np.where(seg > 0, 1.0, 0.0)
    if kind != "one voxel":
        dens[8:97, :120] = 1.0     # attenuating between the listed voxels, up to the map's edge
        dens[20:140, 60] = 2.0
        dens[100:140, 10:100] = 0.5
    if kind == "gradient":
        dens = dens + 1e-3 * np.add.outer(np.arange(150) % 7, np.arange(137) % 5)
    inp.seg = seg.flatten(order="F")
    inp.a1 = (2e-6 * dens).astype(np.float32).flatten(order="F")
    inp.a2 = (0.01 * dens).astype(np.float32).flatten(order="F")
    N, C, _ = xt.forward(p, *inp.args(), want_amatrix=False, ctx=ctx)
    rays = some_rays(p, 60, 3)
    Nr, Cr = oracle_lib.forward_rays(inp, rays)[:2]
    assert max_rel_err(N[rays], Nr) < FAST_RTOL
    assert max_rel_err(C[rays], Cr) < FAST_RTOL


# the model matrix over groups of 32 coarse bins: part of one, one and a part,
# exact ones, a second block of eight groups; several passes over the energies
# (large rows); voxels at the materials' borders; tiles and remainders of steps
@pytest.mark.parametrize("nx,ny,es,ed,nwt,mats", [(9, 5, 5, 5, 8, 2), (23, 30, 12, 12, 40, 3), (40, 44, 17, 13, 64, 4),
                                                  (16, 12, 9, 9, 130, 5), (12, 12, 64, 64, 256, 9),
                                                  (12, 14, 12, 12, 300, 2)])
def test_model_matrix_over_bin_groups(ctx, oracle_lib, nx, ny, es, ed, nwt, mats):
    inp = synth.make_inputs(sized_problem(nx, ny, 3, 34, es, ed, 2, nwt=nwt, mats=mats), 400 + nwt)
    p = inp.problem
    if nwt > 100:
        p.dq0 = 0.005
    rays = some_rays(p, 60, nwt)
    Nr, Cr, Ar = oracle_lib.forward_rays(inp, rays, want_a=True)[:3]
    N, C, A = xt.forward_rays(p, rays, *inp.args(), want_amatrix=True, ctx=ctx)
    assert max_rel_err(N, Nr) < FAST_RTOL
    assert max_rel_err(C, Cr) < FAST_RTOL
    assert max_rel_err(A, np.asarray(Ar).reshape(A.shape)) < FAST_RTOL
    N, C, A = xt.forward(p, *inp.args(), ctx=ctx)
    assert max_rel_err(A.reshape(p.rays, p.n_mat, p.nwt)[rays], np.asarray(Ar).reshape(len(rays), p.n_mat, p.nwt)) < FAST_RTOL
    assert np.array_equal(A, xt.forward(p, *inp.args(), ctx=ctx)[2])


def vox_case(nx, ny, views, px, es, ed, dnrg, nwt, seed):
    p = sized_problem(nx, ny, views, px, es, ed, dnrg, nwt=nwt)
    if nwt > 100:
        p.dq0 = 0.004
    inp = synth.make_inputs(p, seed)
    rng = np.random.default_rng(seed)
    x = rng.uniform(0.0, 1.0, (nx * ny, nwt)).astype(np.float32)
    x[inp.seg == 0] = 0.0
    return inp, x.reshape(-1), rng.uniform(0.0, 2.0, p.rays).astype(np.float32)


# the per-voxel operator: one chunk of voxels, remainders of chunks and tiles;
# an odd number of energies and of coarse bins (both come in twos); one bin;
# more bins than a tile has room for twice
@pytest.mark.parametrize("nx,ny,es,ed,dnrg,nwt", [(5, 4, 1, 1, 0, 1), (24, 20, 7, 5, 2, 33), (30, 34, 12, 12, 2, 32),
                                                  (44, 48, 17, 13, 3, 41), (20, 18, 12, 12, 2, 257),
                                                  (12, 12, 65, 64, 5, 24)])
def test_operator_over_splits(ctx, oracle_lib, nx, ny, es, ed, dnrg, nwt):
    inp, x, w = vox_case(nx, ny, 3, 33, es, ed, dnrg, nwt, 500 + nwt)
    p = inp.problem
    op = xt.Operator(p, inp.spectrum, inp.seg, inp.a1, inp.a2, ctx=ctx)
    rays = some_rays(p, 150, nwt)
    ws = np.zeros_like(w)
    ws[rays] = w[rays]
    y_ref, g_ref = oracle_lib.vox_rays(inp, rays, x=x, w=w[rays])
    y = op.forward(x)
    assert max_rel_err(y[rays], y_ref) < FAST_RTOL
    assert max_rel_err(op.adjoint(ws), g_ref.reshape(-1)) < FAST_RTOL
    assert np.array_equal(y, op.forward(x))
    op.close()


def test_window_table_takes_any_order_of_bins(ctx, oracle_lib):
    """Coarse bins whose edges turn back (dq0 NWT far beyond the range): their
    centres are not in order, and the window table must still hold them all."""
    inp, x, w = vox_case(20, 16, 3, 33, 12, 12, 2, 32, 77)
    inp.problem.dq0 = 0.3
    p = inp.problem
    op = xt.Operator(p, inp.spectrum, inp.seg, inp.a1, inp.a2, ctx=ctx)
    rays = np.arange(p.rays)
    y_ref, g_ref = oracle_lib.vox_rays(inp, rays, x=x, w=w)
    assert max_rel_err(op.forward(x), y_ref) < FAST_RTOL
    assert max_rel_err(op.adjoint(w), g_ref.reshape(-1)) < FAST_RTOL
    op.close()


# CT chords: fewer than a warp, remainders, chords along the grid (views at
# multiples of 90 degrees), chords that miss the phantom, source bins in one
# pass, in several, and windows wider than a pass holds
@pytest.mark.parametrize("nx,ny,views,px,es,ed,dnrg", [(5, 4, 1, 3, 1, 1, 0), (33, 20, 4, 41, 12, 12, 2),
                                                       (70, 64, 9, 150, 64, 48, 5), (20, 24, 5, 33, 300, 290, 4),
                                                       (12, 12, 3, 7, 3401, 3, 1700)])
def test_ct_over_passes(ctx, oracle_lib, nx, ny, views, px, es, ed, dnrg):
    p = sized_problem(nx, ny, views, px, es, ed, dnrg)
    p.col_pitch *= 1.6
    inp = synth.make_inputs(p, 600 + nx)
    T, G = xt.ct_sinogram(p, inp.spectrum, inp.a1, inp.a2, ctx=ctx)
    rays = some_rays(p, 500, nx)
    Tr, Gr = oracle_lib.ct_rays(inp, rays)
    assert max_rel_err(T[rays], Tr) < FAST_RTOL
    assert max_rel_err(G[rays], Gr) < 1e-5


@pytest.mark.parametrize("N", [16, 48, 64, 80, 192, 256])
@pytest.mark.parametrize("M,K,off", [(1, 8, 0), (127, 24, 0), (145, 64, 1), (152 * 128 + 17, 40, 0), (40000, 64, 1),
                                     (60000, 16, 0)])
def test_basis_read_back(ctx, M, K, N, off):
    """Column blocks of 64 and 16 of the accumulator's read-back, ragged last
    tiles, several tiles per block, C and I off a 16-byte boundary.  The bound
    is that of the basis tests: each product to about 2^-21, the sum in FP32."""
    torch = pytest.importorskip("torch")
    g = torch.Generator(device="cuda").manual_seed(M + K + N)
    C = torch.randn(M * K + off, device="cuda", generator=g)[off:].view(M, K)
    B = torch.randn(K, N, device="cuda", generator=g)
    I = torch.full((M * N + off + 8,), -7.0, device="cuda")
    torch.cuda.synchronize()
    xt.basis_expand(C, B, I[off:off + M * N].view(M, N), ctx=ctx)
    got = I[off:off + M * N].view(M, N).double()
    bound = C.double().abs() @ B.double().abs()
    assert bool(((got - C.double() @ B.double()).abs() <= 4e-6 * bound + 1e-30).all())
    assert bool((I[:off] == -7.0).all()) and bool((I[off + M * N:] == -7.0).all())


# chords shared by 32, 16, 8, 4, 2 lanes and by one, counts that leave ragged
# warps; one lane with several passes of source bins, and with windows wider
# than a pass
@pytest.mark.parametrize("nx,ny,views,px,es,ed,dnrg", [(60, 50, 37, 43, 16, 12, 2), (60, 50, 37, 143, 16, 12, 2),
                                                       (60, 50, 61, 211, 16, 12, 2), (30, 34, 121, 211, 16, 12, 2),
                                                       (30, 34, 241, 211, 16, 12, 2), (30, 34, 401, 211, 16, 12, 2),
                                                       (12, 12, 401, 211, 2400, 8, 100), (12, 12, 401, 211, 2400, 8, 1000)])
def test_ct_lanes_per_chord(ctx, oracle_lib, nx, ny, views, px, es, ed, dnrg):
    p = sized_problem(nx, ny, views, px, es, ed, dnrg)
    p.col_pitch *= 1.6
    inp = synth.make_inputs(p, 700 + nx)
    T, G = xt.ct_sinogram(p, inp.spectrum, inp.a1, inp.a2, ctx=ctx)
    rays = some_rays(p, 400, nx + px)
    Tr, Gr = oracle_lib.ct_rays(inp, rays)
    assert max_rel_err(T[rays], Tr) < FAST_RTOL
    assert max_rel_err(G[rays], Gr) < 1e-5


@pytest.mark.parametrize("K", [4, 8, 12, 16, 20, 32, 36, 64, 68, 128, 132, 256, 260, 384, 388, 512, 516, 640, 644, 768,
                               772, 896, 900, 1024])
@pytest.mark.parametrize("rays", [1, 37, 2433, 20011])
def test_matrix_mlem_row_shapes(ctx, K, rays):
    """Every lanes-per-row and chunk count of the pass, at both ends of its
    range of K, with fewer rows than warps, ragged visits and several steps of
    the ring, both directions.  A, x, y and c are positive, so errors are
    relative: a chain of 4 products per chunk and 5 partner sums, the ratio, a
    chain of the warp's rows, its row groups, 16 warps and the update round
    e = (4 * 8 + 5 + 4 + rows + 5 + 16 + 4) 2^-24 at most, and an error of x
    comes back as twice that after an iteration: 7 e after three."""
    torch = pytest.importorskip("torch")
    it = 3
    g = torch.Generator(device="cuda").manual_seed(K + rays)
    A = torch.rand(rays, K, device="cuda", generator=g) + 0.1
    x0 = torch.rand(K, device="cuda", generator=g) + 0.1
    c = torch.rand(rays, device="cuda", generator=g) + 0.1
    y = (torch.rand(rays, device="cuda", generator=g) + 0.1) * K
    want, a = x0.double(), A.double()
    for _ in range(it):
        want = want * (a.T @ (y.double() / (a @ want + c.double() + 1e-20))) / (a.sum(0) + 1e-7)
    got = x0.clone()
    torch.cuda.synchronize()
    xt.mlem_matrix(A, y, c, got, it, ctx=ctx)
    per_warp = -(-rays // (152 * 8))
    tol = 7 * (66 + per_warp) * 2.0 ** -24
    rel = float(((got.double() - want).abs() / want).max())
    assert rel <= tol, (rel, tol)
