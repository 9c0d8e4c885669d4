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
