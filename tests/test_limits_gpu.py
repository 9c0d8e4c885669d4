"""Geometries, sizes and values at the ends of what the entry points accept:
distant sources and detectors, a flat fan, voxels of any side, tables of any
shape, infinite unknowns, calls that fail half way -- against the FP64 oracle."""
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
