"""GPU parity of the streaming density filter and of the OC sensitivity filter against the FP64 oracle at
the sizes where their split changes: radii whose taps are compiled in and radii between them, one and four
rows per thread, cells narrower than the filter (voxels cut at both ends), rows and planes that end inside
a tile or a z chunk, pitched sources. Tolerance as the other filter tests: FP32 sums of at most a few
hundred taps of like sign, 1e-5 of the largest value."""
import numpy as np
import pytest

import oracle as ora
from opentm_b200 import workloads as wl
from tests.helpers import rel_field

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

FILTER_TOL = 1e-5

CASES = [((5, 4, 3), 1, 2.0), ((3, 2, 4), 0, 2.5), ((6, 17, 33), 0, 1.5), ((9, 15, 31), 1, 2.0), ((11, 18, 65), 1, 2.3),
         ((35, 20, 40), 1, 3.0), ((13, 9, 70), 0, 3.5), ((21, 33, 34), 1, 4.0), ((12, 13, 35), 0, 4.4),
         ((16, 16, 33), 1, 5.2), ((70, 130, 128), 1, 2.5), ((40, 140, 200), 0, 4.0), ((4, 4, 4), 1, 0.4), ((7, 8, 9), 1, 1.2),
         ((14, 15, 16), 0, 6.2)]


@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("shape,weight,radius", CASES)
def test_filter_sizes(shape, weight, radius, periodic):
    from opentm_b200 import filter_backward, filter_forward
    n = int(np.prod(shape))
    nz, ny, nx = shape
    src = wl.uniform(n + 1, n).reshape(shape).astype(np.float32)
    g = (wl.uniform(n + 2, n).reshape(shape) - 0.5).astype(np.float32)
    padded = torch.full((nz, ny, nx + 3), 99.0, device="cuda")
    padded[:, :, :nx] = torch.from_numpy(src).cuda()
    dst, ws = filter_forward(padded, (nx, ny, nz), radius, weight, periodic, src_pitchT=nx + 3)
    ref, ref_ws = ora.conv_forward(src, weight, radius, periodic)
    assert rel_field(dst.cpu().numpy(), ref)[0] <= FILTER_TOL
    assert rel_field(ws.cpu().numpy(), ref_ws)[0] <= FILTER_TOL
    gs = filter_backward(torch.from_numpy(g).cuda(), ws, (nx, ny, nz), radius, weight, periodic)
    assert rel_field(gs.cpu().numpy(), ora.conv_backward(g, ref_ws, weight, radius, periodic))[0] <= FILTER_TOL


@pytest.mark.parametrize("shape,radius", [((5, 4, 3), 2.0), ((9, 17, 33), 1.5), ((12, 10, 40), 3.0), ((14, 20, 35), 4.2)])
def test_oc_filter_sizes(shape, radius):
    from opentm_b200 import OCOptimizer
    n = int(np.prod(shape))
    nz, ny, nx = shape
    rho = (0.1 + 0.9 * wl.uniform(n + 3, n)).reshape(shape).astype(np.float32)
    s = -wl.uniform(n + 4, n).reshape(shape).astype(np.float32)
    st = torch.zeros((nz, ny, nx + 5), device="cuda")
    rt = torch.full((nz, ny, nx + 5), 7.0, device="cuda")
    st[:, :, :nx] = torch.from_numpy(s).cuda()
    rt[:, :, :nx] = torch.from_numpy(rho).cuda()
    OCOptimizer(n).filterSens(st, rt, nx + 5, (nx, ny, nz), radius)
    assert rel_field(st.cpu().numpy()[:, :, :nx], ora.oc_filter_sens(s, rho, radius))[0] <= FILTER_TOL
    assert bool((st[:, :, nx:] == 0).all())


@pytest.mark.parametrize("shape", [(2, 300000, 2), (300000, 1, 3), (2, 3, 300000)])
def test_filter_long_axis(shape):
    """An axis of more tiles than a launch has blocks along y or z."""
    from opentm_b200 import OCOptimizer, filter_forward
    n = int(np.prod(shape))
    nz, ny, nx = shape
    src = wl.uniform(n + 5, n).reshape(shape).astype(np.float32)
    dst, _ = filter_forward(torch.from_numpy(src).cuda(), (nx, ny, nz), 1.5, 1, False)
    assert rel_field(dst.cpu().numpy(), ora.conv_forward(src, 1, 1.5, False)[0])[0] <= FILTER_TOL
    rho = (0.1 + 0.9 * wl.uniform(n + 6, n)).reshape(shape).astype(np.float32)
    st = torch.from_numpy(-src).cuda()
    OCOptimizer(n).filterSens(st, torch.from_numpy(rho).cuda(), nx, (nx, ny, nz), 2.0)
    assert rel_field(st.cpu().numpy(), ora.oc_filter_sens(-src, rho, 2.0))[0] <= FILTER_TOL
