"""GPU parity of the coarse tile sweeps on both sides of the line between the two kernels: a level of at
most 148 tiles (a lane per vertex and load case, stencils in shared memory) and one of more. The level is
smoothed by the tiles; the solve takes as many iterations as with the colour passes (a wrong sweep costs
iterations, not accuracy), the two agree and the tiled one meets the oracle gates. One V-cycle keeps its bits:
checksums recorded with CUDA 12.9 for sm_100a from the kernel that serves more than 148 tiles, whose arithmetic
and order the other one shares."""
import zlib

import numpy as np
import pytest

from opentm_b200 import workloads as wl
from tests.helpers import random_k, rel_c
from tests.test_gpu_homo import check_against_oracle, gpu_run

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


# tiles of the first coarse level: 12, 32, 144 and 160
@pytest.mark.parametrize("shape", [(48, 32, 64), (64, 64, 64), (96, 96, 128), (128, 160, 64)])
def test_coarse_tile_counts(shape):
    k, _ = random_k(shape, seed=sum(shape) + 1)
    H1, C1, E1, s1 = gpu_run(k, tol=1e-7, cluster_cycle=0)
    H2, C2, _, _ = gpu_run(k, tol=1e-7, cluster_cycle=0, smoother="color")
    assert H1.level(1).smoother == 1 and H2.level(1).smoother == 0
    assert abs(H1.stats().iterations - H2.stats().iterations) <= 1
    assert rel_c(C1, C2) <= 2e-6
    check_against_oracle(k, C1, E1, s1)


# (nz, ny, nx), cluster cycle, sweeps per leg -> CRC-32 of the correction
RECORDED = {((48, 32, 64), 0, 2): 0xcce2aefe, ((64, 64, 64), 0, 2): 0x40963ad6, ((64, 64, 64), 1, 2): 0x72ecc1fd,
            ((64, 64, 64), 1, 3): 0xc572a5d8, ((96, 96, 128), 1, 2): 0x697cfc1c, ((128, 160, 64), 0, 2): 0x1652e3f9,
            ((64, 48, 32), 1, 2): 0xc86d9aeb}


@pytest.mark.parametrize("shape,cluster,sweeps", list(RECORDED))
def test_tiled_cycle_bits(shape, cluster, sweeps):
    from opentm_b200 import HomoConfig, Homogenization_H
    nz, ny, nx = shape
    n = nz * ny * nx
    k = (1e-3 + wl.uniform(7, n).reshape(shape) ** 3).astype(np.float32)
    f = (wl.uniform(9, 3 * n).reshape((3,) + shape) - 0.5).astype(np.float32)
    f -= f.mean((1, 2, 3), keepdims=True)
    H = Homogenization_H(HomoConfig(reso=(nx, ny, nz), pre_smooth=sweeps, post_smooth=sweeps, cluster_cycle=cluster))
    H.update(torch.from_numpy(k).cuda())
    assert H.stats().smoother == 1 and H.level(1).smoother == 1
    u = H.v_cycle(torch.from_numpy(f).cuda(), pre=sweeps, post=sweeps).cpu().numpy()
    assert zlib.crc32(np.ascontiguousarray(u).tobytes()) == RECORDED[(shape, cluster, sweeps)]
