"""The cluster V-cycle keeps its results to the last bit: checksums of one V-cycle (colour smoother on the
levels above the cluster) on fixed inputs, recorded with CUDA 12.9 for sm_100a. The order in which a vertex's
27 products are summed shows here and nowhere else (the solver's gates do not see it), and a design run
carries it into its densities. Levels with the stencils in shared memory and in global memory, the residual
in one sum and in eight, one and several planes per CTA."""
import zlib

import numpy as np
import pytest

from opentm_b200 import workloads as wl

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

# (nz, ny, nx), sweeps per leg -> CRC-32 of the correction
RECORDED = {((16, 16, 16), 2): 0xbb7f1156, ((32, 32, 32), 2): 0xb6d3c846, ((32, 32, 32), 1): 0x656abe76,
            ((64, 64, 64), 1): 0xa659eb23, ((64, 64, 64), 2): 0x4818a41d, ((72, 56, 40), 2): 0xe946b28f,
            ((32, 56, 40), 2): 0x9d5f9a4d, ((96, 64, 128), 1): 0x771f0c85, ((48, 48, 48), 2): 0xf943ae71,
            ((24, 40, 56), 2): 0xcb79eebd, ((32, 64, 48), 2): 0x143c0293}


@pytest.mark.parametrize("shape,sweeps", list(RECORDED))
def test_cycle_bits(shape, sweeps):
    from opentm_b200 import HomoConfig, Homogenization_H
    nz, ny, nx = shape
    n = nz * ny * nx
    k = (1e-3 + wl.uniform(7, n).reshape(shape) ** 3).astype(np.float32)
    f = (wl.uniform(9, 3 * n).reshape((3,) + shape) - 0.5).astype(np.float32)
    f -= f.mean((1, 2, 3), keepdims=True)
    H = Homogenization_H(HomoConfig(reso=(nx, ny, nz), pre_smooth=sweeps, post_smooth=sweeps, smoother="color"))
    H.update(torch.from_numpy(k).cuda())
    assert H.stats().cluster_level >= 1
    u = H.v_cycle(torch.from_numpy(f).cuda(), pre=sweeps, post=sweeps).cpu().numpy()
    assert zlib.crc32(np.ascontiguousarray(u).tobytes()) == RECORDED[(shape, sweeps)]
