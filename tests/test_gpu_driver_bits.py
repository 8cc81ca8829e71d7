"""Design runs keep their results to the last bit: checksums of the densities and of the objective history
of short runs from fixed densities, recorded with CUDA 12.9 for sm_100a. A run amplifies a changed order of
any sum in the filter, the cycle or the optimiser: a last-bit change in one of them moves densities by 1e-4
and more within ten steps."""
import zlib

import numpy as np
import pytest

from opentm_b200 import workloads as wl

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

# (cells per axis, optimiser, steps, seed) -> CRC-32 of the densities and of the history
RECORDED = {(32, "oc", 10, 21): (0x008d791c, 0xa2a450d3), (64, "oc", 10, 22): (0xd65b9f76, 0x08cd3a8c),
            (48, "oc", 8, 23): (0xff3347f2, 0x8e6bd6fe), (32, "mma", 6, 21): (0x4800b873, 0xf98ec5d4)}


@pytest.mark.parametrize("n,model,steps,seed", list(RECORDED))
def test_design_run_bits(n, model, steps, seed):
    from opentm_b200.driver import DesignConfig, InitWay, Model, run_custom
    rho0 = (0.3 + 0.4 * wl.uniform(seed, n ** 3)).astype(np.float32).reshape(n, n, n)
    rho, info = run_custom(DesignConfig(reso=n, winit=InitWay.IWP, model=Model[model], max_iter=steps, finthres=0.0), rho0)
    got = tuple(zlib.crc32(np.ascontiguousarray(a).tobytes()) for a in (np.asarray(rho), np.asarray(info["history"])))
    assert got == RECORDED[(n, model, steps, seed)]
