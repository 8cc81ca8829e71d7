"""The start of a solve. A handle knows when its solution is zero (fresh, reset, cold) and then starts with
r = b; a solution that the caller has set must not be taken for zero."""
import numpy as np
import pytest

from tests.helpers import KH_TOL, oracle_solution, random_k, rel_c

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "bf16", "fp16"])
@pytest.mark.parametrize("shape", [(32, 32, 32), (20, 24, 28)])
def test_solution_set_after_reset(shape, precision):
    from opentm_b200 import HomoConfig, Homogenization_H
    k, _ = random_k(shape, seed=sum(shape) + 3)
    nz, ny, nx = shape
    C_ref = oracle_solution(k)["C"]
    H = Homogenization_H(HomoConfig(reso=(nx, ny, nz), femRelThres=1e-6, pre_smooth=2, post_smooth=2,
                                    precision=precision))
    H.update(torch.from_numpy(k).cuda())
    C = H.heatMatrix()  # from a fresh handle's zeros
    first = H.stats().iterations
    assert rel_c(C, C_ref) <= KH_TOL
    x = [H.solution(c).clone() for c in range(3)]
    # all three cases set: nothing (or next to nothing) is left to do
    H.reset_displacement()
    for c in range(3):
        H.set_solution(c, x[c])
    assert rel_c(H.heatMatrix(), C_ref) <= KH_TOL
    assert H.stats().iterations <= 1 < first
    # one case set: the other two start from zero
    H.reset_displacement()
    H.set_solution(1, x[1])
    assert rel_c(H.heatMatrix(), C_ref) <= KH_TOL
    # reset alone: the solve from zero again
    H.reset_displacement()
    assert rel_c(H.heatMatrix(), C_ref) <= KH_TOL
    assert H.stats().iterations == first
    # and a further solve starts from its result
    assert rel_c(H.heatMatrix(), C_ref) <= KH_TOL
    assert H.stats().iterations <= 1
