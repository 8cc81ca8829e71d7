"""GPU parity of cells whose coarsest level is solved by the cluster inversion (otm_direct.cuh) at the
sizes where its split changes: fewer unknowns than one block of 16 rows, a last block that is not
full, one block row per CTA and more, rows in shared and in global memory. The gates are those of the
other parity tests (tests/helpers.py); the inverse is in FP64, so its own error does not show in them."""
import numpy as np
import pytest

from tests.helpers import random_k
from tests.test_gpu_homo import check_against_oracle, gpu_run

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


# (nz, ny, nx) -> unknowns of the coarsest level
@pytest.mark.parametrize("shape,n", [((3, 4, 3), 36), ((7, 3, 5), 105), ((12, 10, 8), 120), ((10, 10, 12), 150),
                                     ((36, 28, 20), 315), ((16, 16, 16), 64), ((16, 26, 14), 728), ((20, 22, 18), 990)])
def test_coarsest_inverse_sizes(shape, n):
    k, _ = random_k(shape, seed=n)
    H, C, E, sens = gpu_run(k, tol=1e-7)
    assert int(np.prod(H.stats().coarsest_reso[:])) == n
    check_against_oracle(k, C, E, sens)
