"""GPU parity of the coarse tile sweeps on both sides of the line between the two kernels: a level of at
most 148 tiles (a lane per vertex and load case, stencils in shared memory) and one of more. The tiled
and the colour-pass smoothers agree and the tiled one meets the oracle gates."""
import pytest

from tests.helpers import random_k, rel_c
from tests.test_gpu_homo import check_against_oracle, gpu_run

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


# tiles of the first coarse level: 4, 32 and 160
@pytest.mark.parametrize("shape", [(32, 32, 32), (64, 64, 64), (128, 160, 64)])
def test_coarse_tile_counts(shape):
    k, _ = random_k(shape, seed=sum(shape) + 1)
    H1, C1, E1, s1 = gpu_run(k, tol=1e-7, cluster_cycle=0)
    H2, C2, _, _ = gpu_run(k, tol=1e-7, cluster_cycle=0, smoother="color")
    assert H1.level(1).smoother in (1, -1) and H2.level(1).smoother in (0, -1)
    assert rel_c(C1, C2) <= 2e-6
    check_against_oracle(k, C1, E1, s1)
