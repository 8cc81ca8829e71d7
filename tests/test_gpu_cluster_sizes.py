"""GPU parity of the one-launch cluster V-cycle at the sizes where its colour passes split differently:
a lane per vertex and load case with the common and with a wider stencil stride, a lane per vertex (more
than a third of the CTA's threads have a vertex), stencils in global memory, slabs of no, one and several
planes. The cluster cycle agrees with the per-level kernels as in the other cluster tests (the same
smoother and operators; sums in another order) and meets the oracle gates."""
import pytest

from tests.helpers import random_k, rel_c
from tests.test_gpu_homo import check_against_oracle, gpu_run

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,level", [((16, 16, 16), 1), ((32, 56, 40), 1), ((32, 64, 48), 1), ((72, 56, 40), 1),
                                         ((20, 24, 32), 1), ((80, 16, 24), 1), ((24, 40, 56), 1)])
def test_cluster_pass_splits(shape, level):
    k, _ = random_k(shape, seed=sum(shape))
    H1, C1, E1, s1 = gpu_run(k, tol=1e-7, smoother="color")
    H2, C2, _, _ = gpu_run(k, tol=1e-7, smoother="color", cluster_cycle=0)
    assert H1.stats().cluster_level == level and H2.stats().cluster_level == -1
    assert abs(H1.stats().iterations - H2.stats().iterations) <= 1
    assert rel_c(C1, C2) <= 1e-6
    check_against_oracle(k, C1, E1, s1)
