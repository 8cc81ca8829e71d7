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


# (nz, ny, nx) -> unknowns; from 528 on the rows lie in global memory
@pytest.mark.parametrize("shape,n", [((3, 4, 3), 36), ((7, 3, 5), 105), ((5, 5, 5), 125), ((15, 7, 5), 525),
                                     ((11, 7, 7), 539), ((9, 9, 9), 729), ((11, 9, 10), 990), ((8, 16, 8), 1024)])
def test_inverse_itself(shape, n):
    """A cell of one level: a V-cycle is the inverse applied to the right-hand side, compared with a dense FP64
    solve (in the solver a wrong row would only cost iterations). The device's matrix has FP32 entries, sums of
    at most 8 conductivities times a constant: 8 half-ulps of entries whose rows sum to at most twice the
    diagonal, so 16 * 2^-24 of the matrix and that times its condition of the solution."""
    import oracle as ora
    from opentm_b200 import HomoConfig, Homogenization_H
    k, _ = random_k(shape, seed=n + 7)
    nz, ny, nx = shape
    H = Homogenization_H(HomoConfig(reso=(nx, ny, nz), coarsest_max_dof=1024))
    assert H.stats().levels == 1
    H.update(torch.from_numpy(k).cuda())
    rng = np.random.default_rng(n)
    f = rng.standard_normal((3,) + shape).astype(np.float32)
    u = H.v_cycle(torch.from_numpy(f).cuda()).cpu().numpy().reshape(3, n)
    A = np.empty((n, n))
    for i in range(n):
        e = np.zeros(n)
        e[i] = 1.0
        A[:, i] = ora.apply(1e-9 + k.astype(np.float64), e.reshape(shape)).ravel()
    w = np.linalg.eigvalsh(A)
    fc = f.reshape(3, n).astype(np.float64)
    ref = np.linalg.solve(A + np.trace(A) / n / n, (fc - fc.mean(1, keepdims=True)).T).T
    tol = 16 * 2.0 ** -24 * w[-1] / w[1]
    assert tol < 0.05
    for c in range(3):
        assert np.linalg.norm(u[c] - ref[c]) <= tol * np.linalg.norm(ref[c])
