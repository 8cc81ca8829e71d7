"""GPU parity of the MMA step whose interior-point iteration runs on the device, at the sizes where its
passes change: fewer variables than one block, odd counts (one variable per loop step), one loop step per
thread and several, one to eight constraints. FP64 on both sides: the tolerance of the other MMA test."""
import ctypes

import numpy as np
import pytest

import oracle as ora
from opentm_b200 import _lib
from tests.test_gpu_mma import MMA_TOL, _problem

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(1, 1), (7, 2), (256, 1), (513, 3), (4096, 4), (2001, 5), (1200, 8), (160000, 1)])
def test_mma_sizes(n, m):
    t, w, A = _problem(n, m, 60 + m)
    V = (0.3 + 0.05 * np.arange(m)) * n
    xmin, xmax, o1 = np.zeros(n), np.ones(n), np.full(n, 0.5)
    ref = dict(x=o1.copy(), o1=o1.copy(), o2=o1.copy(), lo=xmin.copy(), up=xmax.copy())
    dev = {k: torch.from_numpy(v.copy()).cuda() for k, v in ref.items()}
    dmin, dmax = torch.from_numpy(xmin).cuda(), torch.from_numpy(xmax).cuda()
    a, c, d = np.zeros(m), np.full(m, 1e3), np.ones(m)
    da, dc, dd = (torch.from_numpy(v).cuda() for v in (a, c, d))
    L, P = _lib.lib(), ctypes.c_void_p
    for it in range(1, 5):
        xc = ref["x"]
        g, dg, df = (A @ xc) / V - 1.0, A / V[:, None], 2 * w * (xc - t)
        ref["x"], ref["o1"], ref["o2"], ref["lo"], ref["up"] = ora.mmasub(
            it, xc, xmin, xmax, ref["o1"], ref["o2"], df, g, dg, ref["lo"], ref["up"], 1.0, a, c, d, 1.0)
        xd = dev["x"].cpu().numpy()
        ddf = torch.from_numpy(2 * w * (xd - t)).cuda()
        dgv = torch.from_numpy((A @ xd) / V - 1.0).cuda()
        dgd = torch.from_numpy(np.ascontiguousarray(A / V[:, None])).cuda()
        pp = _lib.PitchedPtr(dgd.data_ptr(), n * 8, n * 8, m)
        s = L.otm_mmasub_device(m, n, it, P(dev["x"].data_ptr()), P(dmin.data_ptr()), P(dmax.data_ptr()),
                                P(dev["o1"].data_ptr()), P(dev["o2"].data_ptr()), 1.0, P(ddf.data_ptr()),
                                P(dgv.data_ptr()), pp, P(dev["lo"].data_ptr()), P(dev["up"].data_ptr()), 1.0,
                                P(da.data_ptr()), P(dc.data_ptr()), P(dd.data_ptr()), 1.0,
                                P(torch.cuda.current_stream().cuda_stream))
        assert s == 0, _lib.last_error()
        torch.cuda.synchronize()
        for k in ("x", "o1", "o2", "lo", "up"):
            np.testing.assert_allclose(dev[k].cpu().numpy(), ref[k], rtol=0, atol=MMA_TOL, err_msg=f"{k} at {it}")
