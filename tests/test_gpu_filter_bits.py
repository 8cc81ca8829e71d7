"""The valid weight of a zero-padded filter is the sum of the in-bounds taps in the reference's order (x
fastest, z slowest), one FP32 addition after the other: compared bit for bit with that sum in numpy. Cells
cut at one end and at both ends of each axis, with more and with no more planes than the filter is wide, one
and four rows per thread, several z chunks, compiled-in and general radii."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _weights(kind, radius):
    """Normalised FP32 weights of the cube of offsets, (2h+1)^3, z slowest."""
    f = np.float32
    h = int(f(radius) + f(0.5))
    o = np.arange(-h, h + 1, dtype=np.float32)
    q2 = (o[:, None, None] ** 2 + o[None, :, None] ** 2 + o[None, None, :] ** 2) / (f(radius) * f(radius))
    q = np.sqrt(q2)
    w = (f(1) - f(6) * q2 + f(8) * q2 * q - f(3) * q2 * q2) if kind == 0 else f(1) - q
    w = np.where(q2 < 1, w, f(0)).astype(np.float32)
    total = np.cumsum(w.reshape(-1), dtype=np.float32)[-1]
    return h, w / total


def _valid(shape, kind, radius):
    h, w = _weights(kind, radius)
    inside = np.zeros([n + 2 * h for n in shape], dtype=bool)
    inside[tuple(slice(h, h + n) for n in shape)] = True
    acc = np.zeros(shape, dtype=np.float32)
    for z in range(2 * h + 1):
        for y in range(2 * h + 1):
            for x in range(2 * h + 1):
                if w[z, y, x] != 0:
                    acc += np.where(inside[z:z + shape[0], y:y + shape[1], x:x + shape[2]], w[z, y, x], np.float32(0))
    return acc


@pytest.mark.parametrize("shape,kind,radius", [
    ((9, 7, 35), 1, 1.2), ((16, 16, 33), 1, 2.0), ((20, 20, 20), 0, 1.5), ((3, 2, 4), 0, 2.4), ((5, 40, 3), 1, 2.0),
    ((12, 13, 35), 1, 3.0), ((6, 5, 40), 0, 3.2), ((7, 17, 66), 1, 3.0), ((70, 130, 128), 0, 3.0), ((24, 24, 24), 0, 4.0),
    ((70, 140, 130), 1, 4.4), ((8, 9, 3), 0, 4.0), ((14, 15, 16), 0, 5.2), ((10, 33, 34), 1, 6.2)])
def test_valid_weight_bits(shape, kind, radius):
    from opentm_b200 import filter_forward
    nz, ny, nx = shape
    _, ws = filter_forward(torch.ones(shape, device="cuda"), (nx, ny, nz), radius, kind, False)
    assert np.array_equal(ws.cpu().numpy(), _valid(shape, kind, radius))
