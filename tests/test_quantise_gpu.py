"""Morton codes of coordinates on and a few floats beside every cell boundary,
for ranges whose 1024th is no float, tiny and huge ranges, zero, the box's upper
end and just below it: the oracle's IEEE division, bit for bit."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("low,extent", [(0.0, 1024.0), (0.0, 1023.0), (-7.3, 0.1), (0.0, 3e-5),
                                        (0.0, 1e-30), (5.0, 1e12), (-100.0, 200.0), (0.0, 1.0)])
def test_codes_beside_cell_boundaries(low, extent):
    from pipeline_gb300.kernels import k_ComputeMortonCode

    low, extent = np.float32(low), np.float32(extent)
    edge = (np.arange(1025, dtype=np.float64) * float(extent) / 1024 + float(low)).astype(np.float32)
    beside = [edge]
    for step in (np.float32(-np.inf), np.float32(np.inf)):
        x = edge
        for _ in range(6):
            x = np.nextafter(x, step)
            beside.append(x)
    x = np.unique(np.concatenate(beside))
    q = (x - low) / extent
    x = x[(q >= 0) & (q < 1)]  # inside the box: codes are defined
    rng = np.random.default_rng(1)
    pts = np.ones((3 * len(x), 4), np.float32)
    pts[:, :3] = rng.choice(x, (3 * len(x), 3))
    for axis in range(3):
        pts[axis * len(x):(axis + 1) * len(x), axis] = x
    keys = torch.zeros(len(pts), dtype=torch.int32, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    k_ComputeMortonCode(torch.from_numpy(pts).cuda(), keys, len(pts), float(low), float(extent),
                        status=status)
    assert int(status[0]) == 0
    assert keys.cpu().numpy().view(np.uint32).tobytes() == \
        np.asarray(O.morton(pts, float(low), float(extent))).tobytes()
