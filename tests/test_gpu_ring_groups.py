"""Per-warp rings (3-8 FP32 right-hand sides) on segments of few rows, where lane
groups share a chunk's columns: 1 to 8, 9 to 16, 17 to 32 and more rows, ragged tails,
fewer segments than warps and several per warp, in the stage schedules and in the
two-launch schedule of small matrices.  Against the one-warp-per-segment kernel: 5e-7
of the column's norm (both fold their FP32 sums with TwoSum), u += H v included; against
each other bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import hierarchicalmatrices as hm  # noqa: E402


def colrel(a, b):
    a, b = a.double(), b.double()
    return (torch.linalg.norm(a - b, dim=0) / torch.linalg.norm(b, dim=0)).max().item()


@pytest.mark.parametrize("k", [3, 4, 5, 8])
@pytest.mark.parametrize("n,blocksize", [(700, 80), (3000, 8), (3000, 14), (3000, 30), (3000, 60), (40000, 20), (40000, 80),
                                         (400000, 80)])
def test_ring_groups(n, blocksize, k):
    rng = np.random.default_rng(n + blocksize)
    x, y = (np.sort(rng.random(n))[::-1].copy() for _ in range(2))
    H = hm.KernelMatrix(hm.cauchykernel, x, y, 1.0, 0.0, 1.0, 0.0, dtype=np.float32, blocksize=blocksize)
    g = torch.Generator("cuda").manual_seed(k)
    B = torch.randn(k, n, device="cuda", dtype=torch.float32, generator=g).t()
    U0 = torch.randn(k, n, device="cuda", dtype=torch.float32, generator=g).t()
    for accumulate in (False, True):
        U = U0.clone()
        H.mul(U, B, accumulate=accumulate)
        H.set_overlap(1)
        V = U0.clone()
        H.mul(V, B, accumulate=accumulate)
        assert torch.equal(U, V)
        H.set_near_kernel("warp")
        H.mul(V.copy_(U0), B, accumulate=accumulate)
        H.set_near_kernel("auto")
        H.set_overlap(True)
        assert colrel(U, V) <= 5e-7
    assert H.device_status() == 0
    H.free()
