"""FP64 leaf bases and far field with eight panels or row slots per CTA (large trees)
against the lane-per-right-hand-side kernels: the same sums in the same order, so the
same bits; ragged last CTAs, uneven panels and rows, each chunk of right-hand sides and
more than one."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import hierarchicalmatrices as hm  # noqa: E402


@pytest.mark.parametrize("points,n", [("uniform", 36000), ("uniform", 45001), ("beta", 60007), ("grid", 65536)])
def test_flat_equals_wide(points, n):
    rng = np.random.default_rng(n)
    if points == "grid":
        x, y = ((np.arange(n) + 0.75) / n)[::-1].copy(), ((np.arange(n) + 0.25) / n)[::-1].copy()
    else:
        x, y = (np.sort(rng.random(n) if points == "uniform" else rng.beta(0.5, 0.5, n))[::-1].copy() for _ in range(2))
    H = hm.KernelMatrix(hm.cauchykernel, x, y, 1.0, 0.0, 1.0, 0.0)
    for k in (2, 3, 4, 5, 8, 9, 20):
        g = torch.Generator("cuda").manual_seed(k)
        B = torch.randn(k, n, device="cuda", dtype=torch.float64, generator=g).t()
        U = H @ B
        H.set_wide_tree("all")
        W = H @ B
        H.set_wide_tree(True)
        assert torch.equal(U, W), k
        if k == 2:                                       # one right-hand side: its own chunk width
            for q in range(2):
                u = H @ B[:, q].contiguous()
                assert torch.linalg.norm(u - U[:, q]) <= 1e-15 * n ** 0.5 * torch.linalg.norm(U[:, q])
    assert H.device_status() == 0
    H.free()
