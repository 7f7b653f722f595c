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


@pytest.mark.parametrize("dtype", [np.float64, "df64"])
@pytest.mark.parametrize("n,blocksize", [(700, 80), (3000, 8), (3000, 14), (3000, 30), (40000, 20), (40000, 80)])
def test_low_segments(dtype, n, blocksize):
    """Near-field columns dealt out to lane groups on segments of few rows: the stage
    schedules against the two-launch one bit for bit, FP64 against the streamed CTAs
    (another order of sums) to 1e-13, HM_DF64 against FP64 to 1e-12 of | |A||x| |'s bound
    (its pairs hold 48 bits)."""
    rng = np.random.default_rng(n + blocksize)
    x, y = (np.sort(rng.random(n))[::-1].copy() for _ in range(2))
    H = hm.KernelMatrix(hm.cauchykernel, x, y, 1.0, 0.0, 1.0, 0.0, dtype=dtype, blocksize=blocksize)
    F = hm.KernelMatrix(hm.cauchykernel, x, y, 1.0, 0.0, 1.0, 0.0, blocksize=blocksize)
    for k in (1, 2, 4, 8):
        g = torch.Generator("cuda").manual_seed(k)
        B = torch.randn(k, n, device="cuda", dtype=torch.float64, generator=g).t()
        U0 = torch.randn(k, n, device="cuda", dtype=torch.float64, generator=g).t()
        for accumulate in (False, True):
            U = H.mul(U0.clone(), B, accumulate=accumulate)
            H.set_overlap(1)
            V = H.mul(U0.clone(), B, accumulate=accumulate)
            H.set_overlap(True)
            assert torch.equal(U, V)
            F.set_near_kernel("stream")
            R = F.mul(U0.clone(), B, accumulate=accumulate)
            F.set_near_kernel("auto")
            err = torch.linalg.norm(U - R, dim=0) / torch.linalg.norm(R, dim=0)
            assert (err <= (1e-13 if dtype is np.float64 else 1e-12)).all()
    assert H.device_status() == 0
    H.free()
    F.free()
