"""The default schedule's rules (where the near field starts, which tree kernels
run) only choose among forms of one sum: the default product equals the plainest
forms bit for bit on both sides of each rule's lines (n / 30 coefficient slots
against 2,048, 8,192 and 16,384; 4/5, 8/9, 16/17 and 31/32 right-hand sides), also with
right-hand sides read from page-locked host memory."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import hierarchicalmatrices as hm  # noqa: E402


@pytest.fixture(scope="module", params=[(20000, np.float32), (70000, np.float32), (300000, np.float32),
                                        (600000, np.float32), (70000, "df64")])
def mat(request):
    n, dt = request.param
    rng = np.random.default_rng(n)
    x, y = (np.sort(rng.random(n))[::-1].copy() for _ in range(2))
    H = hm.KernelMatrix(hm.logkernel, x, y, 1.0, 0.0, 1.0, 0.0, dtype=dt)
    yield n, torch.float32 if dt == np.float32 else torch.float64, H
    H.free()


def columns(k, n, tdt):
    g = torch.Generator("cuda").manual_seed(k)
    return torch.randn(k, n, device="cuda", dtype=tdt, generator=g).t()


@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 8, 9, 16, 17, 31, 32])
def test_default_matches_one_stream_and_narrow_kernels(mat, k):
    n, tdt, H = mat
    B = columns(k, n, tdt)
    U = H @ B
    try:
        H.set_overlap(1)                                # tree and near field side by side, stage kernels
        assert torch.equal(H @ B, U)
        H.set_wide_tree(False)
        assert torch.equal(H @ B, U)
    finally:
        H.set_overlap(True)
        H.set_wide_tree(True)
    assert H.device_status() == 0


@pytest.mark.parametrize("k", [1, 3, 8])
def test_pinned_host_product(mat, k):
    n, tdt, H = mat
    B = columns(k, n, tdt)
    U = H @ B
    v = B.t().contiguous().cpu().pin_memory()
    u = torch.zeros_like(v).pin_memory()
    for _ in range(3):                                  # plain, captured, replayed
        H.mul_host(u.numpy().T, v.numpy().T, accumulate=False)
        assert torch.equal(u.t(), U.cpu())
