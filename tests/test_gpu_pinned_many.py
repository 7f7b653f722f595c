"""Products of more than eight right-hand sides from and to page-locked host memory
(mul_host): the leaf stage brings the vectors in, so the near field must not start before
it.  Other vectors on every call, so that values of the call before would show; the same
bits as the product on device tensors.  Sizes on both sides of the chunked panels' lines
(400 and 1,200 coefficient slots, about n / 30; tensor cores from 16 FP32 vectors)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import hierarchicalmatrices as hm  # noqa: E402

TDT = {np.float64: torch.float64, np.float32: torch.float32}


@pytest.fixture(scope="module", params=[(9000, np.float64), (50000, np.float64), (50000, np.float32),
                                        (90001, np.float32)])
def mat(request):
    n, dt = request.param
    rng = np.random.default_rng(n)
    x, y = (np.sort(rng.random(n))[::-1].copy() for _ in range(2))
    H = hm.KernelMatrix(hm.cauchykernel, x, y, 1.0, 0.0, 1.0, 0.0, dtype=dt)
    yield n, dt, H
    H.free()


@pytest.mark.parametrize("k", [9, 13, 15, 16, 20, 40])
@pytest.mark.parametrize("overlap", [True, 0, 2, 3, 4])
def test_fresh_vectors(mat, k, overlap):
    n, dt, H = mat
    u = torch.empty(k, n, dtype=TDT[dt]).pin_memory()
    H.set_overlap(overlap)
    try:
        for i in range(4):                               # plain, captured, replayed
            v = torch.randn(k, n, dtype=TDT[dt], generator=torch.Generator().manual_seed(100 * k + i)).pin_memory()
            H.mul_host(u.numpy().T, v.numpy().T, accumulate=False)
            assert torch.equal(u.t(), (H @ v.cuda().t()).cpu()), i
    finally:
        H.set_overlap(True)
    assert H.device_status() == 0
