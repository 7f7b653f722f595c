"""Products with two to eight right-hand sides, whose tree passes run in chunks
of 2, 4 or 8: every column against the one-vector product of the same handle,
at a rank with unrolled kernels (20), one without (13), and an odd one (7).

Both sum the same stored values in the storage type, in chains of at most 64
near-field terms per fold, `rank` terms per transfer and 24 transfers; the
difference is a few roundings of each: 1e-13 relative in FP64, 1e-6 in FP32
(the library's tolerances)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import hierarchicalmatrices as hm  # noqa: E402


@pytest.mark.parametrize("dtype,tol", [(np.float64, 1e-13), (np.float32, 1e-6), ("df64", 1e-12)])
@pytest.mark.parametrize("rank", [7, 13, 20])
@pytest.mark.parametrize("k", [2, 3, 4, 5, 8, 9])
def test_columns_equal_single_products(dtype, tol, rank, k):
    n, m = 3001, 2500
    rng = np.random.default_rng(rank)
    x, y = np.sort(rng.random(n))[::-1].copy(), np.sort(rng.random(m))[::-1].copy()
    H = hm.KernelMatrix(hm.logkernel, x, y, 1.0, 0.0, 1.0, 0.0, dtype=dtype, rank=rank, blocksize=40)
    tdt = torch.float32 if dtype == np.float32 else torch.float64
    X = torch.randn(k, m, device="cuda", dtype=tdt, generator=torch.Generator("cuda").manual_seed(k)).t()
    Y = H @ X
    for q in range(k):
        y1 = H @ X[:, q].contiguous()
        assert float(torch.linalg.norm((Y[:, q] - y1).double()) / torch.linalg.norm(y1.double())) <= tol
    U = torch.ones_like(Y)
    H.mul(U, X, accumulate=True)
    assert torch.allclose(U, 1 + Y, rtol=tol, atol=tol * float(Y.abs().max()))
    H.free()
