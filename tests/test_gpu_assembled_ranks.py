"""Assembled matrices whose BarycentricMatrix2D blocks differ in rank: a far-field block reads
as many coefficients as the largest rank has, and those past its own rank must not be what an
earlier product left in the scratch memory.  NaN products come first; the results of the
finite ones are the dense product's, within the rounding of its sums."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import hierarchicalmatrices as hm  # noqa: E402
from hierarchicalmatrices import _lib  # noqa: E402
from test_gpu_assembled_barycentric import TERMS, assemble  # noqa: E402


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("ranks", [(20, 6, 11), (32, 20, 1), (17, 16, 3)])
@pytest.mark.parametrize("overlap", [None, 0, 1])
def test_mixed_ranks_after_nan(dtype, ranks, overlap):
    tdt = torch.float64 if dtype == np.float64 else torch.float32
    H, D, S = assemble([60, 25, 140, 90, 31, 8, 77, 64], [300, 40, 129], lambda i: ranks[i % 3], 3)
    m, n = D.shape
    if overlap is not None:
        _lib.check(_lib.lib.hm_configure(H.handle(dtype), _lib.HM_OPT_OVERLAP, overlap))
    nan = torch.full((8, n), float("nan"), device="cuda", dtype=tdt).t()
    for k in (1, 2, 4, 8, 5):
        assert torch.isnan(H @ nan).all()
        X = torch.randn(k, n, device="cuda", dtype=tdt, generator=torch.Generator("cuda").manual_seed(k)).t()
        got = (H @ (X[:, 0].contiguous() if k == 1 else X)).double().cpu().numpy().reshape(-1, k)
        Xd = X.double().cpu().numpy()
        assert (np.abs(got - D @ Xd) <= TERMS * np.finfo(dtype).eps / 2 * (S @ np.abs(Xd))).all()


def test_without_allocations():
    """The same through hm_mul_noalloc, whose scratch all matrices share."""
    H, D, S = assemble([60, 25, 140], [300, 40, 129], lambda i: (20, 6, 11)[i % 3], 4)
    m, n = D.shape
    st = torch.cuda.current_stream().cuda_stream
    u = torch.empty(m, device="cuda", dtype=torch.float64)

    def run(h, v, out):
        _lib.check(_lib.lib.hm_mul_noalloc(h, v.data_ptr(), out.data_ptr(), 0, st))

    x = np.arange(2000, 0, -1) / 2000
    K = hm.KernelMatrix(hm.cauchykernel, x, x - 1 / 4000, 1.0, 0.0, 1.0, -1 / 4000)
    run(K.handle, torch.full((2000,), float("nan"), device="cuda", dtype=torch.float64),
        torch.empty(2000, device="cuda", dtype=torch.float64))
    v = torch.randn(n, device="cuda", dtype=torch.float64, generator=torch.Generator("cuda").manual_seed(1))
    run(H.handle(np.float64), v, u)
    vd = v.cpu().numpy()
    assert (np.abs(u.cpu().numpy() - D @ vd) <= TERMS * np.finfo(np.float64).eps / 2 * (S @ np.abs(vd))).all()
    K.free()
