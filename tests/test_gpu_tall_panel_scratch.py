"""Many right-hand sides on matrices with basis panels split by rows: the partial sums of at
most 32 of them exist at once (whatever the panels' widths), and their windows give
the sums that a product of fewer right-hand sides gives, bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import hierarchicalmatrices as hm  # noqa: E402
from hierarchicalmatrices import _lib  # noqa: E402

LEAF, RANK = 64, 8


def hodlr(n, rng, dt, rank=RANK):
    if n <= LEAF:
        return torch.tensor(rng.standard_normal((n, n)), device="cuda", dtype=dt)
    H = hm.HierarchicalMatrix(2, 2)
    h = n // 2
    for i, j, m, k in ((1, 2, h, n - h), (2, 1, n - h, h)):
        U, V = (torch.tensor(rng.standard_normal((rank, s)), device="cuda", dtype=dt).t() for s in (m, k))
        H[hm.Block(i), hm.Block(j)] = hm.LowRankMatrix(U, torch.tensor(rng.random(rank) + 0.5, device="cuda", dtype=dt), V)
    H[hm.Block(1), hm.Block(1)] = hodlr(h, rng, dt, rank)
    H[hm.Block(2), hm.Block(2)] = hodlr(n - h, rng, dt, rank)
    return H


def test_scratch_of_many_vectors():
    """256 vectors on 65,536 rows: the library may take the coefficients (two of a slot's
    RANK values per vector, 2,046 slots) and the partial sums of 32 vectors (ten levels
    of 512 parts), with 48 MB to spare for the pool's granularity; sums of 32 values a part
    for all 256 vectors would be 335 MB."""
    n, k = 1 << 16, 256
    H = hodlr(n, np.random.default_rng(0), torch.float64)
    h = H.handle(np.float64)
    X = torch.randn(k, n, device="cuda", dtype=torch.float64).t()
    Y = torch.empty(k, n, device="cuda", dtype=torch.float64).t()
    st = torch.cuda.current_stream().cuda_stream

    def mul(cols):
        _lib.check(_lib.lib.hm_mul(h, X.data_ptr(), n, Y.data_ptr(), n, cols, 0, st))
        torch.cuda.synchronize()
    mul(9)                                               # the same kernels, so that their code is loaded
    before = torch.cuda.mem_get_info()[0]
    mul(k)
    taken = before - torch.cuda.mem_get_info()[0]
    assert taken <= 2 * 2046 * RANK * k * 8 + 10 * 512 * 32 * RANK * 8 + (48 << 20)


@pytest.mark.parametrize("dt", [torch.float64, torch.float32])
@pytest.mark.parametrize("n,rank", [(8192, 8), (20011, 5), (5000, 20)])
def test_windows(dt, n, rank):
    H = hodlr(n, np.random.default_rng(n), dt, rank)
    # panels in one kernel for any number of vectors (by default in chunks of eight up to 32)
    _lib.check(_lib.lib.hm_configure(H.handle(np.float64 if dt == torch.float64 else np.float32),
                                     _lib.HM_OPT_NEAR_KERNEL, 1))
    X = torch.randn(70, n, device="cuda", dtype=dt, generator=torch.Generator("cuda").manual_seed(1)).t()
    kmin = 9 if dt == torch.float64 else 16              # the panel kernels of more than eight vectors (tensor cores: 16)
    Y = H @ X
    for a, b in ((0, kmin), (20, 20 + kmin + 3), (0, 32), (0, 33), (31, 64), (32, 70), (5, 70)):
        assert torch.equal(H @ X[:, a:b], Y[:, a:b]), (a, b)
