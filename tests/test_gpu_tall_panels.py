"""Products whose low-rank factors are taller than one warp's basis panel (128
rows): the panels are split by rows and the parts' sums added in order.  Sizes
at the edges of a part (128 rows) and of a group of parts (64 x 128 rows), one
to nine right-hand sides, against the dense FP64 product of the stored factors.

Every result is a chain of at most 128 row terms, 64 parts, 64 groups, `rank`
far-field terms and a few roundings of inputs: |error| <= (264 + rank) u
(|U| |sigma| |V|^T |x|) with u the unit roundoff of the storage type."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import hierarchicalmatrices as hm  # noqa: E402

UNIT = {torch.float64: 2.0 ** -53, torch.float32: 2.0 ** -24}


def blocks(n, rank, dtype, seed):
    rng = np.random.default_rng(seed)
    U = torch.tensor(rng.standard_normal((rank, 70)), device="cuda", dtype=dtype).t()
    V = torch.tensor(rng.standard_normal((rank, n)), device="cuda", dtype=dtype).t()
    s = torch.tensor(rng.random(rank) + 0.5, device="cuda", dtype=dtype)
    H = hm.HierarchicalMatrix(1, 1)
    H[hm.Block(1), hm.Block(1)] = hm.LowRankMatrix(U, s, V)
    return H, U.double(), s.double(), V.double()


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("n,rank", [(128, 5), (129, 5), (257, 1), (8192, 12), (8193, 16), (8320, 17), (20011, 40)])
@pytest.mark.parametrize("k", [1, 3, 9])
def test_split_panels(dtype, n, rank, k):
    H, U, s, V = blocks(n, rank, dtype, 1000 * rank + n)
    X = torch.randn(k, n, device="cuda", dtype=dtype, generator=torch.Generator("cuda").manual_seed(k)).t()
    if k == 1:
        X = X[:, 0].contiguous()
    Y = H @ X
    ref = (U * s) @ (V.t() @ X.double())
    bound = (264 + rank) * UNIT[dtype] * ((U.abs() * s) @ (V.abs().t() @ X.double().abs()))
    assert ((Y.double() - ref).abs() <= bound).all()
    other = torch.cuda.Stream()
    other.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(other):
        Z = H @ X                       # the arrival counters of another stream
    torch.cuda.synchronize()
    assert torch.equal(H @ X, Y) and torch.equal(Z, Y)
