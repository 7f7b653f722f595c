"""Tensor-core panels (16 and more FP32 right-hand sides) where their tiles and
pipelines end: segments of few columns and of many, fewer items than SMs.

Each FP32 value is split exactly into three BF16 pieces and the products are
summed in FP32: 1e-6 of | |A| |x| | in the 2-norm per column."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import hierarchicalmatrices as hm  # noqa: E402

TOL32 = 1e-6


def columns(rows, k, seed, pad=0):
    g = torch.Generator("cuda").manual_seed(seed)
    return torch.randn(k, rows + pad, device="cuda", dtype=torch.float32, generator=g).t()[:rows]


@pytest.mark.parametrize("cols,k", [(1, 40), (31, 40), (33, 40), (1500, 40), (7000, 130)])
def test_assembled_blocks(cols, k):
    """One dense block of `cols` columns beside a low-rank one of rank 5; 7,000
    columns leave room for a single operand stage."""
    rng = np.random.default_rng(cols)
    A, U, V = rng.standard_normal((130, cols)), rng.standard_normal((130, 5)), rng.standard_normal((70, 5))
    s = rng.random(5) + 1

    def dev(a):
        return torch.tensor(np.ascontiguousarray(a.T), device="cuda", dtype=torch.float32).t()
    H = hm.HierarchicalMatrix(1, 2)
    H[hm.Block(1), hm.Block(1)] = dev(A)
    H[hm.Block(1), hm.Block(2)] = hm.LowRankMatrix(dev(U), torch.tensor(s, device="cuda", dtype=torch.float32), dev(V))
    X = columns(cols + 70, k, 1)
    D = torch.cat([dev(A).double(), (dev(U).double() * torch.tensor(s, device="cuda").float().double()) @ dev(V).double().t()], 1)
    ref = D @ X.double()
    got = H @ X
    bound = TOL32 * torch.linalg.norm(D.abs() @ X.double().abs(), dim=0)
    assert (torch.linalg.norm(got.double() - ref, dim=0) <= bound).all()
