"""Products with user-assembled hierarchical matrices that hold BarycentricMatrix2D
blocks beside low-rank, dense and nested ones, with basis panels of 8 to 300 rows: equal
bit for bit on the default schedule and on the stage kernels, and to the dense product
within the rounding of its sums."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import hierarchicalmatrices as hm  # noqa: E402
from hierarchicalmatrices import _lib  # noqa: E402

Tree = hm.hierarchical("Tree", hm.BarycentricMatrix2D, hm.LowRankMatrix, "Matrix")
# units of one sum: a 300-row panel, a core of 20 columns, 20 far and 500 near columns, and
# the rounding of the stored values
TERMS = 300 + 20 + 20 + 500 + 10


def assemble(rows, cols, rank_of, seed):
    """A grid of len(rows) x len(cols) blocks (3 of 4 barycentric, the others low-rank
    and dense by turns, the first one a nested 2 x 2 matrix), the dense matrix and the
    matrix of absolute sums.  Row points lie in [2, 3], column points in [0, 1]."""
    rng = np.random.default_rng(seed)
    x, y = 2 + np.sort(rng.random(sum(rows)))[::-1], np.sort(rng.random(sum(cols)))[::-1]
    D, S = np.zeros((sum(rows), sum(cols))), np.zeros((sum(rows), sum(cols)))
    count = [0]

    def block(p, m, q, n):
        i, count[0] = count[0], count[0] + 1
        if i % 4 != 3:
            B = hm.BarycentricMatrix2D(hm.cauchykernel, 3.0, 2.0, 1.0, 0.0, x, y, range(p, p + m), range(q, q + n),
                                       rank=rank_of(i))
            U, C, V = (t.cpu().numpy() for t in (B.U, B.F, B.V))
        elif i % 8 == 3:
            r = min(9, m, n)
            U, s, V = rng.standard_normal((m, r)), rng.random(r) + 0.5, rng.standard_normal((n, r))
            C = np.diag(s)
            B = hm.LowRankMatrix(U, s, V)
        else:
            B = U = rng.standard_normal((m, n))
            C, V = np.eye(n), np.eye(n)
        D[p:p + m, q:q + n] = U @ C @ V.T
        S[p:p + m, q:q + n] = np.abs(U) @ np.abs(C) @ np.abs(V).T
        return B

    def grid(p, rs, q, cs, nested):
        H = Tree(len(rs), len(cs))
        at = np.concatenate([[p], p + np.cumsum(rs)]), np.concatenate([[q], q + np.cumsum(cs)])
        for i, m in enumerate(rs):
            for j, n in enumerate(cs):
                inner = nested and i == j == 0
                H[hm.Block(i + 1), hm.Block(j + 1)] = (
                    grid(p, [m // 3, m - m // 3], q, [n // 3, n - n // 3], False) if inner
                    else block(int(at[0][i]), m, int(at[1][j]), n))
        return H

    return grid(0, rows, 0, cols, True), D, S


def check(H, D, S, dtype, k, seed):
    tdt = torch.float64 if dtype == np.float64 else torch.float32
    X = torch.randn(k, D.shape[1], device="cuda", dtype=tdt, generator=torch.Generator("cuda").manual_seed(seed)).t()
    v = X[:, 0].contiguous() if k == 1 else X
    got = H @ v
    for _ in range(5):
        assert torch.equal(H @ v, got)
    _lib.check(_lib.lib.hm_configure(H.handle(dtype), _lib.HM_OPT_OVERLAP, 1))
    assert torch.equal(H @ v, got)
    H._invalidate()                                     # the default schedule again
    Xd = X.double().cpu().numpy()
    err = np.abs(got.double().cpu().numpy().reshape(-1, k) - D @ Xd)
    assert (err <= TERMS * np.finfo(dtype).eps / 2 * (S @ np.abs(Xd))).all()


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("grid", [(1, 1), (3, 2), (5, 3), (11, 3), (30, 3), (9, 6)])
def test_product(dtype, grid):
    rng = np.random.default_rng(grid[0])
    rows = [int(v) for v in rng.integers(8, 150, grid[0])]
    cols = [300, 8, 129, 40, 20, 3][:grid[1]]
    H, D, S = assemble(rows, cols, lambda i: 20, grid[0])
    for k in (1, 2, 4, 8) + ((9,) if grid[1] <= 3 else ()):      # above 8, panels of at most 363 FP64 columns
        check(H, D, S, dtype, k, k)


def test_strided_accumulating_product():
    H, D, S = assemble([60, 90, 20], [300, 8, 129], lambda i: 20, 1)
    m, n = D.shape
    g = torch.Generator("cuda").manual_seed(4)
    x, y0 = (torch.randn(3 * s, device="cuda", dtype=torch.float64, generator=g) for s in (n, m))
    y = y0.clone()
    H.mul(y, x, 3, 2, 2, 3)
    xs = x[1:1 + 2 * n:2].cpu().numpy()
    want = y0.clone()
    want[2::3][:m] += torch.tensor(D @ xs, device="cuda")
    bound = TERMS * np.finfo(np.float64).eps / 2 * (S @ np.abs(xs) + np.abs(y0[2::3][:m].cpu().numpy()))
    assert (np.abs((y - want)[2::3][:m].cpu().numpy()) <= bound).all()
    rest = torch.ones_like(y, dtype=torch.bool)
    rest[2::3] = False
    assert torch.equal(y[rest], y0[rest])
