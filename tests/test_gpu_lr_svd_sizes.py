"""Truncated SVDs of low-rank sums (hm_lr_svd) where its forms change: panels of
16/17, 32/33, 64/65, 128/129 and 256/257 rows, one row or column, fewer rows than
columns, panels that fit in shared memory and that do not, cores of 1 to 64, batches of
more problems than SMs, strongly graded spectra, one-sided QR.

The sum is compared as a matrix with the oracle's dense sum: 1e-12 (FP64) and 2e-5
(FP32) of its Frobenius norm; the factors are orthonormal to 1e-12 and 4 max(q,
20) eps, singular values descend."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import hierarchicalmatrices as hm  # noqa: E402
from hierarchicalmatrices import algebra as G  # noqa: E402

TOL = {torch.float64: 1e-12, torch.float32: 2e-5}


def factor(rng, m, n, r, decay, dt):
    U, _ = np.linalg.qr(rng.standard_normal((m, r)))
    V, _ = np.linalg.qr(rng.standard_normal((n, r)))
    s = decay ** np.arange(U.shape[1])[:V.shape[1]]
    q = len(s)
    L = hm.LowRankMatrix(*(torch.tensor(np.ascontiguousarray(a.T), dtype=dt, device="cuda").t() if a.ndim == 2 else
                           torch.tensor(a, dtype=dt, device="cuda") for a in (U[:, :q], s, V[:, :q])))
    return L, dense(L)


def dense(L):
    U, s, V = (t.double().cpu().numpy() for t in (L.U, L.sigma, L.V))
    return (U * s) @ V.T


def check(got, ref, dt):
    assert np.linalg.norm(dense(got) - ref) <= TOL[dt] * np.linalg.norm(ref)
    s = got.sigma.double().cpu().numpy()
    assert np.all(np.diff(s) <= 0) and np.all(s >= 0)
    tol = 1e-12 if dt == torch.float64 else 4 * max(len(s), 20) * 1.19e-7
    for F in (got.U, got.V):
        F = F.double().cpu().numpy()
        assert np.all(np.abs(F.T @ F - np.eye(F.shape[1])) < tol)          # rank 0: nothing to hold


SIZES = [(1, 1, 1, 1), (1, 40, 1, 1), (3, 40, 3, 3), (16, 17, 3, 4), (32, 33, 8, 8), (64, 65, 5, 5), (64, 64, 8, 9),
         (128, 129, 10, 6), (256, 257, 12, 12), (300, 20, 9, 9), (4000, 4000, 6, 6), (2000, 3000, 32, 32)]


@pytest.mark.parametrize("dt", [torch.float64, torch.float32])
@pytest.mark.parametrize("m,n,r1,r2", SIZES)
def test_sum(m, n, r1, r2, dt):
    rng = np.random.default_rng(m + n)
    for decay in (0.9, 0.3, 0.02):
        (L1, D1), (L2, D2) = factor(rng, m, n, r1, decay, dt), factor(rng, m, n, r2, decay, dt)
        check(G.lr_add(L1, L2), D1 + D2, dt)
        check(G.lr_sub(L1, L2), D1 - D2, dt)


@pytest.mark.parametrize("dt", [torch.float64, torch.float32])
def test_many_problems(dt):
    rng = np.random.default_rng(5)
    b, refs = G._SvdBatch(dt), []
    for i in range(200):
        m, n, r = 20 + i, 219 - i, 1 + i % 9
        (L1, D1), (L2, D2) = factor(rng, m, n, r, 0.5, dt), factor(rng, m, n, r, 0.5, dt)
        b.add(m, n, P=[(L1.U, r), (L2.U, r)], Q=[(L1.V, r), (L2.V, r)], s=[L1.sigma, L2.sigma])
        refs.append(D1 + D2)
    for got, ref in zip(b.run(), refs):
        check(got, ref, dt)


@pytest.mark.parametrize("dt", [torch.float64, torch.float32])
@pytest.mark.parametrize("m,n", [(1, 1), (17, 16), (33, 10), (65, 64), (257, 30), (1000, 100)])
def test_dense_block(m, n, dt):
    A = torch.randn(n, m, generator=torch.Generator().manual_seed(m), dtype=torch.float64).to("cuda", dt).t()
    check(hm.svdtrunc(A), A.double().cpu().numpy(), dt)
