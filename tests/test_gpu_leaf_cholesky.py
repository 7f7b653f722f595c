"""Dense diagonal leaves of the native hierarchical Cholesky at the sizes where its
forms change (1, 2, 31 to 33, 63 to 65, 80, 95 to 97, 130 rows): the factor R of [A B; B^T C]
against the FP64 dense factor, and the pivot that fails first.

R'R = A holds to n eps of |A| row by row for any order of the sums, so the factor of a matrix
of condition below 10 is compared to 1e-12 (FP64) and 1e-4 (FP32) of its norm."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import hierarchicalmatrices as hm  # noqa: E402

TOL = {torch.float64: 1e-12, torch.float32: 1e-4}
SIZES = [1, 2, 31, 32, 33, 63, 64, 65, 80, 95, 96, 97, 130]


def tree(K, n1, dt):
    def dev(a):
        return torch.tensor(np.ascontiguousarray(a.T), dtype=dt, device="cuda").t()
    H = hm.HierarchicalMatrix(2, 2, dtype=np.float64 if dt == torch.float64 else np.float32)
    u, s, vt = np.linalg.svd(K[:n1, n1:], full_matrices=False)
    H[hm.Block(1), hm.Block(1)] = dev(K[:n1, :n1])
    H[hm.Block(1), hm.Block(2)] = hm.LowRankMatrix(dev(u[:, :1]), torch.tensor(s[:1], dtype=dt, device="cuda"), dev(vt[:1].T))
    H[hm.Block(2), hm.Block(2)] = dev(K[n1:, n1:])
    return H


def matrix(n, rng):
    """Symmetric, eigenvalues in about [1, 3]; its off-diagonal block of rank one."""
    K = np.eye(n) * 2.0
    for lo, hi in ((0, n // 2), (n // 2, n)):
        G = rng.standard_normal((hi - lo, hi - lo))
        G = (G + G.T) / 2
        K[lo:hi, lo:hi] += 0.5 * G / max(np.linalg.norm(G, 2), 1e-300)
    u, v = rng.standard_normal(n // 2), rng.standard_normal(n - n // 2)
    B = 0.4 * np.outer(u, v) / (np.linalg.norm(u) * np.linalg.norm(v))
    K[:n // 2, n // 2:], K[n // 2:, :n // 2] = B, B.T
    return K


@pytest.mark.parametrize("dt", [torch.float64, torch.float32])
@pytest.mark.parametrize("leaf", SIZES)
def test_factor(leaf, dt):
    n = 2 * leaf
    K = matrix(n, np.random.default_rng(leaf))
    if dt == torch.float32:
        K = K.astype(np.float32).astype(np.float64)
    R = hm.hierarchicalcholesky(tree(K, leaf, dt))
    ref = np.linalg.cholesky(K).T
    R11, R22 = (R.block(i, i).double().cpu().numpy() for i in (0, 1))
    for got, want in ((R11, ref[:leaf, :leaf]), (R22, ref[leaf:, leaf:])):
        assert np.linalg.norm(got - want) <= TOL[dt] * np.linalg.norm(want)
        assert np.all(np.tril(got, -1) == 0)


@pytest.mark.parametrize("leaf", [1, 33, 64, 65, 96, 130])
def test_first_failing_pivot(leaf):
    for bad in sorted({0, leaf // 2, leaf - 1}):
        K = matrix(2 * leaf, np.random.default_rng(leaf))
        K[bad, bad] = -1.0
        with pytest.raises(np.linalg.LinAlgError, match=rf"pivot {bad + 1}$"):
            hm.hierarchicalcholesky(tree(K, leaf, torch.float64))
