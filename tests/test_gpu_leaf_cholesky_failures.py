"""Failing pivots of the hierarchical Cholesky's dense leaves, over and over, in the forms of
the leaf kernel (registers up to 64 and 96 rows, shared memory beyond)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import hierarchicalmatrices as hm  # noqa: E402
from test_gpu_leaf_cholesky import matrix, tree  # noqa: E402


@pytest.mark.parametrize("leaf", [3, 64, 96, 130])
def test_failures_repeat(leaf):
    """Two pivots fail in neighbouring steps: every repetition reports the first one, and
    the factor of a definite matrix between the failures stays the same."""
    good, bad = matrix(2 * leaf, np.random.default_rng(leaf)), matrix(2 * leaf, np.random.default_rng(leaf))
    at = leaf // 2
    bad[at, at] = bad[at + 1, at + 1] = -1.0
    G, B = tree(good, leaf, torch.float64), tree(bad, leaf, torch.float64)
    first = [hm.hierarchicalcholesky(G).block(i, i).clone() for i in (0, 1)]
    for _ in range(30):
        with pytest.raises(np.linalg.LinAlgError, match=rf"pivot {at + 1}$"):
            hm.hierarchicalcholesky(B)
        R = hm.hierarchicalcholesky(G)
        assert torch.equal(R.block(0, 0), first[0])
        # its solve takes a leaf's inverse where that is made by then: other roundings
        assert float(torch.linalg.norm(R.block(1, 1) - first[1])) <= 1e-12 * float(torch.linalg.norm(first[1]))
