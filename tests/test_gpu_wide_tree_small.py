"""HM_OPT_WIDE_TREE 2 ("all") is followed on small trees too: their products then take the
lane-per-right-hand-side kernels, as stages, instead of the two-launch form; same bits."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import hierarchicalmatrices as hm  # noqa: E402


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("n", [300, 1000, 3000])
def test_option_is_followed(dt, n):
    rng = np.random.default_rng(n)
    x, y = (np.sort(rng.random(n))[::-1].copy() for _ in range(2))
    H = hm.KernelMatrix(hm.logkernel, x, y, 1.0, 0.0, 1.0, 0.0, dtype=dt)
    for k in (1, 2, 3, 4, 8):
        X = torch.randn(k, n, device="cuda", dtype=torch.float32 if dt == np.float32 else torch.float64,
                        generator=torch.Generator("cuda").manual_seed(k)).t()
        ref = H @ X
        fused = H.stats()["fused_products"]
        H.set_wide_tree("all")
        for _ in range(4):
            assert torch.equal(H @ X, ref), k
        taken = H.stats()["fused_products"] - fused
        assert taken == 0 if k > 1 else taken in (0, 4)  # one right-hand side: not a wide product
        H.set_wide_tree(True)
    H.free()
