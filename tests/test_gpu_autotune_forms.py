"""The autotuner times its candidates in the form that products later run in (hm_stats): as
CUDA graphs where a repeated product is one, plainly where it is not, and the first
product with the chosen schedule has the bits of the later ones."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import hierarchicalmatrices as hm  # noqa: E402


@pytest.mark.parametrize("n,dt,k,graphs", [(50000, np.float32, 1, True), (50000, np.float64, 2, True),
                                           (50000, np.float32, 16, True), (50000, np.float64, 16, False)])
def test_trials_run_as_products_do(n, dt, k, graphs):
    rng = np.random.default_rng(n)
    x, y = (np.sort(rng.random(n))[::-1].copy() for _ in range(2))
    H = hm.KernelMatrix(hm.cauchykernel, x, y, 1.0, 0.0, 1.0, 0.0, dtype=dt)
    B = torch.randn(k, n, device="cuda", dtype=torch.float32 if dt == np.float32 else torch.float64,
                    generator=torch.Generator("cuda").manual_seed(k)).t()
    H.autotune(k, reps=3)
    assert (H.stats()["graph_products"] > 0) == graphs
    assert H.stats()["failed_captures"] == 0
    ref = H @ B
    for _ in range(5):
        assert torch.equal(H @ B, ref)
    assert H.stats()["failed_captures"] == 0 and H.device_status() == 0
    H.free()
