"""Which form a repeated product runs in (hm_stats): small trees in two launches, other forms
as a CUDA graph from the third call on, panels in chunks (more than eight vectors without
tensor cores) always as plain launches, and no capture is tried that cannot succeed."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import hierarchicalmatrices as hm  # noqa: E402

TDT = {np.float64: torch.float64, np.float32: torch.float32, "df64": torch.float64}
PLAIN, GRAPH, FUSED = "plain", "graph", "fused"


@pytest.mark.parametrize("n,dt,k,form", [
    (1000, np.float32, 3, FUSED), (1000, np.float64, 1, FUSED), (1000, "df64", 1, FUSED),
    (1000, np.float64, 9, GRAPH), (50000, np.float32, 1, GRAPH), (50000, np.float64, 3, GRAPH),
    (50000, "df64", 9, GRAPH), (50000, np.float32, 16, GRAPH), (50000, np.float32, 40, GRAPH),
    (50000, np.float64, 9, PLAIN), (50000, np.float64, 16, PLAIN), (50000, np.float64, 64, PLAIN),
    (50000, np.float32, 9, PLAIN), (50000, np.float32, 13, PLAIN)])
def test_forms(n, dt, k, form):
    rng = np.random.default_rng(n)
    x, y = (np.sort(rng.random(n))[::-1].copy() for _ in range(2))
    H = hm.KernelMatrix(hm.cauchykernel, x, y, 1.0, 0.0, 1.0, 0.0, dtype=dt)
    B = torch.randn(k, n, device="cuda", dtype=TDT[dt], generator=torch.Generator("cuda").manual_seed(k)).t()
    ref = H @ B
    for _ in range(6):
        assert torch.equal(H @ B, ref)
    st = H.stats()
    assert st["failed_captures"] == 0
    assert st["fused_products"] == (7 if form == FUSED else 0)
    assert st["graph_products"] == (5 if form == GRAPH else 0)
    H.free()
