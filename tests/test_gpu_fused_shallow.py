"""The two-launch schedule on trees of one level (leaf bases and far-field blocks, no
transfers between): batches of matrices of 161 to 260 points with uneven panels, whose
leaf bases and far field keep several warps of a CTA busy at the same time.  Equal bit
for bit to the stage schedule, and to the dense product within the rank-20 error."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import hierarchicalmatrices as hm  # noqa: E402

TDT = {"f64": torch.float64, "f32": torch.float32, "df64": torch.float64}
STORE = {"f64": np.float64, "f32": np.float32, "df64": "df64"}


def shallow_points(count, seed):
    """Point sets of interleaved random sizes whose plans have far-field blocks and no transfers."""
    rng, xs, ys = np.random.default_rng(seed), [], []
    while len(xs) < count:
        n, m = rng.integers(161, 261, 2)
        x, y = np.sort(rng.random(n))[::-1].copy(), np.sort(rng.random(m))[::-1].copy()
        p = hm.Plan(x, y, 1.0, 0.0, 1.0, 0.0)
        if len(p.table("up_tasks")) == 0 and len(p.table("m2l_rows")) > 0:
            xs.append(x)
            ys.append(y)
    return xs, ys


@pytest.mark.parametrize("dtype", ["f64", "f32", "df64"])
@pytest.mark.parametrize("count", [5, 8, 20, 30])
def test_batches_without_transfers(dtype, count):
    xs, ys = shallow_points(count, count)
    H = hm.KernelMatrixBatch(hm.cauchykernel, xs, ys, [(1.0, 0.0, 1.0, 0.0)] * count, dtype=STORE[dtype])
    n, m = H.shape
    for k in (1, 2, 4, 8):
        g = torch.Generator("cuda").manual_seed(k)
        X = torch.randn(k, m, device="cuda", dtype=TDT[dtype], generator=g).t()
        H.set_overlap(1)
        staged = H @ X
        H.set_overlap(True)
        for _ in range(20):
            assert torch.equal(H @ X, staged), (count, k)
        at = 0
        for i, (x, y) in enumerate(zip(xs, ys)):
            D = 1.0 / (torch.tensor(x)[:, None] - torch.tensor(y)[None, :])
            ref = D @ X[H.col_offsets[i]:H.col_offsets[i + 1]].double().cpu()
            got = staged[at:at + len(x)].double().cpu()
            at += len(x)
            # against the rows' absolute sums (close pairs cancel): some 260 terms rounded
            # to 2^-24, and as much again for the rank-20 factors; FP64 and double-float
            # are bound by the rank-20 compression
            scale = D.abs() @ X[H.col_offsets[i]:H.col_offsets[i + 1]].double().cpu().abs()
            assert float(((got - ref).abs() / scale).max()) <= (3e-5 if dtype == "f32" else 1e-11)
    assert H.device_status() == 0
    H.free()
