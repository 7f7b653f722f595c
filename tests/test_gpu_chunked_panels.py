"""More than eight right-hand sides without the tensor cores (FP64; FP32 below 16 or with
them off) in chunks of eight on large trees, against one panel kernel for all of them
(near_kernel "warp"): 5e-7 and 1e-13 of the column's norm (FP32 sums folded with TwoSum,
FP64); last chunks of 1 to 8, u += H v, strided columns, one stream and two."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import hierarchicalmatrices as hm  # noqa: E402

TOL = {torch.float32: 5e-7, torch.float64: 1e-13}


@pytest.mark.parametrize("dtype,n", [(np.float32, 37000), (np.float32, 70001), (np.float64, 15000), (np.float64, 40001)])
def test_chunks(dtype, n):
    tdt = torch.float32 if dtype is np.float32 else torch.float64
    rng = np.random.default_rng(n)
    x, y = (np.sort(rng.random(n))[::-1].copy() for _ in range(2))
    H = hm.KernelMatrix(hm.cauchykernel, x, y, 1.0, 0.0, 1.0, 0.0, dtype=dtype)
    H.set_tensor_cores(False)
    for k in (9, 10, 12, 13, 16, 17, 24, 33):
        g = torch.Generator("cuda").manual_seed(k)
        B = torch.randn(k, n + 3, device="cuda", dtype=tdt, generator=g).t()[:n]
        U0 = torch.randn(k, n + 5, device="cuda", dtype=tdt, generator=g).t()[:n]
        for accumulate in (False, True):
            out = []
            for overlap, near in ((True, "auto"), (False, "auto"), (True, "warp")):
                H.set_overlap(overlap)
                H.set_near_kernel(near)
                U = torch.empty(k, n + 5, device="cuda", dtype=tdt).t()[:n]
                U.copy_(U0)
                H.mul(U, B, accumulate=accumulate)
                out.append(U)
            H.set_overlap(True)
            H.set_near_kernel("auto")
            assert torch.equal(out[0], out[1])
            err = torch.linalg.norm((out[0] - out[2]).double(), dim=0) / torch.linalg.norm(out[2].double(), dim=0)
            assert (err <= TOL[tdt]).all(), k
    assert H.device_status() == 0
    H.free()
