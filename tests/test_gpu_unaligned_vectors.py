"""Right-hand sides and results that start off a 16-byte boundary (views into larger
buffers), every product form by size and column count: the product of the view equals
the product of an aligned copy bit for bit (where no form chooses its copies by
alignment) or to the storage type's rounding."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import hierarchicalmatrices as hm  # noqa: E402

TDT = {"f32": torch.float32, "f64": torch.float64, "df64": torch.float64}
DT = {"f32": np.float32, "f64": np.float64, "df64": "df64"}


@pytest.mark.parametrize("n", [2000, 72000])
@pytest.mark.parametrize("dtype", ["f32", "f64", "df64"])
def test_offset_views(n, dtype):
    x = ((np.arange(n) + 0.75) / n)[::-1].copy()
    y = ((np.arange(n) + 0.25) / n)[::-1].copy()
    H = hm.KernelMatrix(hm.cauchykernel, x, y, 1.0, 0.0, 1.0, 0.0, dtype=DT[dtype])
    tdt = TDT[dtype]
    for k in (1, 2, 3, 8, 9, 17, 24, 40):
        g = torch.Generator("cuda").manual_seed(k)
        A = torch.randn(k, n, device="cuda", dtype=tdt, generator=g)
        ref = H @ (A.t() if k > 1 else A[0])
        ld = n + 4                                       # columns keep their distance mod 16 bytes
        for off in (1, 3):
            buf = torch.zeros(k * ld + 8, device="cuda", dtype=tdt)
            out = torch.full((k * ld + 8,), -7.0, device="cuda", dtype=tdt)
            B = buf[off:off + k * ld].view(k, ld)[:, :n]
            U = out[off:off + k * ld].view(k, ld)[:, :n]
            B.copy_(A)
            H.mul(U.t() if k > 1 else U[0], B.t() if k > 1 else B[0], accumulate=False)
            got = U.t() if k > 1 else U[0]
            err = torch.linalg.norm((got - ref).double()) / torch.linalg.norm(ref.double())
            assert err <= (1e-6 if dtype == "f32" else 1e-13)
            assert (out[:off] == -7.0).all()
            assert k == 1 or (out[off:off + k * ld].view(k, ld)[:, n:] == -7.0).all()
    assert H.device_status() == 0
    H.free()
