"""HM_OPT_OVERLAP says where the near field starts: the values 1 to 4 literally, whatever the
default's rule (5) would take: no earlier than the named stage on the stages' times; a small matrix runs in two
launches by the rule only; the tuner's report names one of 0 to 4."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import hierarchicalmatrices as hm  # noqa: E402
from hierarchicalmatrices import _lib  # noqa: E402

TDT = {np.float64: torch.float64, np.float32: torch.float32}


def matrix(n, dt):
    i = np.arange(n)
    return hm.KernelMatrix(hm.cauchykernel, (i / n + 1 / (2 * n))[::-1].copy(), (i / n)[::-1].copy(), 1.0, 0.0, 1.0, 0.0,
                           dtype=dt)


def stages(H, u, b):
    H.profile()
    H.mul(u, b, accumulate=False)
    out = np.zeros(3 * 16)
    k = _lib.lib.hm_profile_timeline(H.handle, out.ctypes.data_as(ctypes.c_void_p), 16)
    H.profile([])
    H.stage_times(reset=True)
    return {_lib.STAGES[int(s)]: (a, b) for s, a, b in out[:3 * k].reshape(k, 3)}


# (above 8,192 slots, and for FP64 above 24,576, the rule starts the near field before the upward pass ends)
@pytest.mark.parametrize("n,dt", [(1 << 16, np.float32), (1 << 20, np.float32), (1 << 20, np.float64)])
def test_near_field_starts_after_the_named_stage(n, dt):
    H = matrix(n, dt)
    b = torch.randn(n, device="cuda", dtype=TDT[dt])
    ref = H @ b
    u = torch.empty_like(b)
    for mode in (0, 1, 2, 3, 4, 5):
        H.set_overlap(mode)
        for _ in range(3):
            t = stages(H, u, b)
            assert torch.equal(u, ref) and sorted(t) == sorted(_lib.STAGES)
            if mode == 2:
                assert t["expand"][0] >= t["up"][1]
            elif mode in (0, 3):                         # "down" holds the far-field stage and the downward pass
                assert t["expand"][0] >= t["down"][0 if mode == 3 else 1]
    H.set_overlap(True)
    H.free()


def test_two_launches_by_the_rule_only():
    H = matrix(2000, np.float64)
    b = torch.randn(2000, device="cuda", dtype=torch.float64)
    ref = H @ b
    for mode, count in ((0, 0), (1, 0), (2, 0), (3, 0), (4, 0), (5, 2), (True, 2)):
        H.set_overlap(mode)
        before = H.stats()["fused_products"]
        assert torch.equal(H @ b, ref) and torch.equal(H @ b, ref)
        assert H.stats()["fused_products"] - before == count, mode
    assert 0 <= H.schedule(1)["overlap"] <= 4
    for bad in (-1, 6):
        with pytest.raises(hm.HMError):
            H.set_overlap(bad)
    H.free()
